// Prints what the host-side launch rules of the CUDA library choose; one question per argument, its fields separated by commas:
//   pieces,M,Kp,sms             128-row pieces that a tile of a plain GEMM may have
//   conv,N,W,H,k,stride,C,Oc    an implicit convolution with SAME padding, on 148 SMs: M tiles, N tiles, columns of a tile, of a
//                               column block, whether no CTA gets a second tile
//   gemm,M,K,Oc                 a plain GEMM, the same answers
//   im2col,N,W,H,C,kw,kh,sx,sy,same,sms   output rows that a block of the first layer's im2col takes, how many blocks there are, output rows
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "kernels.h"

int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i) {
    std::vector<int> v;
    const std::string what(argv[i], std::strcspn(argv[i], ","));
    for (const char* p = std::strchr(argv[i], ','); p; p = std::strchr(p + 1, ',')) v.push_back(std::atoi(p + 1));
    if (what == "pieces" && v.size() == 3) std::printf("%d\n", b2vx::gemm_tc_max_pieces(v[0], v[1], v[2]));
    else if (what == "conv" && v.size() == 7) {
      b2vx::ConvGeom g = {};
      g.N = v[0]; g.W = v[1]; g.H = v[2]; g.kw = g.kh = v[3]; g.sx = g.sy = v[4]; g.dx = g.dy = 1;
      g.Wo = (g.W + g.sx - 1) / g.sx; g.Ho = (g.H + g.sy - 1) / g.sy;
      g.C = v[5]; g.Oc = v[6]; g.Cp = (g.C + 15) / 16 * 16; g.Ocp = (g.Oc + 15) / 16 * 16;
      const long long tiles = b2vx::gemm_tc_conv_m_tiles(g);
      const b2vx::GemmTcTiling t = b2vx::gemm_tc_choose_tiling(static_cast<long long>(g.N) * g.Wo * g.Ho, g.Ocp, g.kw * g.kh * g.Cp, 0, tiles);
      std::printf("%lld %d %d %d %d\n", tiles, t.n_tiles, t.data, t.blk_w, t.one_each);
    } else if (what == "gemm" && v.size() == 3) {
      const b2vx::GemmTcTiling t = b2vx::gemm_tc_choose_tiling(v[0], (v[2] + 15) / 16 * 16, (v[1] + 15) / 16 * 16, 0);
      std::printf("%d %d %d %d %d\n", (v[0] + 127) / 128, t.n_tiles, t.data, t.blk_w, t.one_each);
    } else if (what == "im2col" && v.size() == 10) {
      b2vx::ConvGeom g = {};
      g.N = v[0]; g.W = v[1]; g.H = v[2]; g.C = v[3]; g.kw = v[4]; g.kh = v[5]; g.sx = v[6]; g.sy = v[7]; g.dx = g.dy = 1;
      g.Wo = (g.W - (v[8] ? 1 : g.kw)) / g.sx + 1; g.Ho = (g.H - (v[8] ? 1 : g.kh)) / g.sy + 1;
      const int padk = g.kw <= 4 ? 4 : 8;
      int Kp = (g.kh * g.C * padk + 15) / 16 * 16;
      if (Kp > 64) Kp = (Kp + 63) / 64 * 64;
      const int rows = b2vx::im2col_whcn8_rows(g, Kp, padk, v[9]);
      std::printf("%d %d %d\n", rows, g.N * ((g.Ho + rows - 1) / rows), g.Ho);
    } else return 2;
  }
  return 0;
}
