// Depthwise 3x3 convolution (stride 1 or 2, no dilation) on the warp-level tensor instruction.
//
// What bounds a depthwise layer is memory; what bounded the dp2a form of it (kernels_simt.cu) was issue: 28 - 38
// instructions per output.  Here one mma.sync.m16n8k32 does three taps (a filter row) of eight channels for sixteen
// pixels: K = 4 taps x 8 channels, the weight operand is diagonal in the channels (an eighth of the multiply-adds are
// real, the fourth tap is zero), and still an instruction that takes 8.5 cycles of a scheduler replaces 24 dp2a.  The
// fragment layout of the instruction makes the input side free: lane (g, q) holds, for pixel row g, the bytes of
// K slots 4 q .. 4 q + 3 and 16 + 4 q ..; calling those slots "tap q, channels 0 - 7" turns a lane's operand registers into
// one 16-byte shared-memory read of the pixel g + q, which serves two channel blocks.
//   - A warp owns 16 channels of a strip of 8 output columns and walks down its rows two at a time (rows of the
//     instruction: 8 columns x 2 output rows), keeping the input rows two units share in registers: at stride 1 two
//     16-byte reads and six tensor instructions per 256 outputs.
//   - Requantization in 64-bit fixed point (requant_fixed4's arithmetic), constants of the thread's four channels in
//     registers for the whole strip; two shuffles gather eight consecutive channels per thread.
//   - A block is G channel groups x NS strips and one warp that moves data.  The input patch of a tile (halo included,
//     zero fill outside the image) comes by TMA into three buffers, the output leaves by TMA from two: the computing
//     warps never wait for one another, so the one that has to redo a value exactly does not hold up the rest (with a
//     block barrier per tile the same layers took up to twice as long), and the output is written in whole pixels (as
//     8-byte stores it took 16 lines of the store path per 256 bytes, and slabs of 48 channels left half sectors).
//   - The slab of a tile is all channels of a pixel up to 144, else whole 32-byte sectors of them.  Pixels sit an odd
//     multiple of 16 bytes apart, so that the eight lanes of a read phase (five pixels) hit different banks; where the
//     slab is an even number of groups the box is one group wider than needed.
//   - Blocks are persistent and work through consecutive tiles of one channel slab, so weights and constants are loaded
//     once or twice.
// Needs: centred weights that fit int8, and padding that reads as zero (input zero point 0 where there is padding).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "kernels.h"
#include "pdl.cuh"
#include "requant.cuh"
#include "tma.cuh"

namespace b2vx {

struct DwMmaPlan {
  CUtensorMap map_x, map_y;
  struct Params {
    int Ho, Wo, N, Cp;
    int pl, pt;
    int groups;                      // G: 16-channel groups of a slab
    int pitch;                       // bytes from pixel to pixel of the patch
    int sx_shift, NI, items;         // tile: 1 << sx_shift strips side by side, NI images; items of a warp
    int TH;                          // output rows of a tile (even)
    int PW, PH;                      // input patch
    int tiles_w, tiles_h, tiles_n, tiles;
    uint32_t in_bytes, out_bytes, tx_bytes;   // one input buffer, one output buffer, one patch
    const int8_t* w;                 // [9][Cp] centred
    const FixedColumn* fix;          // [Cp]
    int shl;
    const int32_t* bias_full;
    const float* acc_scale;
    OutQuant out;
    int* status;
  } p;
  int stride, is_signed, warps, grid;
  size_t smem;
};

namespace {

// d = A B + c (c = 0 or d itself)
template <bool XS, bool FIRST>
__device__ __forceinline__ void mma_16832(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  const int c0 = FIRST ? 0 : d[0], c1 = FIRST ? 0 : d[1], c2 = FIRST ? 0 : d[2], c3 = FIRST ? 0 : d[3];
  if (XS)
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
  else
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}

constexpr int kStagesIn = 3;
constexpr int kMaxWarps = 9;         // computing warps of a block

struct DwExact { int bias; float scale; };   // of a channel, in shared memory: what the exact sequence needs besides the registers

// Those of a thread's four values (channels ch, ch + 1, ch + 8, ch + 9) whose fraction lies in the window, unless the
// integers on both sides of it saturate to the same result.
static __device__ __noinline__ uint32_t dw_redo4(uint32_t word, int x0, int x1, int x2, int x3, int4 mul, longlong2 add01, longlong2 add23,
                                             int shl, uint32_t window, const DwExact* exact, OutQuant oq) {
  const long long v0 = mad_wide(x0 << shl, mul.x, add01.x), v1 = mad_wide(x1 << shl, mul.y, add01.y);
  const long long v2 = mad_wide(x2 << shl, mul.z, add23.x), v3 = mad_wide(x3 << shl, mul.w, add23.y);
  uint32_t hits = (static_cast<uint32_t>(v0) < window ? 1u : 0u) | (static_cast<uint32_t>(v1) < window ? 2u : 0u) |
                  (static_cast<uint32_t>(v2) < window ? 4u : 0u) | (static_cast<uint32_t>(v3) < window ? 8u : 0u);
#pragma unroll 1
  while (hits) {
    const int k = __ffs(hits) - 1;
    hits &= hits - 1;
    const int acc = k & 2 ? (k & 1 ? x3 : x2) : (k & 1 ? x1 : x0);
    const int hi = static_cast<int>((k & 2 ? (k & 1 ? v3 : v2) : (k & 1 ? v1 : v0)) >> 32);
    if (static_cast<uint32_t>(hi - 1) >= 255u) continue;
    const DwExact d = exact[(k & 1) + (k >> 1) * 8];
    const float real = __fmul_rn(__int2float_rn(acc + d.bias), d.scale);
    word = (word & ~(0xFFu << (8 * k))) | requant_near_half(real, hi, oq) << (8 * k);
  }
  return word;
}

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(src)
               : "memory");
}

// SHL: some multiplier had to be halved to fit 31 bits (p.shl)
template <int S, bool XS, bool SHL>
__global__ void __launch_bounds__((kMaxWarps + 1) * 32, 2)
depthwise_mma_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y, const __grid_constant__ DwMmaPlan::Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ unsigned long long in_full[kStagesIn], out_full[2], out_free[2];
  __shared__ int abort_flag;
  __shared__ DwExact exact_of[kMaxWarps][16];
  pdl_trigger();
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, out_base = base + kStagesIn * p.in_bytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (blockDim.x >> 5) - 1;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStagesIn; ++i) mbar_init(smem_u32(&in_full[i]), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&out_full[i]), warps);
      mbar_init(smem_u32(&out_free[i]), 1);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // this block's run of consecutive tiles; tile order: columns, rows, images, slabs
  const int t0 = static_cast<int>(static_cast<long long>(p.tiles) * blockIdx.x / gridDim.x);
  const int t1 = static_cast<int>(static_cast<long long>(p.tiles) * (blockIdx.x + 1) / gridDim.x);
  struct Tile { int tw, th, tn, slab; };
  auto next = [&](Tile& k) {
    if (++k.tw < p.tiles_w) return;
    k.tw = 0;
    if (++k.th < p.tiles_h) return;
    k.th = 0;
    if (++k.tn < p.tiles_n) return;
    k.tn = 0;
    ++k.slab;
  };
  Tile cur;
  {
    int t = t0;
    cur.tw = t % p.tiles_w; t /= p.tiles_w;
    cur.th = t % p.tiles_h; t /= p.tiles_h;
    cur.tn = t % p.tiles_n;
    cur.slab = t / p.tiles_n;
  }
  const int slab_ch = 16 * p.groups, tile_w = 8 << p.sx_shift;
  __syncthreads();

  if (warp == warps) {
    // ------------------------------------------------------------ data movement
    if (lane != 0) return;
    Tile ahead = cur;                  // next tile to load
    auto load = [&](int st) {
      const uint32_t bar = smem_u32(&in_full[st]);
      mbar_arrive_expect_tx(bar, p.tx_bytes);
      tma_load_4d(base + st * p.in_bytes, &map_x, ahead.slab * slab_ch, ahead.tw * tile_w * S - p.pl, ahead.th * p.TH * S - p.pt, ahead.tn * p.NI, bar);
      next(ahead);
    };
    pdl_wait();
    for (int t = t0; t < t1 && t < t0 + kStagesIn; ++t) load(t - t0);
    int st = 0;
    bool ok = true;
    for (int t = t0; t < t1; ++t, next(cur)) {
      const int b = (t - t0) & 1;
      ok = mbar_wait(smem_u32(&out_full[b]), ((t - t0) >> 1) & 1, &abort_flag, p.status, 31);
      if (!ok) break;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tma_store_4d(&map_y, out_base + b * p.out_bytes, cur.slab * slab_ch, cur.tw * tile_w, cur.th * p.TH, cur.tn * p.NI);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      if (t + kStagesIn < t1) load(st);          // every warp is done with this tile's input
      if (++st == kStagesIn) st = 0;
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      mbar_arrive(smem_u32(&out_free[b]));
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    // gave up: let the copies in flight land before the shared memory is handed on (bounded again)
    if (!ok)
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    return;
  }

  // -------------------------------------------------------------- arithmetic
  const int strip = warp / p.groups, cg = warp - strip * p.groups, strips = warps / p.groups;
  const int g = lane >> 2, q = lane & 3;
  uint32_t bw[3][2][2];              // [filter row][8-channel block][operand register]
  int4 mul = make_int4(0, 0, 0, 0);
  longlong2 add01 = make_longlong2(0, 0), add23 = make_longlong2(0, 0);
  uint32_t window = 0;
  int cur_slab = -1, st = 0;
  uint32_t st_phase = 0;
  const DwExact* exact = &exact_of[warp][2 * q];
  const uint32_t flip = p.out.lo < 0 ? 0x80808080u : 0u;
  const int shl = SHL ? p.shl : 0;
  const uint32_t row_pitch = static_cast<uint32_t>(p.PW * p.pitch), out_row = static_cast<uint32_t>(tile_w * slab_ch);
  for (int t = t0; t < t1; ++t, next(cur)) {
    const int b = (t - t0) & 1;
    const int c0 = cur.slab * slab_ch + cg * 16;
    const bool live = c0 < p.Cp;
    if (cur.slab != cur_slab) {
      cur_slab = cur.slab;
      if (live) {
        // operand B: lane (n = g, tap q) holds channel n's weight of tap q, at byte n of register 0 (n < 4) or n - 4 of 1
#pragma unroll
        for (int ky = 0; ky < 3; ++ky)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t v = q < 3 ? static_cast<uint32_t>(static_cast<uint8_t>(__ldg(p.w + (ky * 3 + q) * p.Cp + c0 + h * 8 + g))) << (8 * (g & 3)) : 0u;
            bw[ky][h][0] = g < 4 ? v : 0u;
            bw[ky][h][1] = g < 4 ? 0u : v;
          }
        const int ch = c0 + 2 * q;     // first of this thread's channels
        const FixedColumn f0 = p.fix[ch], f1 = p.fix[ch + 1], f2 = p.fix[ch + 8], f3 = p.fix[ch + 9];
        mul = make_int4(f0.mul, f1.mul, f2.mul, f3.mul);
        add01 = make_longlong2(f0.add, f1.add);
        add23 = make_longlong2(f2.add, f3.add);
        window = f0.window;
        __syncwarp();
        if (lane < 16) exact_of[warp][lane] = {__ldg(p.bias_full + c0 + lane), __ldg(p.acc_scale + c0 + lane)};
        __syncwarp();
      }
    }
    bool ok = mbar_wait(smem_u32(&in_full[st]), st_phase, &abort_flag, p.status, 30);
    if (ok && t - t0 >= 2) ok = mbar_wait(smem_u32(&out_free[b]), (((t - t0) >> 1) & 1) ^ 1, &abort_flag, p.status, 32);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) return;
    const int rows = min(p.TH, p.Ho - cur.th * p.TH);
    if (live) {
      for (int it = 0, item = strip; it < p.items; ++it, item += strips) {
        const int xs = item & ((1 << p.sx_shift) - 1), ni = item >> p.sx_shift;
        if (cur.tn * p.NI + ni >= p.N || cur.tw * tile_w + xs * 8 >= p.Wo) continue;
        uint32_t at = base + st * p.in_bytes + static_cast<uint32_t>((ni * p.PH * p.PW + (xs * 8 + g) * S + q) * p.pitch + cg * 16);
        uint32_t dst = out_base + b * p.out_bytes + static_cast<uint32_t>(((ni * p.TH + (q & 1)) * tile_w + xs * 8 + g) * slab_ch + cg * 16 + 8 * (q >> 1));
        auto next_row = [&](uint32_t (&v)[4]) {   // 16 channels of this lane's pixel; rows are read in order
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at));
          at += row_pitch;
        };
        // One unit: the next two output rows from patch rows r0, r1, r2 and s0, s1, s2.
        auto unit = [&](const uint32_t (&r0)[4], const uint32_t (&r1)[4], const uint32_t (&r2)[4], const uint32_t (&s0)[4], const uint32_t (&s1)[4],
                        const uint32_t (&s2)[4]) {
          int lo[4], hi[4];
          mma_16832<XS, true>(lo, r0[0], s0[0], r0[1], s0[1], bw[0][0][0], bw[0][0][1]);
          mma_16832<XS, true>(hi, r0[2], s0[2], r0[3], s0[3], bw[0][1][0], bw[0][1][1]);
          mma_16832<XS, false>(lo, r1[0], s1[0], r1[1], s1[1], bw[1][0][0], bw[1][0][1]);
          mma_16832<XS, false>(hi, r1[2], s1[2], r1[3], s1[3], bw[1][1][0], bw[1][1][1]);
          mma_16832<XS, false>(lo, r2[0], s2[0], r2[1], s2[1], bw[2][0][0], bw[2][0][1]);
          mma_16832<XS, false>(hi, r2[2], s2[2], r2[3], s2[3], bw[2][1][0], bw[2][1][1]);
          const int xa[4] = {lo[0], lo[1], hi[0], hi[1]}, xb[4] = {lo[2], lo[3], hi[2], hi[3]};
          uint32_t la, lb;
          uint32_t wa = requant_fixed4(xa, mul, add01, add23, shl, la), wb = requant_fixed4(xb, mul, add01, add23, shl, lb);
          if (min(la, lb) < window) {
            if (la < window) wa = dw_redo4(wa, xa[0], xa[1], xa[2], xa[3], mul, add01, add23, shl, window, exact, p.out);
            if (lb < window) wb = dw_redo4(wb, xb[0], xb[1], xb[2], xb[3], mul, add01, add23, shl, window, exact, p.out);
          }
          // bytes of a word: channels 2q, 2q+1, 8+2q, 9+2q.  Even lanes end up with the first row, odd ones with the
          // second, then lanes 0, 1 of a quad with channels 0-7 and lanes 2, 3 with channels 8-15.
          const bool odd = q & 1, upper = q & 2;
          const uint32_t keep = odd ? wb : wa, got = __shfl_xor_sync(0xffffffffu, odd ? wa : wb, 1);
          const uint32_t first = odd ? got : keep, second = odd ? keep : got;
          const uint32_t l4 = __byte_perm(first, second, 0x5410), h4 = __byte_perm(first, second, 0x7632);
          const uint32_t far = __shfl_xor_sync(0xffffffffu, upper ? l4 : h4, 2);
          asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(dst), "r"((upper ? far : l4) ^ flip), "r"((upper ? h4 : far) ^ flip) : "memory");
          dst += 2 * out_row;
        };
        if (S == 1) {
          uint32_t r0[4], r1[4], r2[4], r3[4];
          next_row(r0);
          next_row(r1);
          for (int u = 0; u < rows; u += 4) {
            next_row(r2);
            next_row(r3);
            unit(r0, r1, r2, r1, r2, r3);
            if (u + 2 >= rows) break;
            next_row(r0);
            next_row(r1);
            unit(r2, r3, r0, r3, r0, r1);
          }
        } else {
          uint32_t r0[4], r1[4], r2[4], r3[4], r4[4];
          next_row(r0);
          for (int u = 0; u < rows; u += 2) {
            next_row(r1);
            next_row(r2);
            next_row(r3);
            next_row(r4);
            unit(r0, r1, r2, r2, r3, r4);
#pragma unroll
            for (int k = 0; k < 4; ++k) r0[k] = r4[k];
          }
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the output goes on by TMA
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&out_full[b]));
    if (++st == kStagesIn) { st = 0; st_phase ^= 1; }
  }
}

typedef void (*DwMmaKernel)(CUtensorMap, CUtensorMap, DwMmaPlan::Params);

template <bool SHL>
DwMmaKernel dw_kernel(int stride, bool is_signed) {
  return stride == 1 ? (is_signed ? depthwise_mma_kernel<1, true, SHL> : depthwise_mma_kernel<1, false, SHL>)
                     : (is_signed ? depthwise_mma_kernel<2, true, SHL> : depthwise_mma_kernel<2, false, SHL>);
}
DwMmaKernel dw_kernel(const DwMmaPlan& pl) { return pl.p.shl ? dw_kernel<true>(pl.stride, pl.is_signed != 0) : dw_kernel<false>(pl.stride, pl.is_signed != 0); }

}  // namespace

DwMmaPlan* dw_mma_plan_create(const void* x, int x_signed, const int8_t* w, const FixedColumn* fix, int shl, const int32_t* bias_full,
                              const float* acc_scale, const ConvGeom& g, OutQuant out, void* y, int* status) {
  const int S = g.sx, all = g.Cp / 16;
  if (g.kh != 3 || g.kw != 3 || g.dx != 1 || g.dy != 1 || g.sx != g.sy || (S != 1 && S != 2) || g.Cp != g.Ocp) return nullptr;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  DwMmaPlan* pl = new DwMmaPlan();
  std::memset(pl, 0, sizeof(*pl));
  DwMmaPlan::Params& p = pl->p;
  // Channel groups of a slab: all of them up to nine, else whole sectors (an even number), the split that leaves the
  // fewest groups idle; among equals the one that fills a block with eight warps (8 groups, or 4 of two strips) before the one
  // that makes six: two blocks of either share an SM.  Batch 256: 28 x 28 x 192 57.1 us with 6 groups, 43.0 with 4; 14 x 14 x 576
  // 46.1 and 34.5; 7 x 7 x 960 25.1 and 22.5.  (Fewest idle groups first is not always fastest: at 288, 480 and 672 channels 6
  // groups leave none idle, and eight warps with some idle take less: 28 x 28 x 288 at batch 256 65.8 us with 6 groups and 58.3 with 4,
  // 14 x 14 x 480 34.5 and 29.1 with 8, 14 x 14 x 672 41.4 and 34.6 with 4.  Below one wave of tiles the widths are within 0.5 us.)
  p.groups = all;
  if (all > kMaxWarps) {
    int best_idle = 1 << 30;
    for (int c : {8, 4, 6}) {
      const int idle = (all + c - 1) / c * c - all;
      if (idle < best_idle) { best_idle = idle; p.groups = c; }
    }
  }
  const int G = p.groups, slabs = (all + G - 1) / G;
  const int ns = G == 1 ? 8 : G == 2 ? 4 : G <= 4 ? 2 : 1;
  pl->warps = G * ns;
  p.pitch = 16 * (G | 1);
  // Tile: strips side by side x rows x images.  Three blocks per SM where their registers fit (up to six warps), or two, each
  // with its share of the shared memory.  A tile costs its units (two rows of a strip) or the bytes it moves, whichever is more,
  // plus a fixed part (units of 2 rows; 8.4 KB is what an SM moves from DRAM in the time of one); the launch as many
  // waves of that as the tiles make.
  const int per_sm_target = pl->warps + 1 <= 6 ? 3 : 2;
  const size_t budget = (per_sm_target == 3 ? 74 : 112) * 1024;
  const int strips_w = (g.Wo + 7) / 8;
  double best_cost = -1.0;
  for (int sh = 0; sh <= 3 && (sh == 0 || (1 << (sh - 1)) < strips_w); ++sh)
    for (int ni = 1; ni <= 16 && (ni <= ns || ni < 2 * g.N); ni *= 2) {
      const int strips_t = ni << sh;
      if (strips_t % ns) continue;
      for (int th = 2; th <= 32 && th < g.Ho + 2; th += 2) {
        const int pw = ((8 << sh) - 1) * S + 3, ph = (th - 1) * S + 3;
        const size_t in = (static_cast<size_t>(ni) * ph * pw + 1) * p.pitch, ob = static_cast<size_t>(ni) * th * (8 << sh) * 16 * G;
        if (kStagesIn * (in + 1024) + 2 * (ob + 1024) + 1024 > budget || pw > 256) continue;
        const int tw = (strips_w + (1 << sh) - 1) >> sh, thn = (g.Ho + th - 1) / th, tn = (g.N + ni - 1) / ni;
        const double tiles = static_cast<double>(tw) * thn * tn * slabs, slots = static_cast<double>(per_sm_target) * sms;
        const double waves = tiles <= slots ? 1.0 : tiles <= 8 * slots ? std::ceil(tiles / slots) : tiles / slots;
        const double work = static_cast<double>(strips_t / ns) * (0.5 * th + 0.7), move = (in + ob) * per_sm_target / 8400.0;
        const double cost = waves * (std::max(work, move) + 2.0);
        if (best_cost < 0.0 || cost < best_cost) {
          best_cost = cost;
          p.sx_shift = sh; p.NI = ni; p.TH = th; p.PW = pw; p.PH = ph;
          p.items = strips_t / ns;
          p.tiles_w = tw; p.tiles_h = thn; p.tiles_n = tn;
        }
      }
    }
  const double tiles = static_cast<double>(p.tiles_w) * p.tiles_h * p.tiles_n * slabs;
  if (best_cost < 0.0 || tiles > 1e9) { delete pl; return nullptr; }
  p.tiles = static_cast<int>(tiles);
  p.tx_bytes = static_cast<uint32_t>(p.NI * p.PH * p.PW * p.pitch);
  p.in_bytes = (p.tx_bytes + p.pitch + 1023u) & ~1023u;   // + the zero tap's pixel behind the last row
  p.out_bytes = static_cast<uint32_t>(p.NI * p.TH * (8 << p.sx_shift) * 16 * G + 1023) & ~1023u;
  pl->smem = kStagesIn * static_cast<size_t>(p.in_bytes) + 2 * static_cast<size_t>(p.out_bytes) + 1024;
  p.Ho = g.Ho; p.Wo = g.Wo; p.N = g.N; p.Cp = g.Cp; p.pl = g.pl; p.pt = g.pt;
  p.w = w; p.fix = fix; p.shl = shl; p.bias_full = bias_full; p.acc_scale = acc_scale; p.out = out;
  p.status = status;
  pl->stride = S; pl->is_signed = x_signed;
  const uint64_t xdims[4] = {static_cast<uint64_t>(g.Cp), static_cast<uint64_t>(g.W), static_cast<uint64_t>(g.H), static_cast<uint64_t>(g.N)};
  const uint64_t ydims[4] = {static_cast<uint64_t>(g.Cp), static_cast<uint64_t>(g.Wo), static_cast<uint64_t>(g.Ho), static_cast<uint64_t>(g.N)};
  const uint32_t xbox[4] = {static_cast<uint32_t>(p.pitch), static_cast<uint32_t>(p.PW), static_cast<uint32_t>(p.PH), static_cast<uint32_t>(p.NI)};
  const uint32_t ybox[4] = {static_cast<uint32_t>(16 * G), static_cast<uint32_t>(8 << p.sx_shift), static_cast<uint32_t>(p.TH), static_cast<uint32_t>(p.NI)};
  const DwMmaKernel k = dw_kernel(*pl);
  int per_sm = 0;
  if (!encode_u8(&pl->map_x, x, 4, xdims, xbox, nullptr, CU_TENSOR_MAP_SWIZZLE_NONE) ||
      !encode_u8(&pl->map_y, y, 4, ydims, ybox, nullptr, CU_TENSOR_MAP_SWIZZLE_NONE) ||
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * (pl->warps + 1), pl->smem) != cudaSuccess || per_sm < 1) {
    delete pl;
    return nullptr;
  }
  pl->grid = static_cast<int>(std::min(static_cast<double>(per_sm) * sms, tiles));
  return pl;
}

void dw_mma_plan_destroy(DwMmaPlan* p) { delete p; }

cudaError_t dw_mma_launch(const DwMmaPlan* pl, cudaStream_t s) {
  return launch_pdl(dw_kernel(*pl), dim3(pl->grid), dim3(32 * (pl->warps + 1)), pl->smem, s, pl->map_x, pl->map_y, pl->p);
}

}  // namespace b2vx
