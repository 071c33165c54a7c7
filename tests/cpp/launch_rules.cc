// Prints what the host-side launch rules of the CUDA library choose; one question per argument, its fields separated by commas:
//   pieces,M,Kp,sms             128-row pieces that a tile of a plain GEMM may have
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
    else return 2;
  }
  return 0;
}
