// Launch shapes (huji-rich_gb300/csrc/rg_internal.cuh), host build: a shape that
// a caller or the autotuner set is launched as it is on every mesh; a built-in
// one gives every SM two blocks where the items and the smallest block allow.
#include <cstdio>

#include "rg_internal.cuh"

int main() {
  int bad = 0;
  const long long counts[] = {0, 1, 31, 64, 1000, 9696, 19455, 19456, 77823, 77824, 155647, 155648, 3000000};
  for (long long items : counts) {
    for (int block : {32, 64, 96, 128, 256, 480, 512})
      for (int max_blocks : {0, 7, 304}) {
        const rg::LaunchShape set{block, max_blocks, 0};
        const rg::LaunchShape got = rg::fit_shape(set, items);
        if (got.block != block || got.max_blocks != max_blocks || got.variant != 0) {
          std::printf("set %d x %d launched as %d x %d on %lld items\n", block, max_blocks, got.block,
                      got.max_blocks, items);
          ++bad;
        }
      }
    for (int sms : {76, 152})
      for (int block : {128, 256, 512}) {
        const int got = rg::fit_shape(rg::LaunchShape{block, 0, 0, sms}, items).block;
        int want = 64;  // the largest halving, no less than 64, with two blocks for every SM
        for (int b = block; b > 64; b /= 2)
          if (items >= 2LL * sms * b) {
            want = b;
            break;
          }
        if (got != want) {
          std::printf("built-in %d on %d SMs: %d, not %d, for %lld items\n", block, sms, got, want, items);
          ++bad;
        }
      }
  }
  return bad != 0;
}
