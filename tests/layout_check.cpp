// A mesh slot's layout (huji-rich_gb300/csrc/rg_handle.cuh), host build: on the
// FP32-mixed path the FP64 slopes' centroid offsets take no memory of their own
// (they lie in the per-face scratch of the direct FP32 geometry pass), on the
// FP64 path they follow the other arrays.
#include <cstdio>

#include "rg_handle.cuh"

int main() {
  int bad = 0;
  const int sizes[][4] = {{1, 0, 0, 0}, {1, 1, 1, 1}, {64, 32, 209, 386}, {9696, 390, 29483, 58174}, {1048576, 4096, 3149824, 6291456}};
  for (const auto& s : sizes)
    for (const bool mixed : {false, true})
      for (const bool cyl : {false, true}) {
        rgh::SlotLayout L;
        const int n = s[0], g = s[1], e = s[2], m = s[3];
        L.compute(n, g, e, m, mixed, cyl);
        const size_t dmf_end = L.dmf + 8 * static_cast<size_t>(m), frec_end = L.frec32 + 32 * static_cast<size_t>(e);
        const bool ok = L.dmf == L.frec32 && (mixed ? dmf_end <= frec_end : true) &&
                        L.ghost_real == rgh::align_up(mixed ? frec_end : dmf_end) &&
                        L.total == rgh::align_up(L.icdv32 + (mixed ? 4 * static_cast<size_t>(n) : 0));
        if (!ok) {
          std::printf("n %d e %d m %d mixed %d: dmf %zu..%zu, scratch %zu..%zu, total %zu\n", n, e, m, mixed, L.dmf,
                      dmf_end, L.frec32, frec_end, L.total);
          ++bad;
        }
      }
  return bad != 0;
}
