// mul_check.cu -- huji-rich_gb300/csrc/rg_mul.cuh against the IEEE product,
// bit for bit: built by g++ (-x c++) the host form, by nvcc the device form.
// Prints one JSON line: cases, mismatches, products taken by the fast path.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "mul_cases.h"
#include "rg_mul.cuh"

#ifdef __CUDACC__
__global__ void k(const double* a, const double* b, int n, unsigned long long* bad, unsigned long long* fast) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double want = __dmul_rn(a[i], b[i]);
  double f;
  if (rg::mul_rn_fast(a[i], b[i], &f)) atomicAdd(fast, 1ull);
  const double one = rg::mul_rn(a[i], b[i]);
  double x, y;
  rg::mul_rn2(rg::mul_factor(a[i]), a[i], b[i], a[i], x, y);
  const double sq = __dmul_rn(a[i], a[i]);
  const bool nan = isnan(want), nan2 = isnan(sq);
  const bool ok = (nan ? isnan(one) && isnan(x) : __double_as_longlong(one) == __double_as_longlong(want) &&
                                                      __double_as_longlong(x) == __double_as_longlong(want)) &&
                  (nan2 ? isnan(y) : __double_as_longlong(y) == __double_as_longlong(sq));
  if (!ok) atomicAdd(bad, 1ull);
}
#endif

int main(int, char** argv) {
  std::mt19937_64 rng(std::strtoull(argv[2], nullptr, 10));
  std::vector<double> a, b;
  mulcases::generate(rng, std::strtoll(argv[1], nullptr, 10), [&](double x, double y) {
    a.push_back(x);
    b.push_back(y);
  });
  unsigned long long bad = 0, fast = 0;
#ifdef __CUDACC__
  const int n = static_cast<int>(a.size());
  double *da, *db;
  unsigned long long* cnt;
  cudaMalloc(&da, 8 * a.size());
  cudaMalloc(&db, 8 * a.size());
  cudaMalloc(&cnt, 16);
  cudaMemset(cnt, 0, 16);
  cudaMemcpy(da, a.data(), 8 * a.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(db, b.data(), 8 * a.size(), cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(da, db, n, cnt, cnt + 1);
  unsigned long long h[2] = {1, 0};
  if (cudaMemcpy(h, cnt, 16, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  bad = h[0];
  fast = h[1];
#else
  for (size_t i = 0; i < a.size(); ++i) {
    double p;
    if (!rg::mul_rn_fast(a[i], b[i], &p)) continue;
    ++fast;
    const volatile double w = a[i] * b[i];
    const double want = w;
    bad += std::memcmp(&p, &want, 8) != 0;
  }
#endif
  std::printf("{\"cases\": %zu, \"mismatches\": %llu, \"fast\": %llu}\n", a.size(), bad, fast);
  return bad != 0;
}
