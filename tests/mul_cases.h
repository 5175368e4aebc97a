// mul_cases.h -- operand families for the FP64 multiplication check
// (tests/mul_check.cu: the host build and, with a GPU, the device build).
#pragma once
#include <cstdint>
#include <cstring>
#include <random>

namespace mulcases {

inline double from(uint64_t u) {
  double x;
  std::memcpy(&x, &u, 8);
  return x;
}

// calls check(a, b) for about 6 n pairs
template <class F>
void generate(std::mt19937_64& rng, long long n, F&& check) {
  const uint64_t f = (uint64_t(1) << 52) - 1;
  auto any = [&](int lo, int hi) {
    return from((rng() & 1) << 63 | (lo + rng() % static_cast<uint64_t>(hi - lo)) << 52 | (rng() & f));
  };
  auto few = [&](int bits) {  // significands of few bits: exact products, ties at the 54th bit
    return from((rng() & 1) << 63 | (1000 + rng() % 46) << 52 | ((rng() & f) >> (52 - bits) << (52 - bits)));
  };
  const double edge[] = {0.0, -0.0, 1.0, -1.0, 2.0, from(1), from(f), from(f + 1), from(f + 2), from(0x7fefffffffffffffull),
                         from(0x7ff0000000000000ull), from(0xfff0000000000000ull), from(0x3fefffffffffffffull),
                         from(0x3ff0000000000001ull), from(0x1ff0000000000000ull), from(0x2000000000000000ull),
                         from(0x5fe0000000000000ull), from(0x5fffffffffffffffull)};
  for (double a : edge)
    for (double b : edge) check(a, b);
  for (long long i = 0; i < n; ++i) {
    check(from(rng()), from(rng()));                                // every class
    check(any(1, 2047), any(1, 2047));                              // normals
    check(any(1000, 1046), any(1000, 1046));                        // the physics range
    const int b = static_cast<int>(rng() % 53);
    check(few(b), few(b < 53 ? 53 - b > 52 ? 52 : 53 - b : 0));     // 54-bit products: ties
    check(few(static_cast<int>(rng() % 53)), few(static_cast<int>(rng() % 53)));
    const int e = 1 + static_cast<int>(rng() % 2046);               // results at both ends of the range
    const int s = (rng() & 1) ? 1024 : 3068;
    const int o = s - e + static_cast<int>(rng() % 5) - 2;
    if (o > 0 && o < 2047) check(from(uint64_t(e) << 52 | (rng() & f)), from(uint64_t(o) << 52 | (rng() & f)));
  }
}

}  // namespace mulcases
