// Host entry points of the fixed-point arithmetic (csrc/fx.cuh) for test_fixed_point.py.
#include "fx.cuh"

#include <cstring>

using namespace ib::fx;

// float-float conversion of v[i] 2^-q: first part as bits, the rest r 2^e
extern "C" void to_pair(int n, const i64* v, int q, unsigned* hi, int* r, int* e) {
  for (int i = 0; i < n; ++i) {
    const pair_float p = from_fixed_pair(v[i], q);
    hi[i] = p.hi;
    r[i] = p.r;
    e[i] = p.e;
  }
}

// x[i] in units of 2^-(kInBits + 1022 - ex)
extern "C" void to_units(int n, const double* x, int ex, i64* v) {
  for (int i = 0; i < n; ++i) {
    u64 b;
    std::memcpy(&b, x + i, 8);
    v[i] = to_fixed(b, ex);
  }
}
extern "C" int exponent(double x) {
  u64 b;
  std::memcpy(&b, &x, 8);
  return (int)(mag_hi(b) >> 20);
}
