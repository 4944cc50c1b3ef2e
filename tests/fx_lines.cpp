// Host entry points of the fixed-point arithmetic (csrc/fx.cuh) for test_fixed_point.py.
#include "fx.cuh"

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
