// Host entry points of the fixed-point arithmetic (csrc/fx.cuh) for test_fixed_point.py.
#include "fx.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

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
extern "C" int input_bits() { return kInBits; }
extern "C" int exponent(double x) {
  u64 b;
  std::memcpy(&b, &x, 8);
  return (int)(mag_hi(b) >> 20);
}

// ---- a whole line: DST-I of y[0..n-2], F_k = sum_j y_j sin(pi j k / n), by the kernels' steps in sequence ----
namespace {

constexpr long double kPi = 3.141592653589793238462643383279502884L;

// The factors and the arithmetic of the two forms
struct Fixed {
  using real = i64;
  using cplx = cpx;
  using factor = cwgt;
  static wgt weight(long double w) {
    const long long v = llrintl(w * (long double)(1LL << 60));
    const int h = (int)((v + (1LL << 29)) >> 30);
    return {h, (int)(v - h * (1LL << 30))};
  }
  static factor cis(long double num, long double den) {  // e^{-2 pi i num / den}
    const long double ang = -2.0L * kPi * num / den;
    const wgt c = weight(cosl(ang)), s = weight(sinl(ang));
    return {c.h, c.l, s.h, s.l};
  }
  static i64 times(i64 v, long double w) { return mul(v, weight(w)); }
  static cpx times(cpx v, factor w) { return cmul(v, w); }
  template <int R> static void dft(cpx* v) { Dft<R>::run(v); }
};
struct Double {
  using real = double;
  struct cplx { double x, y; };
  using factor = cplx;
  static factor cis(long double num, long double den) {
    return {(double)cosl(-2.0L * kPi * num / den), (double)sinl(-2.0L * kPi * num / den)};
  }
  static double times(double v, long double w) { return v * (double)w; }
  static cplx times(cplx v, factor w) { return {v.x * w.x - v.y * w.y, v.x * w.y + v.y * w.x}; }
  template <int R> static void dft(cplx* v) {
    cplx o[R];
    for (int k = 0; k < R; ++k) {
      o[k] = v[0];
      for (int r = 1; r < R; ++r) {
        const cplx t = times(v[r], cis(r * k % R, R));
        o[k] = {o[k].x + t.x, o[k].y + t.y};
      }
    }
    for (int k = 0; k < R; ++k) v[k] = o[k];
  }
};

int bits_of(i64 v) {
  int b = 0;
  for (u64 m = (u64)(v < 0 ? ~v : v); m; m >>= 1) ++b;
  return b;
}
void shift(cpx* z, int M, int d) {
  for (int i = 0; i < M; ++i) z[i] = {shr_rne(z[i].x, d), shr_rne(z[i].y, d)};
}
int excess(const cpx* z, int M, int limit) {
  int b = 0;
  for (int i = 0; i < M; ++i) b = std::max(b, std::max(bits_of(z[i].x), bits_of(z[i].y)));
  return std::max(0, b - limit);
}

// FFT of M = product of the radices; shifts: of the fixed form
template <class A>
void fft(std::vector<typename A::cplx>& z, int M, int& shifts) {
  using C = typename A::cplx;
  const Radices p = radices(M);
  std::vector<C> out(M);
  int ns = 1;
  for (int st = 0; st < p.n; ++st) {
    const int R = p.r[st], nb = M / R;
    if constexpr (std::is_same<A, Fixed>::value) {
      const int d = st ? excess(z.data(), M, kStageBits) : 0;
      shifts += d;
      shift(z.data(), M, d);
    }
    for (int j = 0; j < nb; ++j) {
      const int k = j % ns;
      C v[8];
      for (int r = 0; r < R; ++r) {
        v[r] = z[j + r * nb];
        if (r && ns > 1) v[r] = A::times(v[r], A::cis(r * k, ns * R));
      }
      if (R == 8) A::template dft<8>(v);
      else if (R == 4) A::template dft<4>(v);
      else if (R == 6) A::template dft<6>(v);
      else if (R == 5) A::template dft<5>(v);
      else if (R == 3) A::template dft<3>(v);
      else A::template dft<2>(v);
      for (int r = 0; r < R; ++r) out[(j - k) * R + k + r * ns] = v[r];
    }
    z.swap(out);
    ns *= R;
  }
}

}  // namespace

extern "C" void line_fixed(int n, const double* y, double* F) {
  const int M = n / 2, hM = M / 2;
  std::vector<u64> b(n - 1);
  std::memcpy(b.data(), y, sizeof(double) * (n - 1));
  unsigned m = 0;
  for (u64 x : b) m = std::max(m, mag_hi(x));
  const int ex = std::max(1, (int)(m >> 20));
  std::vector<i64> u(n);
  unsigned asum = 0;
  for (int j = 0; j < M; ++j) {
    const i64 va = to_fixed(b[(j ? j : M) - 1], ex), vb = j ? to_fixed(b[n - j - 1], ex) : 0;
    asum += ((unsigned)((int)(va >> 32) ^ (int)(va >> 63)) >> (kInBits - 52)) + ((unsigned)((int)(vb >> 32) ^ (int)(vb >> 63)) >> (kInBits - 52)) + 2u;
    if (j == 0) {
      u[0] = 0;
      u[M] = 4 * va;
      continue;
    }
    const i64 p = Fixed::times(va + vb, 2.0L * sinl(kPi * (long double)j / (long double)n));
    u[j] = p + (va - vb);
    u[n - j] = p - (va - vb);
  }
  std::vector<cpx> z(M);
  for (int i = 0; i < M; ++i) z[i] = {u[2 * i], u[2 * i + 1]};
  int shifts = 0;
  fft<Fixed>(z, M, shifts);
  int sum_bits = kInBits - 18;
  for (unsigned t = asum - 1u; t; t >>= 1) ++sum_bits;
  const int d = std::max(excess(z.data(), M, kPostBits), sum_bits - kOutBits - shifts);
  shifts += d;
  if (d > 0) shift(z.data(), M, d);
  std::vector<i64> D(M), E(M + 1);
  D[0] = z[0].x + z[0].y;
  D[hM] = 2 * z[hM].x;
  E[hM] = 2 * z[hM].y;
  for (int k = 1; k < hM; ++k) {
    const cpx a = z[k], c = z[M - k];
    const i64 er = a.x + c.x, ei = a.y - c.y;
    const cpx r = cmul({a.y + c.y, c.x - a.x}, Fixed::cis(k, n));
    D[k] = er + r.x;
    D[M - k] = er - r.x;
    E[k] = -(ei + r.y);
    E[M - k] = ei - r.y;
  }
  const int q = kInBits + 1022 - ex - shifts + 2;
  auto value = [&](i64 v) {
    const u64 o = from_fixed(v, q);
    double x;
    std::memcpy(&x, &o, 8);
    return x;
  };
  // prefix sums of D: within chunks of 8, of the chunks' totals by doubling, both together
  const int chunks = (M + 7) / 8;
  std::vector<i64> total(chunks);
  for (int k = 0; k < M; ++k) {
    if (k % 8) D[k] = add_wrap(D[k - 1], D[k]);
    total[k / 8] = D[k];
  }
  for (int w = 1; w < chunks; w <<= 1)
    for (int t = chunks - 1; t >= w; --t) total[t] = add_wrap(total[t], total[t - w]);
  for (int k = 0; k < M; ++k) {
    F[2 * k] = value(k < 8 ? D[k] : add_wrap(D[k], total[k / 8 - 1]));
    if (k) F[2 * k - 1] = value(E[k]);
  }
}

// RODFT00 of a field of (ny - 1) x (nx - 1) values by such lines: 4 times both transforms
extern "C" void dst2_fixed(int nx, int ny, const double* in, double* out) {
  const int ncol = nx - 1, nrow = ny - 1;
  std::vector<double> w((size_t)ncol * nrow), line(ncol + 1), col(nrow), res(nrow + 1);
  for (int J = 0; J < nrow; ++J) {
    line_fixed(nx, in + (size_t)J * ncol, line.data());
    for (int I = 0; I < ncol; ++I) w[(size_t)I * nrow + J] = line[I];
  }
  for (int I = 0; I < ncol; ++I) {
    line_fixed(ny, w.data() + (size_t)I * nrow, res.data());
    for (int J = 0; J < nrow; ++J) out[(size_t)J * ncol + I] = 4.0 * res[J];
  }
}

// the same steps in FP64, prefix sums compensated
extern "C" void line_double(int n, const double* y, double* F) {
  const int M = n / 2, hM = M / 2;
  std::vector<Double::cplx> z(M);
  std::vector<double> u(n);
  u[M] = 2 * y[M - 1];
  for (int j = 1; j < M; ++j) {
    const double p = Double::times(y[j - 1] + y[n - j - 1], sinl(kPi * j / n)), df = 0.5 * (y[j - 1] - y[n - j - 1]);
    u[j] = p + df;
    u[n - j] = p - df;
  }
  for (int i = 0; i < M; ++i) z[i] = {u[2 * i], u[2 * i + 1]};
  int none = 0;
  fft<Double>(z, M, none);
  std::vector<double> D(M);
  D[0] = 0.5 * (z[0].x + z[0].y);
  D[hM] = z[hM].x;
  F[2 * hM - 1] = z[hM].y;
  for (int k = 1; k < hM; ++k) {
    const Double::cplx a = z[k], c = z[M - k];
    const double er = 0.5 * (a.x + c.x), ei = 0.5 * (a.y - c.y);
    const Double::cplx r = Double::times({0.5 * (a.y + c.y), 0.5 * (c.x - a.x)}, Double::cis(k, n));
    D[k] = er + r.x;
    D[M - k] = er - r.x;
    F[2 * k - 1] = -(ei + r.y);
    F[2 * (M - k) - 1] = ei - r.y;
  }
  double s = 0, c = 0;
  for (int k = 0; k < M; ++k) {
    const double t = D[k] - c, v = s + t;
    c = (v - s) - t;
    s = v;
    F[2 * k] = s;
  }
}

// relative errors (2-norm) of the two against the sums in extended precision
extern "C" void line_errors(int n, const double* y, double* fixed, double* dbl) {
  std::vector<long double> sn(2 * n);
  for (int i = 0; i < 2 * n; ++i) {
    const int a = i % n, m = std::min(a, n - a);
    sn[i] = (i < n ? 1 : -1) * sinl(kPi * m / n);
  }
  std::vector<double> f(n), g(n);
  line_fixed(n, y, f.data());
  line_double(n, y, g.data());
  long double ef = 0, eg = 0, ss = 0;
  for (int k = 1; k < n; ++k) {
    long double s = 0;
    int a = 0;
    for (int j = 1; j < n; ++j) {
      a += k;
      if (a >= 2 * n) a -= 2 * n;
      if (y[j - 1] != 0) s += y[j - 1] * sn[a];
    }
    ef += (f[k - 1] - s) * (f[k - 1] - s);
    eg += (g[k - 1] - s) * (g[k - 1] - s);
    ss += s * s;
  }
  *fixed = (double)sqrtl(ef / ss);
  *dbl = (double)sqrtl(eg / ss);
}
