// Block fixed-point arithmetic of the sine transforms (dstfx.cu).
//
// GB300 issues an FP64 instruction for 2 lanes per SM and clock; a 64-bit integer add runs at 54
// and a 32 x 32 + 64 multiply-add (IMAD.WIDE) at 63 (measured, independent chains on a full GPU),
// so a transform whose values are 64-bit integers on one scale per line is an order of magnitude
// cheaper in pipe time than the same transform in FP64: an add is 2 instructions, a product with a
// tabulated factor 3 multiply-adds and a rounding shift.
//
// A line of doubles becomes integers v = round(x 2^q) with q from the line's largest magnitude,
// max |v| <= 2^57.  Adds are exact.  Products with a factor w (stored as w 2^60 = h 2^30 + l, h and
// l 32-bit, |l| <= 2^29) are rounded to one unit.  Between the stages of the transform the line is
// shifted down, all of it by the same count and rounded to nearest even, only as far as its
// largest value then asks for (block floating point).  The noise of a transform is below that of
// the FP64 transform it replaces (tests/test_fixed_point.py, over lines of 8 to 2048 cells against sums in
// extended precision): its error is 0.04 to 0.18 of the FP64 one's in the mean of a kind of data, most where
// one value stands out of its line.  With inputs of 55 bits it was 0.06 to 0.45, and up to 4 times as large for
// single lines of that sort, where the rounding of the folded small values, 1 / sin(pi j / n) times as large in
// terms of the inputs, shows; with 56 up to 2.3 times.  The shifts that the two bits more ask for cost 0.5% at most
// (2048^2 solve of two fields 533 -> 536 us, eight 1024^2 x 4 FP64 steps 8473 -> 8518 us).
//
// Plain C++ (host and device), so that the arithmetic can be checked without a GPU.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD inline
#endif

namespace ib {
namespace fx {

typedef long long i64;
typedef unsigned long long u64;

struct alignas(16) cpx {
  i64 x, y;
};
// a factor w: w 2^60 = h 2^30 + l
struct wgt {
  int h, l;
};
// a complex factor
struct alignas(16) cwgt {
  int rh, rl, ih, il;
};

// Bounds that keep every intermediate in range:
//   inputs |v| <= 2^57, so the folded line (4 times the largest input) stays within 2^59, which only the middle
//   value can reach;
//   components of a stage's inputs below 2^59: a radix-8 stage sums 8 complex values, a factor
//   sqrt(1/2) meets sums below 2^61, where the split of a product's factor ends;
//   components of the FFT's result below 2^60 before the real split, which sums pairs of them;
//   the odd outputs, prefix sums bounded by the sum of the line's magnitudes, below 2^63
//   (sums of some of the differences may wrap, the outputs do not).
constexpr int kInBits = 57, kStageBits = 59, kPostBits = 60, kOutBits = 63;

// a + b of partial sums, which may wrap on the way to a sum that does not
FX_HD i64 add_wrap(i64 a, i64 b) { return (i64)((u64)a + (u64)b); }
FX_HD i64 mad(int a, int b, i64 c) { return (i64)a * b + c; }

// arithmetic shift right by d < 31 (the same on every thread of a line), rounded to nearest even
FX_HD i64 shr_rne(i64 v, int d) {
  if (d == 0) return v;
  v += (i64)(u64)(((1u << (d - 1)) - 1u) + (((unsigned)v >> d) & 1u));
#if defined(__CUDA_ARCH__)
  const int hi = (int)(v >> 32);
  return (i64)((u64)(unsigned)__funnelshift_r((unsigned)v, (unsigned)hi, d) | ((u64)(unsigned)(hi >> d) << 32));
#else
  return v >> d;
#endif
}
FX_HD i64 half_rne(i64 v) { return (v + (int)((v >> 1) & 1)) >> 1; }

// split of |v| < 2^61: v = h 2^30 + l, 0 <= l < 2^30
struct split {
  int h, l;
};
FX_HD split cut(i64 v) { return {(int)(v >> 30), (int)v & 0x3fffffff}; }

constexpr i64 kHalf30 = (i64)1 << 29;

// v w
FX_HD i64 mul(i64 v, wgt w) {
  const split s = cut(v);
  return mad(s.h, w.h, mad(s.h, w.l, mad(s.l, w.h, kHalf30)) >> 30);
}
// a u + b w
FX_HD i64 mul2(split a, wgt u, split b, wgt w) {
  const i64 lo = mad(a.h, u.l, mad(a.l, u.h, mad(b.h, w.l, mad(b.l, w.h, kHalf30)))) >> 30;
  return mad(a.h, u.h, mad(b.h, w.h, lo));
}
FX_HD cpx cmul(cpx a, cwgt w) {
  const split x = cut(a.x), y = cut(a.y);
  return {mul2(x, {w.rh, w.rl}, y, {-w.ih, -w.il}), mul2(x, {w.ih, w.il}, y, {w.rh, w.rl})};
}
FX_HD cpx add(cpx a, cpx b) { return {a.x + b.x, a.y + b.y}; }
FX_HD cpx sub(cpx a, cpx b) { return {a.x - b.x, a.y - b.y}; }
FX_HD cpx mul_mi(cpx a) { return {a.y, -a.x}; }  // -i a

// ---- small forward DFTs (e^{-2 pi i / R}) --------------------------------------------------------
constexpr wgt kSqrtHalf = {759250125, -6429112};        // sqrt(1/2)
constexpr wgt kSin60 = {929887697, -333032134};
constexpr wgt kCos72 = {331804471, 200954849}, kCos144 = {-868675383, -200954849};
constexpr wgt kSin72 = {1021189159, -500531281}, kSin144 = {631129609, -89313545};

FX_HD wgt neg(wgt w) { return {-w.h, -w.l}; }

template <int R> struct Dft;
template <> struct Dft<2> {
  FX_HD static void run(cpx* v) {
    const cpx a = v[0], b = v[1];
    v[0] = add(a, b);
    v[1] = sub(a, b);
  }
};
template <> struct Dft<4> {
  FX_HD static void run(cpx* v) {
    const cpx t0 = add(v[0], v[2]), t1 = sub(v[0], v[2]);
    const cpx t2 = add(v[1], v[3]), t3 = mul_mi(sub(v[1], v[3]));
    v[0] = add(t0, t2);
    v[2] = sub(t0, t2);
    v[1] = add(t1, t3);
    v[3] = sub(t1, t3);
  }
};
// decimation in frequency: the factors sqrt(1/2) meet sums of two inputs only (|.| <= 2 sqrt 2 in)
template <> struct Dft<8> {
  FX_HD static void run(cpx* v) {
    cpx e[4], o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      e[k] = add(v[k], v[k + 4]);
      o[k] = sub(v[k], v[k + 4]);
    }
    o[1] = {mul(o[1].x + o[1].y, kSqrtHalf), mul(o[1].y - o[1].x, kSqrtHalf)};
    o[2] = mul_mi(o[2]);
    o[3] = {mul(o[3].y - o[3].x, kSqrtHalf), mul(-o[3].x - o[3].y, kSqrtHalf)};
    Dft<4>::run(e);
    Dft<4>::run(o);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[2 * k] = e[k];
      v[2 * k + 1] = o[k];
    }
  }
};
template <> struct Dft<3> {
  FX_HD static void run(cpx* v) {
    const cpx t = add(v[1], v[2]), d = sub(v[1], v[2]);
    const cpx m = {v[0].x - half_rne(t.x), v[0].y - half_rne(t.y)};
    const cpx r = {mul(d.y, kSin60), -mul(d.x, kSin60)};  // -i sin60 (v1 - v2)
    v[0] = add(v[0], t);
    v[1] = add(m, r);
    v[2] = sub(m, r);
  }
};
// 2 x 3, coprime: no factors between
template <> struct Dft<6> {
  FX_HD static void run(cpx* v) {
    cpx a[3] = {v[0], v[2], v[4]}, b[3] = {v[3], v[5], v[1]};
    Dft<3>::run(a);
    Dft<3>::run(b);
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = (k & 1) ? sub(a[k % 3], b[k % 3]) : add(a[k % 3], b[k % 3]);
  }
};
template <> struct Dft<5> {
  FX_HD static void run(cpx* v) {
    const cpx a1 = add(v[1], v[4]), b1 = sub(v[1], v[4]), a2 = add(v[2], v[3]), b2 = sub(v[2], v[3]), z = v[0];
    const split a1x = cut(a1.x), a1y = cut(a1.y), a2x = cut(a2.x), a2y = cut(a2.y);
    const split b1x = cut(b1.x), b1y = cut(b1.y), b2x = cut(b2.x), b2y = cut(b2.y);
    const cpx r1 = {z.x + mul2(a1x, kCos72, a2x, kCos144), z.y + mul2(a1y, kCos72, a2y, kCos144)};
    const cpx r2 = {z.x + mul2(a1x, kCos144, a2x, kCos72), z.y + mul2(a1y, kCos144, a2y, kCos72)};
    // -i (sin72 b1 + sin144 b2), -i (sin144 b1 - sin72 b2)
    const cpx i1 = {mul2(b1y, kSin72, b2y, kSin144), -mul2(b1x, kSin72, b2x, kSin144)};
    const cpx i2 = {mul2(b1y, kSin144, b2y, neg(kSin72)), -mul2(b1x, kSin144, b2x, neg(kSin72))};
    v[0] = add(z, add(a1, a2));
    v[1] = add(r1, i1);
    v[4] = sub(r1, i1);
    v[2] = add(r2, i2);
    v[3] = sub(r2, i2);
  }
};

// Radices of the FFT of M points: eights where many values lie in a thread's registers (M >= 384), fours
// where lines are short; a left-over 2 makes a six with a 3, or an eight.
constexpr int kMaxRadices = 10;
struct Radices {
  int n, r[kMaxRadices];
};
constexpr Radices radices(int M) {
  Radices p{};
  int twos = 0, threes = 0, fives = 0, eights = 0, fours = 0, sixes = 0;
  const bool large = M >= 384;
  for (; M % 2 == 0; M /= 2) ++twos;
  for (; M % 3 == 0; M /= 3) ++threes;
  for (; M % 5 == 0; M /= 5) ++fives;
  const int over = large ? twos % 3 : twos % 2;  // large: twos left over by eights; else by fours
  if (over == 1 && threes > 0) {
    sixes = 1;
    --twos;
    --threes;
  }
  if (large) {
    while (twos % 3 != 0 && twos >= 2) {
      ++fours;
      twos -= 2;
    }
  } else if (twos % 2 != 0 && twos >= 3) {
    eights = 1;
    twos -= 3;
  }
  if (large) {
    eights = twos / 3;
    twos %= 3;
  } else {
    fours = twos / 2;
    twos %= 2;
  }
  for (int i = 0; i < eights; ++i) p.r[p.n++] = 8;
  for (int i = 0; i < fours; ++i) p.r[p.n++] = 4;
  for (int i = 0; i < sixes; ++i) p.r[p.n++] = 6;
  for (int i = 0; i < twos; ++i) p.r[p.n++] = 2;
  for (int i = 0; i < threes; ++i) p.r[p.n++] = 3;
  for (int i = 0; i < fives; ++i) p.r[p.n++] = 5;
  return p;
}

// ---- doubles to integers and back, on their bits -------------------------------------------------
// high word of |x|: ordered like |x| over a line, exponent in bits 20..30
FX_HD unsigned mag_hi(u64 bits) { return (unsigned)(bits >> 32) & 0x7fffffffu; }

// x 2^q rounded to nearest, q = kInBits + 1022 - ex, for |x| < 2^(ex - 1022), ex the biased exponent
// of the line's largest magnitude (at least 1): |result| <= 2^kInBits.  (Ties go away from zero: in
// magnitude, at most 2^-54 of the value.)
FX_HD i64 to_fixed(u64 bits, int ex) {
  const unsigned hi = mag_hi(bits);
  const int e = (int)(hi >> 20);
  const unsigned mh = (hi & 0xfffffu) | (e > 0 ? 0x100000u : 0u);
  const u64 m = (((u64)mh << 32) | (unsigned)bits) << 10;
  // m 2^-(63 - kInBits) is the value of the largest exponent; m < 2^63, so that nothing is left of a value below
  // half a unit however far it is shifted
  int s = 62 - kInBits + ex - (e > 0 ? e : 1);
  if (s > 63) s = 63;
  const i64 r = (i64)(((m >> s) + 1) >> 1);
  const i64 sg = (i64)bits >> 63;
  return (r ^ sg) - sg;
}

// The same for a float given by its bits, ex the biased exponent (at least 1) of the largest float of
// the line's values: x 2^q, q = kInBits + 126 - ex.
FX_HD i64 to_fixed_float(unsigned bits, int ex) {
  const int e = (int)(bits >> 23) & 255;
  const unsigned m = (bits & 0x7fffffu) | (e > 0 ? 0x800000u : 0u);
  int s = ex - (e > 0 ? e : 1);
  if (s > 63) s = 63;
  const i64 r = (i64)(((((u64)m << (kInBits - 23)) >> s) + 1) >> 1);
  const i64 sg = (i64)((int)bits >> 31);
  return (r ^ sg) - sg;
}

FX_HD int clz64(u64 v) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}

// The bits of the double nearest v 2^-q.  `safe`: every nonzero |v| < 2^63 gives a normal double
// (1 <= 1023 - q, and 1087 - q <= 2046 with a carry).
FX_HD bool safe_scale(int q) { return q <= 1022 && q >= -959; }
FX_HD u64 from_fixed(i64 v, int q) {
  const u64 sg = (u64)v & 0x8000000000000000ull;
  u64 m = v < 0 ? (u64)0 - (u64)v : (u64)v;
  const int lz = clz64(m);
  m <<= (lz & 63);
  // exponent field of the leading bit minus one: the implicit bit carries into it
  const u64 e = (u64)(unsigned)(1023 + 62 - q - lz);
  const u64 r = (e << 52) + (m >> 11) + ((m >> 10) & 1);
  return v == 0 ? 0 : (r | sg);
}

// The float-float number nearest v 2^-q: its first part as bits, the rest as an integer r times 2^e.
// Beyond the float range: zero, or infinity.
struct pair_float {
  unsigned hi;
  int r, e;
};
FX_HD pair_float from_fixed_pair(i64 v, int q) {
  const unsigned sg = (unsigned)((u64)v >> 32) & 0x80000000u;
  u64 m = v < 0 ? (u64)0 - (u64)v : (u64)v;
  const int lz = clz64(m);
  m <<= (lz & 63);
  const unsigned t = (unsigned)(m >> 40) + ((unsigned)(m >> 39) & 1u);  // 24 bits, rounded
  // what is left, in 2^8 units of m.  At a tie it is -2^31, which has no negative in an int: one unit less
  // becomes the same float
  int rem = (int)((i64)(m - ((u64)t << 40)) >> 8);
  rem = rem < -0x7fffffff ? -0x7fffffff : rem;
  const int eh = 127 + 63 - lz - q;                                     // biased exponent of the leading bit
  pair_float p;
  p.hi = sg | (eh > 254 ? 0x7f800000u : ((unsigned)(eh - 1) << 23) + t);
  p.r = eh > 254 ? 0 : (sg ? -rem : rem);
  p.e = 8 - lz - q;
  if (v == 0 || eh < 1) p = {0u, 0, 0};
  return p;
}

}  // namespace fx
}  // namespace ib
