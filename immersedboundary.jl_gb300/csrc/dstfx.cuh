// The kernels of the FP64 and float-float sine-transform passes (launched by dstfx.cu): every line is
// transformed in 64-bit block fixed point (fx.cuh).
//
// Replaces, like dst.cu, the FFTW RODFT00 plan + `LaplacianInv` call of the reference
// (src/streamfcn/fluid-ops.jl:19-56) and the CN multipliers of `A_Ainv_linearmaps`
// (src/streamfcn/cnab/ops.jl:14-42).  The algorithm of a line is dst.cu's (fold, half-length complex
// FFT, split of the real transform, prefix sum of the differences); its values are integers.
//
// A group of NT threads (32, 64 or 128, by the axis length: M = n/2 <= PP NT) owns a line:
//   1. each thread loads the pairs (y_j, y_{n-j}) of j = t + NT i straight into registers, the group
//      finds the line's largest exponent and turns the pairs into folded integers in shared memory
//   2. Stockham stages of radix 8, 4, 2, 3, 5: read, group barrier, shift + twiddle + DFT in
//      registers, write in place; the bits the results occupy (one OR per value) give the next
//      stage's shift.  Complex values are padded one slot in eight
//   3. split into even outputs and differences D_k; the odd outputs are D's exact prefix sums
//   4. doubles (or float-float pairs) leave by their bits (leading-zero count, round, pack)
// A line with an infinity or NaN becomes NaN throughout, as the FP64 transform made it.  Sums of
// integers do not depend on their order, so results are the same bits for any NT.
//
// A pass reads its lines as they lie in memory and stores them transposed (the forward x pass, the y
// pass), so that the next pass's lines lie in memory: 32 or 64 bytes at a time, written without
// waiting, where a transposing load would stall the block.
//
// What bounds it: the integer pipes (ncu, 1024-cell lines: ALU 60% and FMA-heavy 45% busy, an instruction
// issued in 59% of cycles, waits mostly for a busy pipe), and the latency of a line's chain where
// a launch has few lines.  Measured against the FP64-arithmetic passes (shared-memory Stockham, one
// warp per line at 2048 cells), which the FP64 pipe's two lanes per SM bound: a 2048^2 Poisson call
// on two fields 2.09 -> 0.54 ms with a tenth of the error (1.6e-15 against 2.2e-14); steps by these
// passes alone: 1024^2 x 4 3.75 -> 1.16 ms, 384 x 256 x 4 RKC 0.88 -> 0.40, 200^2 x 5 0.81 -> 0.39, 128^2 x
// 3 0.53 -> 0.28.
#pragma once

#include "fx.cuh"
#include "ib_common.cuh"

namespace ib {

namespace fxp {

using fx::cpx;
using fx::cwgt;
using fx::i64;
using fx::Radices;
using fx::radices;
using fx::u64;
using fx::wgt;

static_assert(fx::kMaxRadices == kMaxStages, "a stage per radix");
constexpr unsigned kAll = 0xffffffffu;
constexpr int kRedSlots = 2 + kMaxStages;  // reductions of one transform: largest, sum, one per stage

// padded index of a complex value / of a result: one spare slot after every 8
__host__ __device__ constexpr int cpad(int i) { return i + (i >> 3); }

// The results F_i, i = 1..n-1, of a line lie at word cpad(i / 2) of two regions of its buffer, the
// odd ones in the first, the even ones in the second, 8 banks (of 8 bytes) away from the first.
__host__ __device__ constexpr int even_off(int M) { return (M + (M >> 3) + 6 + 7) / 16 * 16 + 8; }
// 8-byte words of one line's buffer: M complex values padded, or both regions; congruent to 2 mod 16,
// so that four lines' words at two successive indices of either parity lie in different banks
__host__ __device__ constexpr int line_words(int M) { return (even_off(M) + cpad(M) + 14) / 16 * 16 + 2; }

// Every accepted length is compiled in (M = n / 2: even, with factors 2, 3 and 5, at most 1024), so
// that index arithmetic is constant: a 200^2 solve 22.8 -> 19.6 us, 600 x 400 38.4 -> 29.1.
//
// Threads of a line's group: the fewest warps that hold it eight pairs a thread at most, and two from
// M = 129 on, where a launch still lasts as long as a line's chain.  Measured, a Poisson solve of one
// field: 512^2 with 64 threads a line and four pairs each 23.1 us, 32 and eight 27.9; 768 x 512 with 64
// and six (x) 30.8, 128 and three 34.5; 1024^2 with 64 and eight 54.5, 128 and four 64.7.
constexpr int group_threads(int M) { return M <= 128 ? 32 : M <= 512 ? 64 : 128; }
constexpr int pairs(int M) { return (M + group_threads(M) - 1) / group_threads(M); }

// barrier of a line's group of threads
template <int NT>
__device__ __forceinline__ void group_bar(int id) {
  if (NT == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "r"(NT) : "memory");
}

template <int NT>
struct Group {
  int t;          // thread in the group
  int id;         // group in the block (barrier id + 1)
  i64* buf;       // the line's buffer
  unsigned* red;  // [kRedSlots][NT / 32]

  __device__ __forceinline__ void bar() const { group_bar<NT>(id); }
  __device__ __forceinline__ void put(int slot, unsigned v) const {  // v: warp-reduced already
    if (NT > 32 && (t & 31) == 0) red[slot * (NT / 32) + (t >> 5)] = v;
  }
  template <class Op>
  __device__ __forceinline__ unsigned get(int slot, unsigned v, Op op) const {
    if (NT == 32) return v;
    unsigned m = red[slot * (NT / 32)];
#pragma unroll
    for (int w = 1; w < NT / 32; ++w) m = op(m, red[slot * (NT / 32) + w]);
    return m;
  }
};

__device__ __forceinline__ unsigned occupied(i64 v) {
  const int h = (int)(v >> 32);
  return (unsigned)(h ^ (h >> 31));
}

// One Stockham stage of radix R, in place, by the threads of a group; NS: product of the radices before.
// The first stage (NS = 1) reads the folded line in its natural layout.  Returns the OR of the bits
// this thread's results occupy.
template <int M, int R, int NS>
__device__ __forceinline__ unsigned stage(const Group<group_threads(M)>& G, const FxAxis& ax, int st, int d) {
  constexpr int NT = group_threads(M), nb = M / R, NB = (nb + NT - 1) / NT;  // butterflies in all, per thread
  constexpr bool kFull = nb % NT == 0;
  const int t = G.t;
  cpx* z = reinterpret_cast<cpx*>(G.buf);
  cpx v[NB][R];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int j = t + NT * b;
    if (!kFull) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[b][r] = {0, 0};  // (a predicated load alone would keep the old value live)
    }
    if (kFull || j < nb) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (NS == 1) v[b][r] = z[j + r * nb];
        else if (nb % 8 == 0) v[b][r] = z[cpad(t) + b * (NT + NT / 8) + r * (nb + nb / 8)];
        else v[b][r] = z[cpad(j + r * nb)];
      }
    }
  }
  G.bar();
  unsigned o = 0;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int j = t + NT * b;
    if (kFull || j < nb) {
      const int k = j % NS;
      if (NS > 1) {
        if (d > 0) {
#pragma unroll
          for (int r = 0; r < R; ++r) v[b][r] = {fx::shr_rne(v[b][r].x, d), fx::shr_rne(v[b][r].y, d)};
        }
        const cwgt* tw = ax.tw + ax.twoff[st] + k;
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const int4 w = __ldg(reinterpret_cast<const int4*>(tw + (r - 1) * NS));
          v[b][r] = fx::cmul(v[b][r], {w.x, w.y, w.z, w.w});
        }
      }
      fx::Dft<R>::run(v[b]);
      const int base = (j - k) * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        o |= occupied(v[b][r].x) | occupied(v[b][r].y);
        if (NS % 8 == 0 || (NS == 1 && R == 8)) z[cpad(base) + (NS == 1 ? r : r * (NS + NS / 8))] = v[b][r];
        else z[cpad(base + r * NS)] = v[b][r];
      }
    }
  }
  return o;
}

// Shift the values now need (bits from the OR of occupied()) to fit `limit` bits.
__device__ __forceinline__ int excess(unsigned o, int limit) { return max(0, 64 - __clz((int)o) - limit); }

// The stages ST.. of the transform; T: the shifts so far, o: the bits the values occupy.
template <int M, int ST, int NS>
__device__ __forceinline__ void stages(const Group<group_threads(M)>& G, const FxAxis& ax, int& T, unsigned& o) {
  constexpr Radices p = radices(M);
  if constexpr (ST < p.n) {
    constexpr int R = p.r[ST];
    const int d = ST > 0 ? excess(o, fx::kStageBits) : 0;
    T += d;
    o = __reduce_or_sync(kAll, stage<M, R, NS>(G, ax, ST, d));
    G.put(2 + ST, o);
    G.bar();
    o = G.get(2 + ST, o, [](unsigned a, unsigned b) { return a | b; });
    stages<M, ST + 1, NS * R>(G, ax, T, o);
  }
}

__device__ __forceinline__ i64* result_at(i64* buf, int M, int i) {
  return buf + ((i & 1) ? 0 : even_off(M)) + cpad(i >> 1);
}
// The words of a thread's pairs (j, n - j), j = t + NT i: at lo + i kStride and hi - i kStride (the
// pair j = 0 stands for the middle value, j = n / 2, alone).
template <int M>
struct Pairs {
  static constexpr int NT = group_threads(M), kStride = NT / 2 + NT / 16;
  i64 *lo, *hi, *mid;
  __device__ __forceinline__ Pairs(i64* buf, int t) {
    lo = buf + ((t & 1) ? 0 : even_off(M)) + cpad(t >> 1);
    hi = buf + ((t & 1) ? 0 : even_off(M)) + cpad(M - ((t + 1) >> 1));
    mid = result_at(buf, M, M);
  }
  __device__ __forceinline__ i64* a(int i, bool middle) const { return middle ? mid : lo + i * kStride; }
  __device__ __forceinline__ i64* b(int i) const { return hi - i * kStride; }
};

// exponent of a line whose values are not finite
constexpr int kNotFinite = 1 << 20;

// the double of a result on a safe scale q
__device__ __forceinline__ double to_double(i64 v, int q) {
  return __longlong_as_double((i64)fx::from_fixed(v, q));
}
__device__ __forceinline__ df64 to_pair(i64 v, int q) {
  const fx::pair_float p = fx::from_fixed_pair(v, q);
  // r 2^e in two factors where the power alone is below the float range
  const int e = 127 + p.e, k = e < 1 ? 100 : 0;
  float lo = __int2float_rn(p.r) * __uint_as_float((unsigned)max(e + k, 0) << 23);
  if (k) lo *= 0x1p-100f;
  return df64(__uint_as_float(p.hi), lo);
}
// not finite, or at the ends of the exponent range (subnormal results, or overflow)
static __device__ __noinline__ double to_double_slow(i64 v, int q) {
  if (q == kNotFinite) return __longlong_as_double(0x7ff8000000000000ll);
  return ldexp((double)v, -q);
}
// What a line's values are: doubles, or float-float pairs (the state of the mixed-precision path).
template <typename T> struct Value;
template <> struct Value<double> {
  static constexpr unsigned kBad = 0x7ff00000u;          // magnitude of an infinity or NaN
  static constexpr int kExpBit = 20, kScale = fx::kInBits + 1022;
  static __device__ __forceinline__ unsigned mag(double x) { return fx::mag_hi((u64)__double_as_longlong(x)); }
  static __device__ __forceinline__ i64 fixed(double x, int ex) { return fx::to_fixed((u64)__double_as_longlong(x), ex); }
};
template <> struct Value<df64> {
  static constexpr unsigned kBad = 0x7f800000u;
  static constexpr int kExpBit = 23, kScale = fx::kInBits + 126;
  static __device__ __forceinline__ unsigned mag(df64 x) {
    return max(__float_as_uint(x.hi) & 0x7fffffffu, __float_as_uint(x.lo) & 0x7fffffffu);
  }
  static __device__ __forceinline__ i64 fixed(df64 x, int ex) {
    return fx::to_fixed_float(__float_as_uint(x.hi), ex) + fx::to_fixed_float(__float_as_uint(x.lo), ex);
  }
};

// DST-I of a line given as pairs a[i] = y_j, b[i] = y_{n-j}, j = t + NT i (j = 0: a = y_{n/2}, b
// unused); the results are in place after the closing barrier.  Returns their scale q
// (F = value 2^-q), the same on every thread of the group.  `before_scan` runs before the last
// phase, with few registers in use: a place for loads that are needed next.
template <int M, typename T, class Hook>
__device__ __forceinline__ int line_transform(const Group<group_threads(M)>& G, const FxAxis& ax,
                                              const T (&a)[pairs(M)], const T (&b)[pairs(M)], Hook before_scan) {
  using V = Value<T>;
  constexpr int NT = group_threads(M), PP = pairs(M), n = 2 * M;
  constexpr bool kEven = M == NT * PP;  // every thread has PP pairs
  const int t = G.t;
  // 1. the line's largest exponent
  unsigned m = 0;
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    m = max(m, max(V::mag(a[i]), V::mag(b[i])));
  }
  m = __reduce_max_sync(kAll, m);
  G.put(0, m);
  G.bar();
  m = G.get(0, m, [](unsigned x, unsigned y) { return max(x, y); });
  if (m >= V::kBad) {
    G.bar();
    return kNotFinite;
  }
  const int ex = max(1, (int)(m >> V::kExpBit));
  // 2. integers, folded
  unsigned asum = 0;
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    const int j = t + NT * i;
    if (kEven || j < M) {
      const i64 va = V::fixed(a[i], ex), vb = V::fixed(b[i], ex);
      // upper bound of |va| + |vb| in units of 2^(kInBits - 20)
      asum += ((unsigned)((int)(va >> 32) ^ (int)(va >> 63)) >> (fx::kInBits - 52)) +
              ((unsigned)((int)(vb >> 32) ^ (int)(vb >> 63)) >> (fx::kInBits - 52)) + 2u;
      const int2 w = __ldg(reinterpret_cast<const int2*>(ax.sin2 + j));
      const i64 p = fx::mul(va + vb, {w.x, w.y}), df = va - vb;
      if (i == 0 && t == 0) {
        G.buf[0] = 0;
        G.buf[M] = 4 * va;
      } else {
        G.buf[j] = p + df;
        G.buf[n - j] = p - df;
      }
    }
  }
  asum = __reduce_add_sync(kAll, asum);
  G.put(1, asum);
  G.bar();
  asum = G.get(1, asum, [](unsigned x, unsigned y) { return x + y; });
  // 3. FFT of length M
  int shifts = 0;
  unsigned o = 0;
  stages<M, 0, 1>(G, ax, shifts, o);
  // 4. split: even outputs and differences, at four times their value
  const int abits = fx::kInBits - 18 + 32 - __clz((int)(asum - 1u));  // 4 sum |y| <= 2^abits
  const int d = max(excess(o, fx::kPostBits), abits - fx::kOutBits - shifts);
  shifts += d;
  {
    constexpr int hM = M / 2, PQ = (hM + NT - 1) / NT;
    constexpr bool kAllK = hM == NT * PQ;  // exactly PQ values of k per thread
    const cpx* z = reinterpret_cast<const cpx*>(G.buf);
    cpx zk[PQ], zm[PQ];
#pragma unroll
    for (int i = 0; i < PQ; ++i) {
      const int k = t + NT * i;
      if (!kAllK) zk[i] = zm[i] = {0, 0};
      if (kAllK || k < hM) {
        zk[i] = z[cpad(t) + i * (NT + NT / 8)];
        zm[i] = z[i == 0 && t == 0 ? cpad(hM) : cpad(M - t) - i * (NT + NT / 8)];
      }
    }
    G.bar();
    i64* D = G.buf;
    i64* E = G.buf + even_off(M);
#pragma unroll
    for (int i = 0; i < PQ; ++i) {
      const int k = t + NT * i;
      if (kAllK || k < hM) {
        if (d > 0) {
          zk[i] = {fx::shr_rne(zk[i].x, d), fx::shr_rne(zk[i].y, d)};
          zm[i] = {fx::shr_rne(zm[i].x, d), fx::shr_rne(zm[i].y, d)};
        }
        if (i == 0 && t == 0) {
          D[0] = zk[i].x + zk[i].y;
          D[cpad(hM)] = 2 * zm[i].x;
          E[cpad(hM)] = 2 * zm[i].y;
        } else {
          const int4 w = __ldg(reinterpret_cast<const int4*>(ax.post + k));
          const i64 er = zk[i].x + zm[i].x, ei = zk[i].y - zm[i].y;
          const cpx r = fx::cmul({zk[i].y + zm[i].y, zm[i].x - zk[i].x}, {w.x, w.y, w.z, w.w});
          const int pk = cpad(t) + i * (NT + NT / 8), pm = cpad(M - t) - i * (NT + NT / 8);
          D[pk] = er + r.x;
          D[pm] = er - r.x;
          E[pk] = -(ei + r.y);
          E[pm] = ei - r.y;
        }
      }
    }
  }
  G.bar();
  before_scan();
  // 5. odd outputs: prefix sums of D, chunk by chunk
  {
    const int k0 = t * PP;
    i64 s[PP], acc = 0;
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      if (kEven || k0 + i < M) acc = fx::add_wrap(acc, G.buf[8 % PP == 0 ? cpad(k0) + i : cpad(k0 + i)]);
      s[i] = acc;
    }
    i64 incl = acc;
#pragma unroll
    for (int w = 1; w < 32; w <<= 1) {
      const i64 v = __shfl_up_sync(kAll, incl, w);
      if ((t & 31) >= w) incl = fx::add_wrap(incl, v);
    }
    i64 excl = (i64)((fx::u64)incl - (fx::u64)acc);
    if (NT > 32) {
      // totals of the warps before this one (spare words after the padded differences)
      i64* tot = G.buf + M + (M >> 3) + 2;
      if ((t & 31) == 31) tot[t >> 5] = incl;
      G.bar();
#pragma unroll
      for (int w = 0; w < NT / 32 - 1; ++w)
        if ((t >> 5) > w) excl = fx::add_wrap(excl, tot[w]);
    }
#pragma unroll
    for (int i = 0; i < PP; ++i)
      if (kEven || k0 + i < M) G.buf[8 % PP == 0 ? cpad(k0) + i : cpad(k0 + i)] = fx::add_wrap(s[i], excl);
  }
  G.bar();
  return V::kScale - ex - shifts + 2;
}

// ------------------------------------------------------------------------------------------------
// passes
// ------------------------------------------------------------------------------------------------
// Lines per block: 4 (stores of 32-byte segments), or 2 of the longest.  Two blocks of 256 threads per
// SM or four of 128 leave 128 registers a thread; capping at 80 or 64 for more warps costs more in
// spills than it hides (1024^2 solve of one field: 54.5 us, 57.7, 62.2).
template <int M>
struct Bounds {
  static constexpr int NT = group_threads(M);
  static constexpr int kLines = NT == 128 ? 2 : 4;
  static constexpr int kThreads = kLines * NT;
  static constexpr int kBlocks = 512 / kThreads;
};

struct Smem {
  i64* line;      // this group's line buffer
  i64* lines;     // line buffer of group 0
  unsigned* red;  // this group's reduction slots
  int* q;         // [lines per block] scales
};
template <int M>
constexpr size_t smem_bytes() {
  return (size_t)Bounds<M>::kLines * (line_words(M) * 8 + kRedSlots * (group_threads(M) / 32) * 4 + 4) + 16;
}
template <int M>
__device__ __forceinline__ Smem carve(int grp) {
  constexpr int NT = group_threads(M), lpb = Bounds<M>::kLines;
  extern __shared__ __align__(16) unsigned char fx_smem[];
  Smem s;
  s.lines = reinterpret_cast<i64*>(fx_smem);
  s.line = s.lines + (size_t)grp * line_words(M);
  unsigned* red = reinterpret_cast<unsigned*>(s.lines + (size_t)lpb * line_words(M));
  s.red = red + grp * (kRedSlots * (NT / 32));
  s.q = reinterpret_cast<int*>(red + lpb * (kRedSlots * (NT / 32)));
  return s;
}

// pairs of a line that lies contiguously in memory
template <int M, typename T>
__device__ __forceinline__ void load_pairs(const T* src, int t, T (&u)[pairs(M)], T (&v)[pairs(M)]) {
  constexpr int NT = group_threads(M), PP = pairs(M);
  const T* lo = src - 1 + t;
  const T* hi = src + 2 * M - 1 - t;
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    const bool mid = i == 0 && t == 0;
    u[i] = v[i] = T(0.0f);
    if (M == NT * PP || t + NT * i < M) {
      u[i] = *(mid ? src + M - 1 : lo + NT * i);
      if (!mid) v[i] = hi[-NT * i];
    }
  }
}

// f(i, middle, F_j, F_{n-j}) for the thread's pairs (of the middle pair only the first value)
template <int M, typename T, class F>
__device__ __forceinline__ void with_results(const Pairs<M>& w, int t, int q, F f) {
  constexpr int NT = group_threads(M), PP = pairs(M);
  if constexpr (is_df64<T>::value) {
    const bool bad = q == kNotFinite;
    const df64 nan = df64(__uint_as_float(0x7fc00000u), __uint_as_float(0x7fc00000u));
#pragma unroll
    for (int i = 0; i < PP; ++i)
      if (M == NT * PP || t + NT * i < M) {
        const bool mid = i == 0 && t == 0;
        f(i, mid, bad ? nan : to_pair(*w.a(i, mid), q), bad ? nan : to_pair(*w.b(i), q));
      }
  } else if (fx::safe_scale(q)) {
#pragma unroll
    for (int i = 0; i < PP; ++i)
      if (M == NT * PP || t + NT * i < M) {
        const bool mid = i == 0 && t == 0;
        f(i, mid, to_double(*w.a(i, mid), q), to_double(*w.b(i), q));
      }
  } else {
#pragma unroll
    for (int i = 0; i < PP; ++i)
      if (M == NT * PP || t + NT * i < M) {
        const bool mid = i == 0 && t == 0;
        f(i, mid, to_double_slow(*w.a(i, mid), q), to_double_slow(*w.b(i), q));
      }
  }
}

// The results of the block's lines line0 .. line0 + lpb - 1 (of `total`, `per` lines to an array of
// `stride` values), transposed: the block's lines at one index are adjacent in memory.
template <int M>
__device__ __forceinline__ void store_transposed(const Smem& sm, int line0, int total, int per, int64_t stride,
                                                 double* out) {
  constexpr int NT = group_threads(M), lpb = Bounds<M>::kLines;
  __syncthreads();
  const int b0 = line0 / per, J0 = line0 - b0 * per, w = threadIdx.x % lpb;
  if (line0 + w >= total) return;
  const int wrap = J0 + w >= per;
  i64* buf = sm.lines + (size_t)w * line_words(M);
  const int q = sm.q[w];
  double* dst = out + (int64_t)(b0 + wrap) * stride + (J0 + w - (wrap ? per : 0));
  if (fx::safe_scale(q)) {
    // (NT indices on, the same parity: a constant step in the buffer)
    const int I0 = threadIdx.x / lpb;
    const i64* r = result_at(buf, M, I0 + 1);
    dst += (int64_t)I0 * per;
    const int64_t step = (int64_t)NT * per;
#pragma unroll 8
    for (int I = I0; I < 2 * M - 1; I += NT, r += Pairs<M>::kStride, dst += step) *dst = to_double(*r, q);
  } else {
#pragma unroll 1
    for (int I = threadIdx.x / lpb; I < 2 * M - 1; I += NT)
      dst[(int64_t)I * per] = to_double_slow(*result_at(buf, M, I + 1), q);
  }
}

// x transform of rows as they lie in memory -> transposed intermediate; optional apply_bc(bc) on the
// edges (fluid-ops.jl:249-275)
template <int M, typename T>
__global__ void __launch_bounds__(Bounds<M>::kThreads, Bounds<M>::kBlocks)
k_fx_fwd(Geometry g, FxAxis ax, const T* __restrict__ in, double* __restrict__ out, int batch,
         const T* __restrict__ bc) {
  pdl_begin();
  constexpr int NT = group_threads(M), PP = pairs(M), lpb = Bounds<M>::kLines;
  const int grp = threadIdx.x / NT;
  const Smem sm = carve<M>(grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int ncol = 2 * M - 1, nrow = g.ny - 1, total = batch * nrow;
  const int row0 = blockIdx.x * lpb, row = row0 + grp;
  if (row < total) {
    const int b = row / nrow, J = row - b * nrow;
    T u[PP], v[PP];
    load_pairs<M>(in + (int64_t)b * g.nG + (int64_t)J * ncol, G.t, u, v);
    if (bc) {
      const T* r = bc + (int64_t)b * g.nbc;
      if (J == 0 || J == nrow - 1) {
        T e[PP], f[PP];
        load_pairs<M>(r + (J == 0 ? g.B : g.T) + 1, G.t, e, f);
#pragma unroll
        for (int i = 0; i < PP; ++i) {
          u[i] += e[i];
          v[i] += f[i];
        }
      }
      if (G.t == 1) {  // the pair of the row's first and last value
        u[0] += r[g.L + 1 + J];
        v[0] += r[g.R + 1 + J];
      }
    }
    const int q = line_transform<M>(G, ax, u, v, [] {});
    if (G.t == 0) sm.q[grp] = q;
  }
  store_transposed<M>(sm, row0, total, nrow, g.nG, out);
}

// y pass: columns of the transposed intermediate, S_y, times m, S_y (or S_y only), times 2^log2scale,
// stored row-major
template <int M>
__global__ void __launch_bounds__(Bounds<M>::kThreads, Bounds<M>::kBlocks)
k_fx_y(Geometry g, FxAxis ax, const double* __restrict__ in, double* __restrict__ out, int batch,
       const double* mult, int64_t mstride, int log2scale) {
  pdl_begin();
  constexpr int NT = group_threads(M), PP = pairs(M), lpb = Bounds<M>::kLines;
  const int grp = threadIdx.x / NT;
  const Smem sm = carve<M>(grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int ncol = g.nx - 1, nrow = 2 * M - 1, total = batch * ncol;
  const int col0 = blockIdx.x * lpb, col = col0 + grp;
  if (col < total) {
    const int b = col / ncol, I = col - b * ncol, t = G.t;
    const Pairs<M> w(G.buf, t);
    const double* m = mult ? mult + (int64_t)b * mstride + (int64_t)I * nrow : nullptr;
    double u[PP], v[PP];
    load_pairs<M>(in + (int64_t)b * g.nG + (int64_t)I * nrow, t, u, v);
    int q;
    // (one copy of the transform's code: two would not fit the instruction cache)
#pragma unroll 1
    for (int pass = 0;; ++pass) {
      const bool more = pass == 0 && m;
      q = line_transform<M>(G, ax, u, v, [&] {
        if (more) load_pairs<M>(m, t, u, v);
      });
      if (!more) break;
      with_results<M, double>(w, t, q, [&](int i, bool mid, double x, double y) {
        u[i] *= x;
        v[i] = mid ? 0.0 : v[i] * y;
      });
    }
    if (G.t == 0) sm.q[grp] = q - (q == kNotFinite ? 0 : log2scale);
  }
  store_transposed<M>(sm, col0, total, ncol, g.nG, out);
}

// Vort2Flux of all levels at once (v2f.cu), first y pass: columns of the transposed intermediate in
// place, S_y times m; and the spectrum's sums for the two quarter rows,
// qrow[b-1][s][I] = sum_j sin(pi j J_s / ny) spec[I][j], J_s = ny/4, 3ny/4 (arrays qls values apart), for
// every level but the finest, whose lines no ring is made of.
template <int M>
__global__ void __launch_bounds__(Bounds<M>::kThreads, Bounds<M>::kBlocks)
k_fx_yspec(Geometry g, FxAxis ax, double* w, int batch, const double* __restrict__ mult, double* __restrict__ qrow,
           int64_t qls) {
  pdl_begin();
  constexpr int NT = group_threads(M), PP = pairs(M), lpb = Bounds<M>::kLines, n = 2 * M;
  const int grp = threadIdx.x / NT;
  const Smem sm = carve<M>(grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int ncol = g.nx - 1, nrow = n - 1, col = blockIdx.x * lpb + grp, t = G.t;
  if (col >= batch * ncol) return;
  const int b = col / ncol, I = col - b * ncol;
  double* line = w + (int64_t)b * g.nG + (int64_t)I * nrow;
  double u[PP], v[PP];
  load_pairs<M>(line, t, u, v);
  const int q = line_transform<M>(G, ax, u, v, [&] { load_pairs<M>(mult + (int64_t)I * nrow, t, u, v); });
  double* lo = line - 1 + t;
  double* hi = line + n - 1 - t;
  double A = 0.0, B = 0.0, C = 0.0;  // sums over j = t mod NT, over n - j, and the middle value
  with_results<M, double>(Pairs<M>(G.buf, t), t, q, [&](int i, bool mid, double x, double y) {
    x *= u[i];
    *(mid ? line + M - 1 : lo + NT * i) = x;
    if (mid) {
      C = x;
    } else {
      y *= v[i];
      hi[-NT * i] = y;
      A += x;
      B += y;
    }
  });
  if (b == 0) return;
  // sin(pi j / 4) for j mod 8, which is one per thread; at 3/4 the even j change sign
  auto quarter = [](int j) {
    const double s = (j & 1) ? 0.70710678118654752440 : ((j & 3) == 2 ? 1.0 : 0.0);
    return (j & 4) ? -s : s;
  };
  const double s = quarter(t) * A + quarter(n - t) * B;
  double sa = s, sb = (t & 1) ? s : -s;
  if (t == 0) {
    sa = fma(quarter(M), C, sa);
    sb = fma(-quarter(M), C, sb);  // (M is even)
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sa += __shfl_xor_sync(kAll, sa, o);
    sb += __shfl_xor_sync(kAll, sb, o);
  }
  if (NT > 32) {
    G.put(0, (unsigned)__double2loint(sa));
    G.put(1, (unsigned)__double2hiint(sa));
    G.put(2, (unsigned)__double2loint(sb));
    G.put(3, (unsigned)__double2hiint(sb));
    G.bar();
    constexpr int W = NT / 32;
    sa = sb = 0.0;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      sa += __hiloint2double((int)G.red[W + k], (int)G.red[k]);
      sb += __hiloint2double((int)G.red[3 * W + k], (int)G.red[2 * W + k]);
    }
  }
  if (t == 0) {
    double* dst = qrow + (b - 1) * qls + I;
    dst[0] = sa;
    dst[ncol] = sb;
  }
}

// Last y pass of the same: the spectrum w plus m times the transform of apply_bc(ring), S_y, stored
// row-major.  A ring's transform is a sum of products of 1-D transforms of its sides, at column
// k = I + 1 and row j
//   sin(pi j/ny) (Fb_k - (-1)^j Ft_k) + sin(pi k/nx) (Fl_j - (-1)^k Fr_j)
// side: per ring Fb, Ft, Fl, Fr; sinx, siny: the sines.  The slots from r.n on have no ring.
template <int M>
__global__ void __launch_bounds__(Bounds<M>::kThreads, Bounds<M>::kBlocks)
k_fx_yring(Geometry g, FxAxis ax, const double* __restrict__ w, double* __restrict__ out, int batch,
           const double* __restrict__ mult, int nring, const double* __restrict__ side,
           const double* __restrict__ sinx, const double* __restrict__ siny) {
  pdl_begin();
  constexpr int NT = group_threads(M), PP = pairs(M), lpb = Bounds<M>::kLines, n = 2 * M;
  const int grp = threadIdx.x / NT;
  const Smem sm = carve<M>(grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int ncol = g.nx - 1, nrow = n - 1, total = batch * ncol;
  const int col0 = blockIdx.x * lpb, col = col0 + grp;
  if (col < total) {
    const int b = col / ncol, I = col - b * ncol, t = G.t;
    double u[PP], v[PP];
    load_pairs<M>(w + (int64_t)b * g.nG + (int64_t)I * nrow, t, u, v);
    if (b < nring) {
      const double* m = mult + (int64_t)I * nrow;
      const double* sd = side + (int64_t)b * 2 * (ncol + nrow);
      const double fb = sd[I], ft = sd[ncol + I];
      const double* fl = sd + 2 * ncol;
      const double* fr = fl + nrow;
      const double sk = sinx[I], sr = (I & 1) ? -sk : sk;
      const double fs = (t & 1) ? fb + ft : fb - ft;  // j has t's parity (t = 0: the middle's, even)
      auto add = [&](double& x, int j) {
        x = fma(m[j - 1], fma(siny[j - 1], fs, fma(sk, fl[j - 1], sr * fr[j - 1])), x);
      };
#pragma unroll
      for (int i = 0; i < PP; ++i) {
        const int j = t + NT * i;
        if (M == NT * PP || j < M) {
          const bool mid = i == 0 && t == 0;
          add(u[i], mid ? M : j);
          if (!mid) add(v[i], n - j);
        }
      }
    }
    const int q = line_transform<M>(G, ax, u, v, [] {});
    if (t == 0) sm.q[grp] = q;
  }
  store_transposed<M>(sm, col0, total, ncol, g.nG, out);
}

// x transform of rows, in place where in is out's memory: out = row, or out = sub_from - row
template <int M, typename T>
__global__ void __launch_bounds__(Bounds<M>::kThreads, Bounds<M>::kBlocks)
k_fx_inv(Geometry g, FxAxis ax, const double* in, T* out, int batch, const T* sub_from) {
  pdl_begin();
  constexpr int NT = group_threads(M), PP = pairs(M), lpb = Bounds<M>::kLines;
  const int grp = threadIdx.x / NT;
  const Smem sm = carve<M>(grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int ncol = 2 * M - 1, nrow = g.ny - 1, row = blockIdx.x * lpb + grp, t = G.t;
  if (row >= batch * nrow) return;
  const int b = row / nrow, J = row - b * nrow;
  const int64_t off = (int64_t)b * g.nG + (int64_t)J * ncol;
  double u[PP], v[PP];
  load_pairs<M>(in + off, t, u, v);
  T a[PP], c[PP];
  const int q = line_transform<M>(G, ax, u, v, [&] {
    if (sub_from) load_pairs<M>(sub_from + off, t, a, c);
  });
  const Pairs<M> w(G.buf, t);
  T* lo = out + off - 1 + t;
  T* hi = out + off + 2 * M - 1 - t;
  with_results<M, T>(w, t, q, [&](int i, bool mid, T x, T y) {
    if (sub_from) {
      x = a[i] - x;
      y = c[i] - y;
    }
    *(mid ? out + off + M - 1 : lo + NT * i) = x;
    if (!mid) hi[-NT * i] = y;
  });
}

template <int M, typename K, typename... Args>
cudaError_t launch(K k, int lines, cudaStream_t s, Args... args) {
  const cudaError_t e = set_smem_limit((const void*)k, smem_bytes<M>());
  if (e != cudaSuccess) return e;
  return launch_k(k, dim3((lines + Bounds<M>::kLines - 1) / Bounds<M>::kLines), dim3(Bounds<M>::kThreads),
                  smem_bytes<M>(), s, args...);
}

// the passes of one length (dstfx.cu has the entry points)
template <int M, typename T>
cudaError_t run_fwd(const Geometry& g, const FxAxis& ax, const T* in, double* out, int batch, const T* bc,
                    cudaStream_t s) {
  return launch<M>(k_fx_fwd<M, T>, batch * (g.ny - 1), s, g, ax, in, out, batch, bc);
}
template <int M>
cudaError_t run_y(const Geometry& g, const FxAxis& ay, const double* in, double* out, int batch, const double* mult,
                  int64_t mstride, int log2scale, cudaStream_t s) {
  return launch<M>(k_fx_y<M>, batch * (g.nx - 1), s, g, ay, in, out, batch, mult, mstride, log2scale);
}
template <int M>
cudaError_t run_yspec(const Geometry& g, const FxAxis& ay, double* w, int batch, const double* mult, double* qrow,
                      int64_t qls, cudaStream_t s) {
  return launch<M>(k_fx_yspec<M>, batch * (g.nx - 1), s, g, ay, w, batch, mult, qrow, qls);
}
template <int M>
cudaError_t run_yring(const Geometry& g, const FxAxis& ay, const double* w, double* out, int batch, const double* mult,
                      const FxRings& r, cudaStream_t s) {
  return launch<M>(k_fx_yring<M>, batch * (g.nx - 1), s, g, ay, w, out, batch, mult, r.n, r.side, r.sinx, r.siny);
}
template <int M, typename T>
cudaError_t run_inv(const Geometry& g, const FxAxis& ax, const double* in, T* out, int batch, const T* sub_from,
                    cudaStream_t s) {
  return launch<M>(k_fx_inv<M, T>, batch * (g.ny - 1), s, g, ax, in, out, batch, sub_from);
}

#define IB_FX_RUN_X(PREFIX, M, T)                                                                              \
  PREFIX template cudaError_t run_fwd<M, T>(const Geometry&, const FxAxis&, const T*, double*, int, const T*,  \
                                            cudaStream_t);                                                     \
  PREFIX template cudaError_t run_inv<M, T>(const Geometry&, const FxAxis&, const double*, T*, int, const T*,  \
                                            cudaStream_t);
#define IB_FX_RUN(PREFIX, M)                                                                                         \
  IB_FX_RUN_X(PREFIX, M, double)                                                                                     \
  IB_FX_RUN_X(PREFIX, M, df64)                                                                                       \
  PREFIX template cudaError_t run_y<M>(const Geometry&, const FxAxis&, const double*, double*, int, const double*,   \
                                       int64_t, int, cudaStream_t);                                                  \
  PREFIX template cudaError_t run_yspec<M>(const Geometry&, const FxAxis&, double*, int, const double*, double*,     \
                                           int64_t, cudaStream_t);                                                   \
  PREFIX template cudaError_t run_yring<M>(const Geometry&, const FxAxis&, const double*, double*, int,              \
                                           const double*, const FxRings&, cudaStream_t);

// the accepted lengths, by the translation unit that compiles their kernels
#define IB_FX_GROUP_1(X) X(4) X(24) X(60) X(108) X(180) X(288) X(450) X(640) X(900)
#define IB_FX_GROUP_2(X) X(6) X(30) X(64) X(120) X(192) X(300) X(480) X(648) X(960)
#define IB_FX_GROUP_3(X) X(8) X(32) X(72) X(128) X(200) X(320) X(486) X(720) X(972)
#define IB_FX_GROUP_4(X) X(10) X(36) X(80) X(144) X(216) X(324) X(500) X(750) X(1000)
#define IB_FX_GROUP_5(X) X(12) X(40) X(90) X(150) X(240) X(360) X(512) X(768) X(1024)
#define IB_FX_GROUP_6(X) X(16) X(48) X(96) X(160) X(250) X(384) X(540) X(800)
#define IB_FX_GROUP_7(X) X(18) X(50) X(100) X(162) X(256) X(400) X(576) X(810)
#define IB_FX_GROUP_8(X) X(20) X(54) X(270) X(432) X(600) X(864)
#define IB_FX_LENGTHS(X)                                                                              \
  IB_FX_GROUP_1(X) IB_FX_GROUP_2(X) IB_FX_GROUP_3(X) IB_FX_GROUP_4(X) IB_FX_GROUP_5(X) IB_FX_GROUP_6(X) \
  IB_FX_GROUP_7(X) IB_FX_GROUP_8(X)

}  // namespace fxp
}  // namespace ib
