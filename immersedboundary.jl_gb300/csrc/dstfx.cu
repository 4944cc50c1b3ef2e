// The FP64 sine-transform passes: every line is transformed in 64-bit block fixed point (fx.cuh).
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
//   4. doubles leave by their bits (leading-zero count, round, pack)
// A line with an infinity or NaN becomes NaN throughout, as the FP64 transform made it.  Sums of
// integers do not depend on their order, so results are the same bits for any NT.
//
// A pass reads its lines as they lie in memory and stores them transposed (the forward x pass, the y
// pass), so that the next pass's lines lie in memory: 32 or 64 bytes at a time, written without
// waiting, where a transposing load would stall the block.
//
// What bounds it: the integer pipes and the latency between them (ncu, 1024-cell lines: ALU 59% and
// FMA-heavy 46% busy, 2.5 of 4 instructions issued per clock), and the latency of a line's chain where
// a launch has few lines.  Measured against the FP64-arithmetic passes (shared-memory Stockham, one
// warp per line at 2048 cells), which the FP64 pipe's two lanes per SM bound: a 2048^2 Poisson solve
// of two fields 2.09 -> 0.54 ms, a 1024^2 x 4-level two-body step 3.75 -> 1.30 ms, 384 x 256 x 4 RKC
// 0.88 -> 0.43, 200^2 x 5 0.81 -> 0.44, 128^2 x 3 0.53 -> 0.28, with a quarter of their error on the
// 2048^2 solve (4.3e-15 against 1.8e-14).
#include "fx.cuh"
#include "ib_common.cuh"

#include <cmath>
#include <vector>

namespace ib {

namespace {

using fx::cpx;
using fx::cwgt;
using fx::i64;
using fx::u64;
using fx::wgt;

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

#ifndef S64
#define S64 32, 2
#endif
#ifndef P64
#define P64 4,4,4
#endif
#ifndef S96
#define S96 32, 3
#endif
#ifndef P96
#define P96 4,4,6
#endif
#ifndef S128
#define S128 32, 4
#endif
#ifndef P128
#define P128 8,4,4
#endif
#ifndef S192
#define S192 32, 6
#endif
#ifndef P192
#define P192 8,4,6
#endif
#ifndef S256
#define S256 32, 8
#endif
#ifndef P256
#define P256 8,8,4
#endif
#ifndef S384
#define S384 64, 6
#endif
#ifndef P384
#define P384 8,8,6
#endif
#ifndef S512
#define S512 64, 8
#endif
#ifndef P512
#define P512 8,8,8
#endif
#ifndef S768
#define S768 128, 6
#endif
#ifndef P768
#define P768 8,4,4,6
#endif
// Radices of the axes with compiled-in lengths, whose index arithmetic is constant: 64 P cells,
// P = 2^k or 3 2^k.  Large radices where many values lie in a thread's registers (M = 384 and up),
// small ones where lines are short and a launch lasts as long as a line's chain.
template <int M> struct Plan {
  static constexpr int n = 0;
  static constexpr int r[1] = {0};
};
#define IB_FX_PLANS(X) \
  X(64, 4, 4, 4) X(96, 4, 4, 6) X(128, 8, 4, 4) X(192, 4, 4, 4, 3) X(256, 4, 4, 4, 4) X(384, 8, 8, 6) X(512, 8, 8, 8) \
  X(768, 8, 4, 4, 6) X(1024, 8, 8, 4, 4)
#define IB_FX_PLAN(M, ...)                                 \
  template <> struct Plan<M> {                             \
    static constexpr int r[] = {__VA_ARGS__};              \
    static constexpr int n = sizeof(r) / sizeof(int);      \
  };
IB_FX_PLANS(IB_FX_PLAN)

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

// One Stockham stage of radix R, in place, by the threads of a group.  M_ > 0: the axis length and
// the product NS_ of the radices before are compiled in.  The first stage (Ns = 1) reads the folded
// line in its natural layout.  Returns the OR of the bits this thread's results occupy.
template <int R, int NT, int PP, int M_, int NS_>
__device__ __forceinline__ unsigned stage(const Group<NT>& G, const FxAxis& ax, int st, int d) {
  const int M = M_ ? M_ : ax.M, nb = M / R, Ns = M_ ? NS_ : ax.ns[st], t = G.t;
  // butterflies per thread (M / R <= PP NT / R)
  constexpr int NB = M_ ? (M_ / R + NT - 1) / NT : (PP + R - 1) / R;
  constexpr bool kFull = M_ && (M_ / R) % NT == 0;
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
        if (Ns == 1) v[b][r] = z[j + r * nb];
        else if (M_ && nb % 8 == 0) v[b][r] = z[cpad(t) + b * (NT + NT / 8) + r * (nb + nb / 8)];
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
      int k = 0;
      if (Ns > 1) {
        k = M_ ? j % Ns : j - (int)__umulhi((unsigned)j, ax.magic[st]) * Ns;
        if (d > 0) {
#pragma unroll
          for (int r = 0; r < R; ++r) v[b][r] = {fx::shr_rne(v[b][r].x, d), fx::shr_rne(v[b][r].y, d)};
        }
        const cwgt* tw = ax.tw + ax.twoff[st] + k;
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const int4 w = __ldg(reinterpret_cast<const int4*>(tw + (r - 1) * Ns));
          v[b][r] = fx::cmul(v[b][r], {w.x, w.y, w.z, w.w});
        }
      }
      fx::Dft<R>::run(v[b]);
      const int base = (j - k) * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        o |= occupied(v[b][r].x) | occupied(v[b][r].y);
        if (M_ && (Ns % 8 == 0 || (Ns == 1 && R == 8))) z[cpad(base) + (Ns == 1 ? r : r * (Ns + Ns / 8))] = v[b][r];
        else z[cpad(base + r * Ns)] = v[b][r];
      }
    }
  }
  return o;
}

// Shift the values now need (bits from the OR of occupied()) to fit `limit` bits.
__device__ __forceinline__ int excess(unsigned o, int limit) { return max(0, 64 - __clz((int)o) - limit); }

template <int R, int NT, int PP, int M_, int NS_>
__device__ __forceinline__ void run_stage(const Group<NT>& G, const FxAxis& ax, int st, int& T, unsigned& o) {
  const int d = st > 0 ? excess(o, fx::kStageBits) : 0;
  T += d;
  o = __reduce_or_sync(kAll, stage<R, NT, PP, M_, NS_>(G, ax, st, d));
  G.put(2 + st, o);
  G.bar();
  o = G.get(2 + st, o, [](unsigned a, unsigned b) { return a | b; });
}
template <int NT, int PP, int M_, int ST, int NS_>
__device__ __forceinline__ void fixed_stages(const Group<NT>& G, const FxAxis& ax, int& T, unsigned& o) {
  if constexpr (ST < Plan<M_>::n) {
    constexpr int R = Plan<M_>::r[ST];
    run_stage<R, NT, PP, M_, NS_>(G, ax, ST, T, o);
    fixed_stages<NT, PP, M_, ST + 1, NS_ * R>(G, ax, T, o);
  }
}

__device__ __forceinline__ i64* result_at(i64* buf, int M, int i) {
  return buf + ((i & 1) ? 0 : even_off(M)) + cpad(i >> 1);
}
// The words of a thread's pairs (j, n - j), j = t + NT i: at lo + i kStride and hi - i kStride (the
// pair j = 0 stands for the middle value, j = n / 2, alone).
template <int NT>
struct Pairs {
  static constexpr int kStride = NT / 2 + NT / 16;
  i64 *lo, *hi, *mid;
  __device__ __forceinline__ Pairs(i64* buf, int M, int t) {
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
// not finite, or at the ends of the exponent range (subnormal results, or overflow)
__device__ __noinline__ double to_double_slow(i64 v, int q) {
  if (q == kNotFinite) return __longlong_as_double(0x7ff8000000000000ll);
  return ldexp((double)v, -q);
}
// DST-I of a line given as pairs a[i] = y_j, b[i] = y_{n-j}, j = t + NT i (j = 0: a = y_{n/2}, b
// unused); the results are in place after the closing barrier.  Returns their scale q
// (F = value 2^-q), the same on every thread of the group.  `before_scan` runs before the last
// phase, with few registers in use: a place for loads that are needed next.
template <int NT, int PP, int M_, class Hook>
__device__ __forceinline__ int line_transform(const Group<NT>& G, const FxAxis& ax, const double (&a)[PP],
                                              const double (&b)[PP], Hook before_scan) {
  const int t = G.t, M = M_ ? M_ : ax.M, n = 2 * M;
  // 1. the line's largest exponent
  unsigned m = 0;
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    m = max(m, fx::mag_hi((u64)__double_as_longlong(a[i])));
    m = max(m, fx::mag_hi((u64)__double_as_longlong(b[i])));
  }
  m = __reduce_max_sync(kAll, m);
  G.put(0, m);
  G.bar();
  m = G.get(0, m, [](unsigned x, unsigned y) { return max(x, y); });
  if (m >= 0x7ff00000u) {
    G.bar();
    return kNotFinite;
  }
  const int ex = max(1, (int)(m >> 20));
  // 2. integers, folded
  unsigned asum = 0;
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    const int j = t + NT * i;
    if (M_ == NT * PP || j < M) {
      const i64 va = fx::to_fixed((u64)__double_as_longlong(a[i]), ex);
      const i64 vb = fx::to_fixed((u64)__double_as_longlong(b[i]), ex);
      // upper bound of |va| + |vb| in units of 2^35
      asum += ((unsigned)((int)(va >> 32) ^ (int)(va >> 63)) >> 3) + ((unsigned)((int)(vb >> 32) ^ (int)(vb >> 63)) >> 3) + 2u;
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
  int T = 0;
  unsigned o = 0;
  if constexpr (M_ > 0) {
    fixed_stages<NT, PP, M_, 0, 1>(G, ax, T, o);
  } else {
    for (int st = 0; st < ax.nstages; ++st) {
      switch (ax.radix[st]) {
        case 8: run_stage<8, NT, PP, 0, 0>(G, ax, st, T, o); break;
        case 4: run_stage<4, NT, PP, 0, 0>(G, ax, st, T, o); break;
        case 2: run_stage<2, NT, PP, 0, 0>(G, ax, st, T, o); break;
        case 3: run_stage<3, NT, PP, 0, 0>(G, ax, st, T, o); break;
        default: run_stage<5, NT, PP, 0, 0>(G, ax, st, T, o); break;
      }
    }
  }
  // 4. split: even outputs and differences, at four times their value
  const int abits = 37 + 32 - __clz((int)(asum - 1u));  // 4 sum |y| <= 2^abits
  const int d = max(excess(o, fx::kPostBits), abits - fx::kOutBits - T);
  T += d;
  {
    constexpr int PQ = (PP + 1) / 2;
    constexpr bool kEven = M_ == NT * PP && PP % 2 == 0;  // exactly PQ values of k per thread
    const cpx* z = reinterpret_cast<const cpx*>(G.buf);
    const int hM = M >> 1;
    cpx zk[PQ], zm[PQ];
#pragma unroll
    for (int i = 0; i < PQ; ++i) {
      const int k = t + NT * i;
      if (!kEven) zk[i] = zm[i] = {0, 0};
      if (kEven || k < hM) {
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
      if (kEven || k < hM) {
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
    constexpr bool kEven = M_ == NT * PP;  // chunks of exactly PP values
    const int C = kEven ? PP : (M + NT - 1) / NT, k0 = t * C;
    i64 s[PP], acc = 0;
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      if (kEven || (i < C && k0 + i < M)) acc += G.buf[kEven && 8 % PP == 0 ? cpad(k0) + i : cpad(k0 + i)];
      s[i] = acc;
    }
    i64 incl = acc;
#pragma unroll
    for (int w = 1; w < 32; w <<= 1) {
      const i64 v = __shfl_up_sync(kAll, incl, w);
      if ((t & 31) >= w) incl += v;
    }
    i64 excl = incl - acc;
    if (NT > 32) {
      // totals of the warps before this one (spare words after the padded differences)
      i64* tot = G.buf + M + (M >> 3) + 2;
      if ((t & 31) == 31) tot[t >> 5] = incl;
      G.bar();
#pragma unroll
      for (int w = 0; w < NT / 32 - 1; ++w)
        if ((t >> 5) > w) excl += tot[w];
    }
#pragma unroll
    for (int i = 0; i < PP; ++i)
      if (kEven || (i < C && k0 + i < M)) G.buf[kEven && 8 % PP == 0 ? cpad(k0) + i : cpad(k0 + i)] = s[i] + excl;
  }
  G.bar();
  return fx::kInBits + 1022 - ex - T + 2;
}

// ------------------------------------------------------------------------------------------------
// passes
// ------------------------------------------------------------------------------------------------
// Lines per block: 4 (stores of 32-byte segments), or 2 of the longest.  Two blocks of 256 threads per
// SM or four of 128 leave 128 registers a thread; capping at 80 or 64 for more warps costs more in
// spills than it hides (1024^2 solve of one field: 54.5 us, 57.7, 62.2).
template <int NT>
struct Bounds {
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
__host__ __device__ inline size_t smem_bytes(int M, int nt, int lpb) {
  return (size_t)lpb * line_words(M) * 8 + (size_t)lpb * (kRedSlots * (nt / 32) * 4) + (size_t)lpb * 4 + 16;
}
template <int NT>
__device__ __forceinline__ Smem carve(int M, int lpb, int grp) {
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
template <int NT, int PP, int M_>
__device__ __forceinline__ void load_pairs(const double* src, int M, int t, double (&u)[PP], double (&v)[PP]) {
  const double* lo = src - 1 + t;
  const double* hi = src + 2 * M - 1 - t;
#pragma unroll
  for (int i = 0; i < PP; ++i) {
    const bool mid = i == 0 && t == 0;
    u[i] = v[i] = 0.0;
    if (M_ == NT * PP || t + NT * i < M) {
      u[i] = *(mid ? src + M - 1 : lo + NT * i);
      if (!mid) v[i] = hi[-NT * i];
    }
  }
}

// f(i, middle, F_j, F_{n-j}) for the thread's pairs (of the middle pair only the first value)
template <int NT, int PP, int M_, class F>
__device__ __forceinline__ void with_results(const Pairs<NT>& w, int M, int t, int q, F f) {
  if (fx::safe_scale(q)) {
#pragma unroll
    for (int i = 0; i < PP; ++i)
      if (M_ == NT * PP || t + NT * i < M) {
        const bool mid = i == 0 && t == 0;
        f(i, mid, to_double(*w.a(i, mid), q), to_double(*w.b(i), q));
      }
  } else {
#pragma unroll
    for (int i = 0; i < PP; ++i)
      if (M_ == NT * PP || t + NT * i < M) {
        const bool mid = i == 0 && t == 0;
        f(i, mid, to_double_slow(*w.a(i, mid), q), to_double_slow(*w.b(i), q));
      }
  }
}

// The results of the block's lines line0 .. line0 + lpb - 1 (of `total`, `per` lines to an array of
// `stride` values), transposed: the block's lines at one index are adjacent in memory.
template <int NT>
__device__ __forceinline__ void store_transposed(const Smem& sm, int M, int line0, int total, int per,
                                                 int64_t stride, double* out) {
  __syncthreads();
  constexpr int lpb = Bounds<NT>::kLines;
  const int b0 = line0 / per, J0 = line0 - b0 * per, w = threadIdx.x % lpb;
  if (line0 + w >= total) return;
  const int wrap = J0 + w >= per;
  i64* buf = sm.lines + (size_t)w * line_words(M);
  const int q = sm.q[w];
  double* dst = out + (int64_t)(b0 + wrap) * stride + (J0 + w - (wrap ? per : 0));
  if (fx::safe_scale(q)) {
#pragma unroll 8
    for (int I = threadIdx.x / lpb; I < 2 * M - 1; I += NT)
      dst[(int64_t)I * per] = to_double(*result_at(buf, M, I + 1), q);
  } else {
#pragma unroll 1
    for (int I = threadIdx.x / lpb; I < 2 * M - 1; I += NT)
      dst[(int64_t)I * per] = to_double_slow(*result_at(buf, M, I + 1), q);
  }
}

// x transform of rows as they lie in memory -> transposed intermediate; optional apply_bc(bc) on the
// edges (fluid-ops.jl:249-275)
template <int NT, int PP, int M_>
__global__ void __launch_bounds__(Bounds<NT>::kThreads, Bounds<NT>::kBlocks)
k_fx_fwd(Geometry g, FxAxis ax, const double* __restrict__ in, double* __restrict__ out, int batch,
         const double* __restrict__ bc, double bcfac) {
  pdl_begin();
  constexpr int lpb = Bounds<NT>::kLines;
  const int M = M_ ? M_ : ax.M, grp = threadIdx.x / NT;
  const Smem sm = carve<NT>(M, lpb, grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int n = 2 * M, ncol = n - 1, nrow = g.ny - 1, total = batch * nrow;
  const int row0 = blockIdx.x * lpb, row = row0 + grp;
  if (row < total) {
    const int b = row / nrow, J = row - b * nrow;
    const double* src = in + (int64_t)b * g.nG + (int64_t)J * ncol;
    double u[PP], v[PP];
    load_pairs<NT, PP, M_>(src, M, G.t, u, v);
    if (bc) {
      const double* r = bc + (int64_t)b * g.nbc;
      if (J == 0 || J == nrow - 1) {
        double e[PP], f[PP];
        load_pairs<NT, PP, M_>(r + (J == 0 ? g.B : g.T) + 1, M, G.t, e, f);
#pragma unroll
        for (int i = 0; i < PP; ++i) {
          u[i] += bcfac * e[i];
          v[i] += bcfac * f[i];
        }
      }
      if (G.t == 1) {  // the pair of the row's first and last value
        u[0] += bcfac * r[g.L + 1 + J];
        v[0] += bcfac * r[g.R + 1 + J];
      }
    }
    const int q = line_transform<NT, PP, M_>(G, ax, u, v, [] {});
    if (G.t == 0) sm.q[grp] = q;
  }
  store_transposed<NT>(sm, M, row0, total, nrow, g.nG, out);
}

// y pass: columns of the transposed intermediate, S_y, times m, S_y (or S_y only), times 2^log2scale,
// stored row-major
template <int NT, int PP, int M_>
__global__ void __launch_bounds__(Bounds<NT>::kThreads, Bounds<NT>::kBlocks)
k_fx_y(Geometry g, FxAxis ax, const double* __restrict__ in, double* __restrict__ out, int batch,
       const double* mult, int64_t mstride, int log2scale) {
  pdl_begin();
  constexpr int lpb = Bounds<NT>::kLines;
  const int M = M_ ? M_ : ax.M, grp = threadIdx.x / NT;
  const Smem sm = carve<NT>(M, lpb, grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int ncol = g.nx - 1, nrow = 2 * M - 1, total = batch * ncol;
  const int col0 = blockIdx.x * lpb, col = col0 + grp;
  if (col < total) {
    const int b = col / ncol, I = col - b * ncol, t = G.t;
    const Pairs<NT> w(G.buf, M, t);
    const double* m = mult ? mult + (int64_t)b * mstride + (int64_t)I * nrow : nullptr;
    double u[PP], v[PP];
    load_pairs<NT, PP, M_>(in + (int64_t)b * g.nG + (int64_t)I * nrow, M, t, u, v);
    int q;
    // (one copy of the transform's code: two would not fit the instruction cache)
#pragma unroll 1
    for (int pass = 0;; ++pass) {
      const bool more = pass == 0 && m;
      q = line_transform<NT, PP, M_>(G, ax, u, v, [&] {
        if (more) load_pairs<NT, PP, M_>(m, M, t, u, v);
      });
      if (!more) break;
      with_results<NT, PP, M_>(w, M, t, q, [&](int i, bool mid, double x, double y) {
        u[i] *= x;
        v[i] = mid ? 0.0 : v[i] * y;
      });
    }
    if (G.t == 0) sm.q[grp] = q - (q == kNotFinite ? 0 : log2scale);
  }
  store_transposed<NT>(sm, M, col0, total, ncol, g.nG, out);
}

// x transform of rows, in place where in == out: out = row, or out = sub_from - row
template <int NT, int PP, int M_>
__global__ void __launch_bounds__(Bounds<NT>::kThreads, Bounds<NT>::kBlocks)
k_fx_inv(Geometry g, FxAxis ax, const double* in, double* out, int batch, const double* sub_from) {
  pdl_begin();
  constexpr int lpb = Bounds<NT>::kLines;
  const int M = M_ ? M_ : ax.M, grp = threadIdx.x / NT;
  const Smem sm = carve<NT>(M, lpb, grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int ncol = 2 * M - 1, nrow = g.ny - 1, row = blockIdx.x * lpb + grp, t = G.t;
  if (row >= batch * nrow) return;
  const int b = row / nrow, J = row - b * nrow;
  const int64_t off = (int64_t)b * g.nG + (int64_t)J * ncol;
  double u[PP], v[PP];
  load_pairs<NT, PP, M_>(in + off, M, t, u, v);
  const int q = line_transform<NT, PP, M_>(G, ax, u, v, [&] {
    if (sub_from) load_pairs<NT, PP, M_>(sub_from + off, M, t, u, v);
  });
  const Pairs<NT> w(G.buf, M, t);
  double* lo = out + off - 1 + t;
  double* hi = out + off + 2 * M - 1 - t;
  with_results<NT, PP, M_>(w, M, t, q, [&](int i, bool mid, double x, double y) {
    if (sub_from) {
      x = u[i] - x;
      y = v[i] - y;
    }
    *(mid ? out + off + M - 1 : lo + NT * i) = x;
    if (!mid) hi[-NT * i] = y;
  });
}

// Threads per line, pairs per thread and compiled-in length, by M; lengths without a plan of their own
// take the runtime indexing.  Measured, a Poisson solve of one field: 512^2 with 64 threads a line and
// four pairs each 23.1 us, 32 and eight 27.9; 768 x 512 with 64 and six (x) 30.8, 128 and three 34.5;
// 1024^2 with 64 and eight 54.5, 128 and four 64.7; 2048^2 x 2 with two lines a block 396, four 424.
#define IB_FX_SHAPE(M, CALL)                  \
  do {                                        \
    switch (M) {                              \
      case 64: { CALL(32, 2, 64); }           \
      case 96: { CALL(32, 3, 96); }           \
      case 128: { CALL(32, 4, 128); }         \
      case 192: { CALL(64, 3, 192); }         \
      case 256: { CALL(64, 4, 256); }         \
      case 384: { CALL(64, 6, 384); }         \
      case 512: { CALL(64, 8, 512); }         \
      case 768: { CALL(128, 6, 768); }        \
      case 1024: { CALL(128, 8, 1024); }      \
      default: break;                         \
    }                                         \
    if ((M) <= 64) { CALL(32, 2, 0); }        \
    else if ((M) <= 128) { CALL(32, 4, 0); }  \
    else if ((M) <= 256) { CALL(64, 4, 0); }  \
    else if ((M) <= 512) { CALL(64, 8, 0); }  \
    else { CALL(128, 8, 0); }                 \
  } while (0)

// radices of an axis: its plan's, or the general ones
int fx_radices(int M, int* radix) {
  switch (M) {
#define IB_FX_COPY(LEN, ...)                                                   \
  case LEN: {                                                                  \
    for (int i = 0; i < Plan<LEN>::n; ++i) radix[i] = Plan<LEN>::r[i];         \
    return Plan<LEN>::n;                                                       \
  }
    IB_FX_PLANS(IB_FX_COPY)
#undef IB_FX_COPY
    default: return plan_radices(M, radix);
  }
}

template <int NT, typename K, typename... Args>
cudaError_t launch(K k, int M, int lines, cudaStream_t s, Args... args) {
  constexpr int lpb = Bounds<NT>::kLines;
  const size_t smem = smem_bytes(M, NT, lpb);
  const cudaError_t e = set_smem_limit((const void*)k, smem);
  if (e != cudaSuccess) return e;
  return launch_k(k, dim3((lines + lpb - 1) / lpb), dim3(lpb * NT), smem, s, args...);
}

}  // namespace

cudaError_t FxTables::build(int n) {
  release();
  if (!dst_axis_supported(n)) return cudaErrorInvalidValue;
  const int M = n / 2;
  d = FxAxis{};
  d.n = n;
  d.M = M;
  d.nstages = fx_radices(M, d.radix);
  const long double pi = 3.141592653589793238462643383279502884L;
  auto split = [](long double w) {
    const i64 v = llrintl(w * (long double)((i64)1 << 60));
    const int h = (int)((v + ((i64)1 << 29)) >> 30);
    return wgt{h, (int)(v - ((i64)h << 30))};
  };
  auto cis = [&](long double num, long double den) {  // e^{-2 pi i num / den}
    const long double ang = -2.0L * pi * num / den;
    const wgt c = split(cosl(ang)), s = split(sinl(ang));
    return cwgt{c.h, c.l, s.h, s.l};
  };
  std::vector<cwgt> tw, post(M / 2 + 1);
  std::vector<wgt> sn(M + 1);
  int Ns = 1;
  for (int st = 0; st < d.nstages; ++st) {
    const int R = d.radix[st];
    d.ns[st] = Ns;
    d.magic[st] = Ns > 1 ? (unsigned)((((u64)1 << 32) + Ns - 1) / Ns) : 0u;  // exact quotients below 2^16
    d.twoff[st] = (int)tw.size();
    if (st > 0)
      for (int r = 1; r < R; ++r)
        for (int k = 0; k < Ns; ++k) tw.push_back(cis((long double)(r * k), (long double)(Ns * R)));
    Ns *= R;
  }
  for (int k = 0; k <= M / 2; ++k) post[k] = cis((long double)k, (long double)n);
  // 2 sin(pi j / n) < 2 for j < M
  for (int j = 0; j < M; ++j) sn[j] = split(2.0L * sinl(pi * (long double)j / (long double)n));
  const size_t btw = tw.size() * sizeof(cwgt), bpost = post.size() * sizeof(cwgt), bsn = sn.size() * sizeof(wgt);
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  cudaError_t e = cudaMalloc(&mem, up(btw) + up(bpost) + up(bsn) + 256);
  if (e != cudaSuccess) { mem = nullptr; return e; }
  char* base = static_cast<char*>(mem);
  if (btw && (e = cudaMemcpy(base, tw.data(), btw, cudaMemcpyHostToDevice)) != cudaSuccess) return e;
  if ((e = cudaMemcpy(base + up(btw), post.data(), bpost, cudaMemcpyHostToDevice)) != cudaSuccess) return e;
  if ((e = cudaMemcpy(base + up(btw) + up(bpost), sn.data(), bsn, cudaMemcpyHostToDevice)) != cudaSuccess) return e;
  d.tw = reinterpret_cast<const cwgt*>(base);
  d.post = reinterpret_cast<const cwgt*>(base + up(btw));
  d.sin2 = reinterpret_cast<const wgt*>(base + up(btw) + up(bpost));
  return cudaSuccess;
}

void FxTables::release() {
  if (mem) cudaFree(mem);
  mem = nullptr;
}

cudaError_t fx_fwd(const Geometry& g, const FxAxis& ax, const double* in, double* out, int batch, const double* bc,
                   double bcfac, cudaStream_t s) {
  if (ax.n != g.nx) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassXPass, s);
#define IB_FX_CALL(NT, PP, ML) \
  return launch<NT>(k_fx_fwd<NT, PP, ML>, ax.M, batch * (g.ny - 1), s, g, ax, in, out, batch, bc, bcfac)
  IB_FX_SHAPE(ax.M, IB_FX_CALL);
#undef IB_FX_CALL
}

cudaError_t fx_ypass(const Geometry& g, const FxAxis& ay, const double* in, double* out, int batch, const double* mult,
                     int64_t mstride, int log2scale, cudaStream_t s) {
  if (ay.n != g.ny) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassYPass, s);
#define IB_FX_CALL(NT, PP, ML) \
  return launch<NT>(k_fx_y<NT, PP, ML>, ay.M, batch * (g.nx - 1), s, g, ay, in, out, batch, mult, mstride, log2scale)
  IB_FX_SHAPE(ay.M, IB_FX_CALL);
#undef IB_FX_CALL
}

cudaError_t fx_inv(const Geometry& g, const FxAxis& ax, const double* in, double* out, int batch,
                   const double* sub_from, cudaStream_t s) {
  if (ax.n != g.nx) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassXPass, s);
#define IB_FX_CALL(NT, PP, ML) \
  return launch<NT>(k_fx_inv<NT, PP, ML>, ax.M, batch * (g.ny - 1), s, g, ax, in, out, batch, sub_from)
  IB_FX_SHAPE(ax.M, IB_FX_CALL);
#undef IB_FX_CALL
}

}  // namespace ib
