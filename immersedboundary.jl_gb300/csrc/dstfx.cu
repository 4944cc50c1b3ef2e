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
// Lines run along x as they lie in memory; the intermediate of a solve is stored transposed (element
// (I, J) of slot b at b*stride + I*(ny-1) + J), so the y pass reads and writes whole columns.
//
// What bounds it: instruction issue (243 instructions per value and transform at 1024 cells, 2.0-2.5
// of 4 issued per clock) at large sizes, the latency of a line's chain at small ones.  Measured
// against the FP64-arithmetic passes (shared-memory Stockham, and one warp per line at 2048 cells),
// which the FP64 pipe's two lanes per SM bound: a 2048^2 Poisson solve of two fields 2.09 -> 0.67 ms,
// a 1024^2 x 4-level two-body step 3.75 -> 1.44 ms, 200^2 x 5 0.81 -> 0.58, 128^2 x 3 0.53 -> 0.33, with
// 0.25 of their error on the 2048^2 solve (4.3e-15 against 1.8e-14).
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

// 8-byte words of one line's buffer: M complex values padded; congruent to 4 mod 16, so that four
// lines' words at one index lie in different banks
__host__ __device__ inline int line_words(int M) { return (2 * M + M / 4 + 8 + 15) / 16 * 16 + 4; }

// Radices of the axes with compiled-in lengths, whose index arithmetic is constant.  Powers of two
// and 3 * 2^k: one butterfly per thread and stage where that fills the group, small radices where
// lines are short (then a call's latency counts, not its throughput).
template <int M> struct Plan {
  static constexpr int n = 0;
  static constexpr int r[1] = {0};
};
#define IB_FX_PLANS(X) \
  X(64, 4, 4, 4) X(96, 4, 4, 6) X(128, 8, 4, 4) X(192, 8, 4, 6) X(256, 8, 8, 4) X(384, 8, 8, 6) X(512, 8, 8, 8) \
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

// The results F_i, i = 1..n-1, of a line lie at word cpad(i / 2) of two regions of its buffer: the
// odd ones in the first, the even ones in the second.
__host__ __device__ constexpr int even_off(int M) { return M + (M >> 3) + 8; }
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

// the double of a result on scale q
__device__ __forceinline__ double to_double(i64 v, int q) {
  if (q == kNotFinite) return __longlong_as_double(0x7ff8000000000000ll);
  if (fx::safe_scale(q)) return __longlong_as_double((i64)fx::from_fixed(v, q));
  return ldexp((double)v, -q);  // at the ends of the exponent range: subnormal results, or overflow
}

// DST-I of a line given as pairs a[i] = y_j, b[i] = y_{n-j}, j = t + NT i (j = 0: a = y_{n/2}, b
// unused); the results are in place after the closing barrier.  Returns their scale q
// (F = value 2^-q), the same on every thread of the group.
template <int NT, int PP, int M_>
__device__ __forceinline__ int line_transform(const Group<NT>& G, const FxAxis& ax, const double (&a)[PP],
                                              const double (&b)[PP]) {
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

template <int NT>
struct Bounds {
  static constexpr int kThreads = NT == 128 ? 512 : 256;
  static constexpr int kBlocks = NT == 128 ? 1 : 3;
};

// x transform of rows as they lie in memory -> transposed intermediate; optional apply_bc(bc) on the
// edges (fluid-ops.jl:249-275)
template <int NT, int PP, int M_>
__global__ void __launch_bounds__(Bounds<NT>::kThreads, Bounds<NT>::kBlocks)
k_fx_fwd(Geometry g, FxAxis ax, const double* __restrict__ in, double* __restrict__ out, int batch,
         const double* __restrict__ bc, double bcfac) {
  pdl_begin();
  const int M = M_ ? M_ : ax.M, lpb = blockDim.x / NT, grp = threadIdx.x / NT;
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
    const int q = line_transform<NT, PP, M_>(G, ax, u, v);
    if (G.t == 0) sm.q[grp] = q;
  }
  __syncthreads();
  // transposed store: the block's rows at one column are adjacent in memory
  const int b0 = row0 / nrow, J0 = row0 - b0 * nrow, sh = 31 - __clz(lpb);
  const int w = threadIdx.x & (lpb - 1);
  if (row0 + w < total) {
    const int wrap = J0 + w >= nrow;
    i64* buf = sm.lines + (size_t)w * line_words(M);
    const int q = sm.q[w];
    double* dst = out + (int64_t)(b0 + wrap) * g.nG + (J0 + w - (wrap ? nrow : 0));
#pragma unroll 4
    for (int I = threadIdx.x >> sh; I < ncol; I += NT)
      dst[(int64_t)I * nrow] = to_double(*result_at(buf, M, I + 1), q);
  }
}

// y pass on the transposed intermediate: column by column S_y, times m, S_y (or scal S_y only)
template <int NT, int PP, int M_>
__global__ void __launch_bounds__(Bounds<NT>::kThreads, Bounds<NT>::kBlocks)
k_fx_y(Geometry g, FxAxis ax, const double* in, double* out, int batch, const double* mult, int64_t mstride,
       double scal) {
  pdl_begin();
  const int M = M_ ? M_ : ax.M, lpb = blockDim.x / NT, grp = threadIdx.x / NT;
  const Smem sm = carve<NT>(M, lpb, grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int n = 2 * M, ncol = g.nx - 1, nrow = n - 1;
  const int col = blockIdx.x * lpb + grp;
  if (col >= batch * ncol) return;
  const int b = col / ncol, I = col - b * ncol, t = G.t;
  const int64_t off = (int64_t)b * g.nG + (int64_t)I * nrow;
  const Pairs<NT> w(G.buf, M, t);
  double u[PP], v[PP];
  load_pairs<NT, PP, M_>(in + off, M, t, u, v);
  int q = line_transform<NT, PP, M_>(G, ax, u, v);
  if (mult) {
    // the products take the results' places in the line buffer: the thread that made them reads them
    const double* m = mult + (int64_t)b * mstride + (int64_t)I * nrow;
#pragma unroll 2
    for (int i = 0; i < PP; ++i) {
      const bool mid = i == 0 && t == 0;
      if (M_ == NT * PP || t + NT * i < M) {
        i64* x = w.a(i, mid);
        *x = __double_as_longlong(to_double(*x, q) * m[mid ? M - 1 : t + NT * i - 1]);
        x = w.b(i);
        if (!mid) *x = __double_as_longlong(to_double(*x, q) * m[n - 1 - t - NT * i]);
      }
    }
#pragma unroll
    for (int i = 0; i < PP; ++i) {
      const bool mid = i == 0 && t == 0;
      u[i] = v[i] = 0.0;
      if (M_ == NT * PP || t + NT * i < M) {
        u[i] = __longlong_as_double(*w.a(i, mid));
        if (!mid) v[i] = __longlong_as_double(*w.b(i));
      }
    }
    q = line_transform<NT, PP, M_>(G, ax, u, v);
    scal = 1.0;
  }
  double* dst = out + off;
#pragma unroll 4
  for (int i = 0; i < PP; ++i) {
    const bool mid = i == 0 && t == 0;
    if (M_ == NT * PP || t + NT * i < M) {
      const double x = to_double(*w.a(i, mid), q), y = to_double(*w.b(i), q);
      dst[mid ? M - 1 : t + NT * i - 1] = mult ? x : x * scal;
      if (!mid) dst[n - 1 - t - NT * i] = mult ? y : y * scal;
    }
  }
}

// transposed intermediate -> x transform -> rows: out = row, or out = sub_from - row
template <int NT, int PP, int M_>
__global__ void __launch_bounds__(Bounds<NT>::kThreads, Bounds<NT>::kBlocks)
k_fx_inv(Geometry g, FxAxis ax, const double* __restrict__ in, double* out, int batch, const double* sub_from) {
  pdl_begin();
  const int M = M_ ? M_ : ax.M, lpb = blockDim.x / NT, grp = threadIdx.x / NT;
  const Smem sm = carve<NT>(M, lpb, grp);
  const Group<NT> G{(int)threadIdx.x % NT, grp, sm.line, sm.red};
  const int n = 2 * M, ncol = n - 1, nrow = g.ny - 1, total = batch * nrow;
  const int row0 = blockIdx.x * lpb;
  {
    const int b0 = row0 / nrow, J0 = row0 - b0 * nrow, sh = 31 - __clz(lpb);
    const int w = threadIdx.x & (lpb - 1);
    if (row0 + w < total) {
      const int wrap = J0 + w >= nrow;
      double* buf = reinterpret_cast<double*>(sm.lines + (size_t)w * line_words(M));
      const double* src = in + (int64_t)(b0 + wrap) * g.nG + (J0 + w - (wrap ? nrow : 0));
#pragma unroll 16
      for (int I = threadIdx.x >> sh; I < ncol; I += NT) buf[I + 1] = src[(int64_t)I * nrow];
    }
  }
  __syncthreads();
  const int row = row0 + grp, t = G.t;
  if (row >= total) return;
  double u[PP], v[PP];
  load_pairs<NT, PP, M_>(reinterpret_cast<const double*>(G.buf) + 1, M, t, u, v);
  const int q = line_transform<NT, PP, M_>(G, ax, u, v);
  const Pairs<NT> w(G.buf, M, t);
  const int b = row / nrow, J = row - b * nrow;
  const int64_t off = (int64_t)b * g.nG + (int64_t)J * ncol;
  double* dst = out + off;
  const double* sf = sub_from ? sub_from + off : nullptr;
#pragma unroll 4
  for (int i = 0; i < PP; ++i) {
    const bool mid = i == 0 && t == 0;
    if (M_ == NT * PP || t + NT * i < M) {
      const int p = mid ? M - 1 : t + NT * i - 1, r = n - 1 - t - NT * i;
      const double x = to_double(*w.a(i, mid), q), y = to_double(*w.b(i), q);
      dst[p] = sf ? sf[p] - x : x;
      if (!mid) dst[r] = sf ? sf[r] - y : y;
    }
  }
}

// Threads per line, pairs per thread and compiled-in length, by M.  A line's group is the fewest warps
// that hold it eight pairs a thread; lengths without a plan of their own take the runtime indexing.
#define IB_FX_SHAPE(M, CALL)                  \
  do {                                        \
    switch (M) {                              \
      case 64: { CALL(32, 2, 64); }           \
      case 96: { CALL(32, 3, 96); }           \
      case 128: { CALL(32, 4, 128); }         \
      case 192: { CALL(32, 6, 192); }         \
      case 256: { CALL(32, 8, 256); }         \
      case 384: { CALL(64, 6, 384); }         \
      case 512: { CALL(64, 8, 512); }         \
      case 768: { CALL(128, 6, 768); }        \
      case 1024: { CALL(128, 8, 1024); }      \
      default: break;                         \
    }                                         \
    if ((M) <= 64) { CALL(32, 2, 0); }        \
    else if ((M) <= 128) { CALL(32, 4, 0); }  \
    else if ((M) <= 256) { CALL(32, 8, 0); }  \
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

int lines_per_block(int M) { return M <= 256 ? 8 : 4; }

template <typename K, typename... Args>
cudaError_t launch(K k, int M, int nt, int lpb, int blocks, cudaStream_t s, Args... args) {
  const size_t smem = smem_bytes(M, nt, lpb);
  const cudaError_t e = set_smem_limit((const void*)k, smem);
  if (e != cudaSuccess) return e;
  return launch_k(k, dim3(blocks), dim3(lpb * nt), smem, s, args...);
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
  const int lpb = lines_per_block(ax.M), blocks = (batch * (g.ny - 1) + lpb - 1) / lpb;
#define IB_FX_CALL(NT, PP, ML)                                                             \
  return launch(k_fx_fwd<NT, PP, ML>, ax.M, NT, lpb, blocks, s, g, ax, in, out, batch, bc, bcfac)
  IB_FX_SHAPE(ax.M, IB_FX_CALL);
#undef IB_FX_CALL
}

cudaError_t fx_ypass(const Geometry& g, const FxAxis& ay, const double* in, double* out, int batch, const double* mult,
                     int64_t mstride, double scal, cudaStream_t s) {
  if (ay.n != g.ny) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassYPass, s);
  const int lpb = lines_per_block(ay.M), blocks = (batch * (g.nx - 1) + lpb - 1) / lpb;
#define IB_FX_CALL(NT, PP, ML)                                                             \
  return launch(k_fx_y<NT, PP, ML>, ay.M, NT, lpb, blocks, s, g, ay, in, out, batch, mult, mstride, scal)
  IB_FX_SHAPE(ay.M, IB_FX_CALL);
#undef IB_FX_CALL
}

cudaError_t fx_inv(const Geometry& g, const FxAxis& ax, const double* in, double* out, int batch,
                   const double* sub_from, cudaStream_t s) {
  if (ax.n != g.nx) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassXPass, s);
  const int lpb = lines_per_block(ax.M), blocks = (batch * (g.ny - 1) + lpb - 1) / lpb;
#define IB_FX_CALL(NT, PP, ML)                                                             \
  return launch(k_fx_inv<NT, PP, ML>, ax.M, NT, lpb, blocks, s, g, ax, in, out, batch, sub_from)
  IB_FX_SHAPE(ax.M, IB_FX_CALL);
#undef IB_FX_CALL
}

}  // namespace ib
