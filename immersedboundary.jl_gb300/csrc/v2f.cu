// Multilevel Vort2Flux with all levels solved together: the ring transfer of the fixed-point form (both
// precisions) and the kernels of the FP32 form (mixed precision, warp-per-line passes).
//
// Vort2Flux (src/streamfcn/fluid-ops.jl:438-472) solves the levels coarse to fine: level l's
// Poisson problem takes its boundary ring from psi_{l+1} (get_bc!, fluid-ops.jl:210-239), so the
// reference order is a chain of one-array solves.  Here the ring of every level is found first
// and all levels are then solved in one batch:
//
//   psi_{l+1} = psi0_{l+1} + H(ring_{l+1}),  psi0 = L^-1 Gamma (zero ring),  H = L^-1 apply_bc
//   ring_l    = get_bc(psi_{l+1})   (0.25 x values on the quarter lines of level l+1)
//
// The quarter lines lie n/4 cells inside level l+1.  Boundary mode k (sine along the side) of
// the harmonic part H decays across the grid as sinh(th_k (n-1-J)) / sinh(th_k n), 2 cosh th_k
// = 4 - 2 cos(pi (k+1)/n), i.e. by ~exp(-pi (k+1)/4) at the quarter lines: Kx (Ky) modes per
// side give H there to FP64 rounding.  ring_l is then a small FP64 product per level:
//   coef = St . sides(ring_{l+1}),  ring_l = ring(psi0_{l+1}) + Aring . coef.
// FP32 form: psi0 on the quarter lines comes from the first refinement sweeps: the previous call's psi
// plus an FP32 solve of its residual (x0) plus the next correction's spectrum evaluated on those
// lines (row sums in the y pass, column sums over the spectrum, then 1-D transforms).  The
// residual carries the rings of the previous call as a predictor, so psi0 above is psi with
// those rings and the chain carries only the change:
//   ring_l = get_bc(psi_old-ring_{l+1}) + Aring . coef(ring_{l+1} - ring_old_{l+1}).
#include <algorithm>
#include <cmath>
#include <vector>

#include "dstw.cuh"

namespace ib {
namespace {

using wdst::kLB;
using wdst::kLines;
using wdst::line_dst;
using wdst::Shape;

// sin(pi m / 4) (row / column n/4) and sin(3 pi m / 4) (row / column 3n/4), m = (index+1) mod 8
__device__ __forceinline__ void quarter_weights(int m, float& qa, float& qb) {
  const float s = 0.70710678118654752f;
  const float mag = (m & 1) ? s : ((m & 3) == 2 ? 1.0f : 0.0f);
  qa = (m & 4) ? -mag : mag;
  qb = (m & 1) ? qa : -qa;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// line (b, k) of the transposed intermediate into U[1..nrow]
template <int NL>
__device__ __forceinline__ void load_line(float* U, const float* src, int nrow, int lane) {
  for (int J0 = lane; J0 < nrow; J0 += kLB * NL) {
    float v[kLB];
#pragma unroll
    for (int u = 0; u < kLB; ++u) v[u] = (J0 + NL * u < nrow) ? src[J0 + NL * u] : 0.0f;
#pragma unroll
    for (int u = 0; u < kLB; ++u)
      if (J0 + NL * u < nrow) U[J0 + NL * u + 1] = v[u];
  }
}

// y pass, spectrum only: S_y, multiply, store the spectrum in place, and the two quarter-row
// sums of its inverse, vrow[b][s][k] = sum_l sin(pi (l+1)(J_s+1)/ny) spec[k][l].
template <int P>
// 8 resident blocks per SM (64 registers), as the warp y pass the autotuner picks at the sizes
// that use the all-levels Vort2Flux
__global__ void __launch_bounds__(kLines * 32, 8)
k_wy_spec(Geometry g, DstAxis<float> ax, float* w, const float* m, int batch, float* vrow) {
  pdl_begin();
  using Sh = Shape<float, P, 32>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int wi = threadIdx.x / 32, lane = threadIdx.x % 32;
  float* U = reinterpret_cast<float*>(smem_raw) + wi * Sh::kStride;
  float* D = U + Sh::kU;
  const int ncol = g.nx - 1, nrow = g.ny - 1;
  float qa, qb;
  quarter_weights((lane + 1) & 7, qa, qb);  // l = lane + 32 u: (l+1) mod 8 is fixed per lane
  for (int col = blockIdx.x * kLines + wi; col < batch * ncol; col += gridDim.x * kLines) {
    const int b = col / ncol, k = col - b * ncol;
    float* line = w + (int64_t)b * g.nG + (int64_t)k * nrow;
    load_line<32>(U, line, nrow, lane);
    __syncwarp();
    line_dst<float, P, 32>(U, D, ax, lane, wi + 1);
    const float* mk = m + (int64_t)k * nrow;
    float sa = 0.0f, sb = 0.0f;
    for (int J0 = lane; J0 < nrow; J0 += kLB * 32) {
      float mv[kLB];
#pragma unroll
      for (int u = 0; u < kLB; ++u) mv[u] = (J0 + 32 * u < nrow) ? __ldg(&mk[J0 + 32 * u]) : 0.0f;
#pragma unroll
      for (int u = 0; u < kLB; ++u) {
        const int l = J0 + 32 * u;
        if (l < nrow) {
          const float v = U[l + 1] * mv[u];
          line[l] = v;
          sa = fmaf(qa, v, sa);
          sb = fmaf(qb, v, sb);
        }
      }
    }
    sa = warp_sum(sa);
    sb = warp_sum(sb);
    if (lane == 0) {
      vrow[(int64_t)(2 * b) * ncol + k] = sa;
      vrow[(int64_t)(2 * b + 1) * ncol + k] = sb;
    }
    __syncwarp();
  }
}

// y pass of the ring sweep: spec[k][l] + m[k][l] * (2-D transform of apply_bc(ring)), S_y, store.
// The transform of the ring's edge terms is separable:
//   sin(pi (l+1)/ny) (Fb_k + (-1)^l Ft_k) + sin(pi (k+1)/nx) (Fl_l + (-1)^k Fr_l)
// with Fb, Ft (Fl, Fr) the x (y) transforms of the bottom / top (left / right) ring sides.
template <int P>
__global__ void __launch_bounds__(kLines * 32, 8)
k_wy_ring(Geometry g, DstAxis<float> ax, float* w, const float* m, int batch, const float* sidex, const float* sidey,
          const float* sinx, const float* siny) {
  pdl_begin();
  using Sh = Shape<float, P, 32>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int wi = threadIdx.x / 32, lane = threadIdx.x % 32;
  float* U = reinterpret_cast<float*>(smem_raw) + wi * Sh::kStride;
  float* D = U + Sh::kU;
  const int nx = g.nx, ny = g.ny, ncol = nx - 1, nrow = ny - 1;
  for (int col = blockIdx.x * kLines + wi; col < batch * ncol; col += gridDim.x * kLines) {
    const int b = col / ncol, k = col - b * ncol;
    float* line = w + (int64_t)b * g.nG + (int64_t)k * nrow;
    const float* mk = m + (int64_t)k * nrow;
    const float fb = sidex[(int64_t)(2 * b) * ncol + k], ft = sidex[(int64_t)(2 * b + 1) * ncol + k];
    const float sk = sinx[min(k + 1, nx - k - 1)];
    const float skr = (k & 1) ? -sk : sk;
    const float* fl = sidey + (int64_t)(2 * b) * nrow;
    const float* fr = sidey + (int64_t)(2 * b + 1) * nrow;
    // l = lane + 32 u: the parity of l is fixed per lane
    const float fbt = (lane & 1) ? fb - ft : fb + ft;
    for (int J0 = lane; J0 < nrow; J0 += kLB * 32) {
      float v[kLB], mv[kLB], a[kLB], c[kLB];
#pragma unroll
      for (int u = 0; u < kLB; ++u) {
        const int l = J0 + 32 * u;
        const bool ok = l < nrow;
        v[u] = ok ? line[l] : 0.0f;
        mv[u] = ok ? __ldg(&mk[l]) : 0.0f;
        a[u] = ok ? fl[l] : 0.0f;
        c[u] = ok ? fr[l] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < kLB; ++u) {
        const int l = J0 + 32 * u;
        if (l < nrow) {
          const float sl = siny[min(l + 1, ny - l - 1)];
          const float bcs = fmaf(sl, fbt, sk * a[u] + skr * c[u]);
          U[l + 1] = fmaf(mv[u], bcs, v[u]);
        }
      }
    }
    __syncwarp();
    line_dst<float, P, 32>(U, D, ax, lane, wi + 1);
#pragma unroll 8
    for (int J = lane; J < nrow; J += 32) line[J] = U[J + 1];
    __syncwarp();
  }
}

// Column sums of the spectrum, in nchunk partial sums over k (chunks of 8 consecutive k, so
// the quarter weights are the same for every chunk):
//   ucolp[b][s][c][l] = sum_{k in chunk c} sin(pi (k+1)(I_s+1)/nx) spec[b][k][l]
constexpr int kColChunk = 32;  // k per thread
__global__ void k_colsum(Geometry g, const float* __restrict__ w, int batch, int nchunk, float* __restrict__ ucolp) {
  pdl_begin();
  const int ncol = g.nx - 1, nrow = g.ny - 1;
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y % nchunk, b = blockIdx.y / nchunk;
  if (l >= nrow || b >= batch) return;
  const int k0 = c * kColChunk;
  const float* src = w + (int64_t)b * g.nG + l;
  float sa = 0.0f, sb = 0.0f;
#pragma unroll
  for (int r = 0; r < kColChunk; r += 8) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = (k0 + r + u < ncol) ? src[(int64_t)(k0 + r + u) * nrow] : 0.0f;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      float qa, qb;
      quarter_weights((u + 1) & 7, qa, qb);  // k0 + r is a multiple of 8
      sa = fmaf(qa, v[u], sa);
      sb = fmaf(qb, v[u], sb);
    }
  }
  ucolp[((int64_t)(2 * b) * nchunk + c) * nrow + l] = sa;
  ucolp[((int64_t)(2 * b + 1) * nchunk + c) * nrow + l] = sb;
}

// ucol[t][l] = sum_c ucolp[t][c][l] in chunk order, t = 2 b + s
__global__ void k_colred(int nlines, int nchunk, int nrow, const float* __restrict__ ucolp, float* __restrict__ ucol) {
  pdl_begin();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)nlines * nrow) return;
  const int t = (int)(i / nrow), l = (int)(i - (int64_t)t * nrow);
  const float* p = ucolp + (int64_t)t * nchunk * nrow + l;
  float s = 0.0f;
  for (int c0 = 0; c0 < nchunk; c0 += 8) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = (c0 + u < nchunk) ? p[(int64_t)(c0 + u) * nrow] : 0.0f;
#pragma unroll
    for (int u = 0; u < 8; ++u) s += v[u];
  }
  ucol[i] = s;
}

// 1-D DST-I (F convention) of `nlines` lines of ax.n-1 values, one warp per line; line t is
// (b = t / 2, s = t % 2), read at in + b in_b + s in_s and written to out + b out_b + s out_s
// (in place allowed).
template <int P>
__global__ void __launch_bounds__(kLines * 32)
k_lines(DstAxis<float> ax, const float* in, int64_t in_b, int64_t in_s, float* out, int64_t out_b, int64_t out_s,
        int nlines) {
  pdl_begin();
  using Sh = Shape<float, P, 32>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int wi = threadIdx.x / 32, lane = threadIdx.x % 32;
  float* U = reinterpret_cast<float*>(smem_raw) + wi * Sh::kStride;
  float* D = U + Sh::kU;
  const int n1 = ax.n - 1;
  const int t = blockIdx.x * kLines + wi;
  if (t >= nlines) return;
  load_line<32>(U, in + (int64_t)(t >> 1) * in_b + (int64_t)(t & 1) * in_s, n1, lane);
  __syncwarp();
  line_dst<float, P, 32>(U, D, ax, lane, wi + 1);
  float* dst = out + (int64_t)(t >> 1) * out_b + (int64_t)(t & 1) * out_s;
  for (int j = lane; j < n1; j += 32) dst[j] = U[j + 1];
}

// ring_l from psi_{l+1} (with its previous ring) on the quarter lines, the previous psi + x0 +
// the next correction, plus (below the second-coarsest level) the harmonic part of the change of
// ring_{l+1}, Aring . coef_{l+1} (AringT: [nK][nbc], coalesced over the ring entries).  A block
// of kEvalWarps warps takes 32 ring nodes: warp w sums coefficients j = w, w + kEvalWarps, ...
// for all 32 (loads coalesced, five in flight), the partial sums are added in warp order in
// shared memory, and warp 0 finishes one node per lane.  FP64; ~nbc/32 blocks, so the FP64
// work spreads over the SMs (GB300 issues a warp's FP64 instruction over ~16 cycles).  `ring`
// holds the previous ring on entry and the new one on return; the change goes to dd (FP64, for
// the next coefficients), dring (float-float, for the residual) and the float sides.
constexpr int kEvalWarps = 8;
__global__ void __launch_bounds__(kEvalWarps * 32)
k_ring_eval(Geometry g, const int4* __restrict__ pts, const df64* __restrict__ xp, const float* __restrict__ x0,
            const float* __restrict__ qline, const double* __restrict__ AringT, const double* __restrict__ coef,
            int nK, double* __restrict__ dd, df64* __restrict__ dring, df64* __restrict__ ring,
            float* __restrict__ sidex, float* __restrict__ sidey) {
  pdl_begin();
  __shared__ double part[kEvalWarps][32];
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int idx = blockIdx.x * 32 + lane;
  // warp 0 starts the node's own loads before its share of the sum
  double v = 0.0;
  df64 old(0.0f);
  if (w == 0 && idx < g.nbc) {
    const int4 p = pts[idx];
    old = ring[idx];
    v = (double)xp[p.x] + ((double)x0[p.x] + (double)qline[p.y]);
    if (p.z >= 0) v = 0.5 * (v + ((double)xp[p.z] + ((double)x0[p.z] + (double)qline[p.w])));
  }
  double h = 0.0;
  if (coef && idx < g.nbc) {
    const double* a = AringT + idx;
    constexpr int U = 5;
    int j = w;
    for (; j + (U - 1) * kEvalWarps < nK; j += U * kEvalWarps) {
      double av[U];
#pragma unroll
      for (int u = 0; u < U; ++u) av[u] = a[(int64_t)(j + u * kEvalWarps) * g.nbc];
#pragma unroll
      for (int u = 0; u < U; ++u) h = fma(av[u], __ldg(&coef[j + u * kEvalWarps]), h);
    }
    for (; j < nK; j += kEvalWarps) h = fma(a[(int64_t)j * g.nbc], __ldg(&coef[j]), h);
  }
  part[w][lane] = h;
  __syncthreads();
  if (w != 0 || idx >= g.nbc) return;
  h = 0.0;
#pragma unroll
  for (int k = 0; k < kEvalWarps; ++k) h += part[k][lane];
  v = 0.25 * v + h;
  const double d = v - (double)old;
  dd[idx] = d;
  dring[idx] = df64(d);
  ring[idx] = df64(v);
  const float df = (float)d;
  const int ncol = g.nx - 1, nrow = g.ny - 1;
  if (idx > g.B && idx < g.B + g.nx) sidex[idx - g.B - 1] = df;
  else if (idx > g.T && idx < g.T + g.nx) sidex[ncol + idx - g.T - 1] = df;
  else if (idx > g.L && idx < g.L + g.ny) sidey[idx - g.L - 1] = df;
  else if (idx > g.R && idx < g.R + g.ny) sidey[nrow + idx - g.R - 1] = df;
}

// ---- fixed-point form (doubles) ------------------------------------------------------------------
//
// Without a predictor: psi0 on the quarter lines is the lines' 1-D transforms of the spectrum's sums,
// exact to FP64 rounding, and the rings' recurrence
//   ring_l = r_l + A c_{l+1},  c_l = St . sides(ring_l),  r_l = get_bc(psi0_{l+1})
// is unrolled: with T = St . sides(A), c0_m = St . sides(r_m),
//   ring_l = r_l + sum_{m > l} A T^(m-l-1) c0_m
// so two launches make every ring, where the recurrence takes two per level (at 200^2 x 5: 38 us of 10
// launches).

// Column sums of the spectrum, levels 1..:
//   qcol[b-1][s][l] = sum_k sin(pi (k+1) I_s / nx) spec[b][k][l],  I_s = nx/4, 3nx/4
// A block takes 16 rows l; each 16 threads take every 32nd group of eight k and sum the values of one
// weight first (one FP64 addition a value); the groups' sums are added in order in shared memory.
constexpr int kSumRows = 16, kSumGroups = 32;
__global__ void __launch_bounds__(kSumRows * kSumGroups)
k_spec_colsum(Geometry g, const double* __restrict__ w, double* __restrict__ qcol, int64_t qls) {
  pdl_begin();
  __shared__ double part[2][kSumGroups][kSumRows];
  const int ncol = g.nx - 1, nrow = g.ny - 1, gr = threadIdx.x / kSumRows, r = threadIdx.x % kSumRows;
  const int l = blockIdx.x * kSumRows + r, b = blockIdx.y + 1;
  double a[6] = {0, 0, 0, 0, 0, 0};
  if (l < nrow) {
    const double* src = w + (int64_t)b * g.nG + l;
#pragma unroll 4
    for (int k0 = 8 * gr; k0 < ncol; k0 += 8 * kSumGroups) {
      double v[6];
#pragma unroll
      for (int u = 0; u < 6; ++u) {
        const int k = k0 + u + (u > 2);  // k + 1 = 1, 2, 3, 5, 6, 7 mod 8
        v[u] = k < ncol ? src[(int64_t)k * nrow] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 6; ++u) a[u] += v[u];
    }
  }
  const double odd = 0.70710678118654752440 * ((a[0] + a[2]) - (a[3] + a[5])), even = a[1] - a[4];
  part[0][gr][r] = odd + even;
  part[1][gr][r] = odd - even;
  __syncthreads();
  if (gr >= 2 || l >= nrow) return;
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < kSumGroups; ++k) s += part[gr][k][r];
  qcol[(b - 1) * qls + (int64_t)gr * nrow + l] = s;
}

// r_l: the values of get_bc from the quarter lines of the level above (their own array, q)
__device__ __forceinline__ double ring0(const int4* pts, const double* q, int idx) {
  const int4 p = pts[idx];
  const double v = q[p.y];
  return p.z >= 0 ? 0.125 * (v + q[p.w]) : 0.25 * v;
}

// coefficient j of side values f(i), i < len: sum_i St[j][i] f(i), by a block of kCoefThreads
constexpr int kCoefThreads = 128;  // (few warps: an FP64 instruction takes a warp 16 cycles, reductions too)
template <class F>
__device__ __forceinline__ double block_coef(const double* row, int len, F f) {
  constexpr int W = kCoefThreads / 32, U = 8;
  __shared__ double red[W];
  const int tid = threadIdx.x;
  double s = 0.0;
  for (int i0 = tid; i0 < len; i0 += U * kCoefThreads) {
    double v[U], r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * kCoefThreads;
      v[u] = r[u] = 0.0;
      if (i < len) {
        r[u] = row[i];
        v[u] = f(i);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * kCoefThreads < len) s = fma(r[u], v[u], s);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((tid & 31) == 0) red[tid / 32] = s;
  __syncthreads();
  s = 0.0;
#pragma unroll
  for (int w = 0; w < W; ++w) s += red[w];
  return s;
}
// its row of St and the first ring entry of its side
struct CoefSide {
  int row, first, len;
};
__device__ __forceinline__ CoefSide coef_side(const Geometry& g, int Kx, int Ky, int j) {
  const int ncol = g.nx - 1, nrow = g.ny - 1;
  if (j < 2 * Kx) return {(j < Kx ? j : j - Kx) * ncol, (j < Kx ? g.B : g.T) + 1, ncol};
  const int jj = j - 2 * Kx;
  return {Kx * ncol + (jj < Ky ? jj : jj - Ky) * nrow, (jj < Ky ? g.L : g.R) + 1, nrow};
}

// c0_m of the rings 1..L-2 (blockIdx.y + 1), one block per coefficient
__global__ void __launch_bounds__(kCoefThreads)
k_fx_coef(Geometry g, const int4* __restrict__ pts, const double* __restrict__ qfx, int64_t qls,
          const double* __restrict__ St, int Kx, int Ky, double* __restrict__ coef) {
  pdl_begin();
  const int j = blockIdx.x, m = blockIdx.y + 1;
  const CoefSide c = coef_side(g, Kx, Ky, j);
  const double* q = qfx + m * qls;  // lines of level m + 1
  const double s = block_coef(St + c.row, c.len, [&](int i) { return ring0(pts, q, c.first + i); });
  if (threadIdx.x == 0) coef[(int64_t)m * (2 * Kx + 2 * Ky) + j] = s;
}

// every ring: N nodes of ring l = blockIdx.y per block, whose lanes' 32 / N groups share the coefficients
// with those of its kRingWarps warps (the coarsest level's ring is zero)
//
// Bound by the FP64 pipe, and by the finest ring's blocks, which have the longest sums: small blocks spread
// them.  With k_fx_coef, 200^2 x 5 and 1024^2 x 4: 32 nodes and 16 warps a block 12.7, 17.4 us; 8 and 8
// 10.3, 15.8.  At 2048^2 x 5, where every SM has blocks enough, 16 nodes (37.4) over 8 (40.3).
constexpr int kRingWarps = 8;
template <typename S, int N>
__global__ void __launch_bounds__(kRingWarps * 32)
k_fx_rings(Geometry g, const int4* __restrict__ pts, const double* __restrict__ qfx, int64_t qls,
           const double* __restrict__ Apow, const double* __restrict__ coef, int nK, S* __restrict__ rings,
           double* __restrict__ side) {
  pdl_begin();
  constexpr int kGroups = 32 / N, kStep = kRingWarps * kGroups;
  __shared__ double part[kRingWarps][N];
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32, node = lane % N, l = blockIdx.y;
  const int idx = blockIdx.x * N + node;
  const bool out = w == 0 && lane < N && idx < g.nbc;
  if (l == g.nlev - 1) {
    if (out) rings[(int64_t)l * g.nbc + idx] = S(0.0);
    return;
  }
  double v = 0.0, h = 0.0;
  if (out) v = ring0(pts, qfx + l * qls, idx);
  if (idx < g.nbc) {
    // coefficients of the rings l+1..L-2 in a row, times A T^0, A T^1, ...
    const int n = (g.nlev - 2 - l) * nK;
    const double* a = Apow + idx;
    const double* c = coef + (int64_t)(l + 1) * nK;
    constexpr int U = 7;
    int j = w * kGroups + lane / N;
    for (; j + (U - 1) * kStep < n; j += U * kStep) {
      double av[U];
#pragma unroll
      for (int u = 0; u < U; ++u) av[u] = a[(int64_t)(j + u * kStep) * g.nbc];
#pragma unroll
      for (int u = 0; u < U; ++u) h = fma(av[u], __ldg(&c[j + u * kStep]), h);
    }
    for (; j < n; j += kStep) h = fma(a[(int64_t)j * g.nbc], __ldg(&c[j]), h);
  }
#pragma unroll
  for (int o = N; o < 32; o <<= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
  if (lane < N) part[w][lane] = h;
  __syncthreads();
  if (!out) return;
  h = 0.0;
#pragma unroll
  for (int k = 0; k < kRingWarps; ++k) h += part[k][node];
  v += h;
  rings[(int64_t)l * g.nbc + idx] = S(v);
  const int ncol = g.nx - 1, nrow = g.ny - 1;
  double* sd = side + l * qls;
  if (idx > g.B && idx < g.B + g.nx) sd[idx - g.B - 1] = v;
  else if (idx > g.T && idx < g.T + g.nx) sd[ncol + idx - g.T - 1] = v;
  else if (idx > g.L && idx < g.L + g.ny) sd[2 * ncol + idx - g.L - 1] = v;
  else if (idx > g.R && idx < g.R + g.ny) sd[2 * ncol + nrow + idx - g.R - 1] = v;
}

// setup: T[i][j] = coefficient i of the ring Aring[j]; Apow[d+1][j] = sum_i T[i][j] Apow[d][i]
__global__ void __launch_bounds__(kCoefThreads)
k_coef_map(Geometry g, const double* __restrict__ AringT, const double* __restrict__ St, int Kx, int Ky,
           double* __restrict__ T) {
  const int i = blockIdx.x, j = blockIdx.y, nK = 2 * Kx + 2 * Ky;
  const CoefSide c = coef_side(g, Kx, Ky, i);
  const double* side = AringT + (int64_t)j * g.nbc + c.first;
  const double s = block_coef(St + c.row, c.len, [&](int k) { return side[k]; });
  if (threadIdx.x == 0) T[(int64_t)i * nK + j] = s;
}
__global__ void k_coef_next(int nbc, int nK, const double* __restrict__ T, const double* __restrict__ A,
                            double* __restrict__ out) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  if (idx >= nbc) return;
  double s = 0.0;
  for (int i = 0; i < nK; ++i) s = fma(T[(int64_t)i * nK + j], A[(int64_t)i * nbc + idx], s);
  out[(int64_t)j * nbc + idx] = s;
}

// FP32 form: coef_l, the first Kx (Ky) sine coefficients of the bottom, top (left, right) ring sides,
// coef[j] = sum_i St[j][i] side_i (S convention, 2 sin).  One block of kCoefThreads per
// coefficient (nK blocks spread the FP64 work over the SMs), a strided sum per thread, then a
// fixed-order tree in shared memory; FP64.
__global__ void __launch_bounds__(kCoefThreads)
k_ring_coef(Geometry g, const double* __restrict__ ringd, const double* __restrict__ St, int Kx, int Ky,
            double* __restrict__ coef) {
  pdl_begin();
  const int j = blockIdx.x;
  const CoefSide c = coef_side(g, Kx, Ky, j);
  const double* side = ringd + c.first;
  const double s = block_coef(St + c.row, c.len, [&](int i) { return side[i]; });
  if (threadIdx.x == 0) coef[j] = s;
}

template <int P>
size_t line_smem() {
  return (size_t)kLines * Shape<float, P, 32>::kStride * sizeof(float);
}

// sin(pi m / n), the angle reduced in integers to at most pi/2 (a product of modes and nodes reaches
// hundreds of periods, where the rounding of the angle alone would be 1e-13)
double sin_pi(int64_t m, int n) {
  m %= 2 * n;
  const bool neg = m >= n;
  if (neg) m -= n;
  const double s = std::sin(3.14159265358979323846 * (double)std::min<int64_t>(m, n - m) / n);
  return neg ? -s : s;
}

// th with 2 cosh th = 4 - 2 cos(pi k / n): cosh th = 1 + e, e = 2 sin^2(pi k / 2n)
double decay_rate(int k, int n) {
  const double s = std::sin(3.14159265358979323846 * k / (2.0 * n)), e = 2.0 * s * s;
  return std::log1p(e + std::sqrt(e * (2.0 + e)));
}

// Response at distance J + 1 from a side to one of its mode coefficients (per 2 sin along the side), from the solves' own multipliers,
//   out[k][J] = 1/4 sum_l mult(k, l) sin(pi (l+1)/m) sin(pi (l+1)(J+1)/m),  J = 0..m-2.
// In exact arithmetic this is sinh(th (m-1-J)) / (2 n sinh(th m)), 2 cosh th = 4 - 2 cos(pi (k+1)/n); the
// multipliers carry the cancellation of their cosines (1e-12 of the smallest eigenvalue at 512 cells),
// which the rings have to share for the two Vort2Flux orders to agree to rounding.  sn: sin(pi i / m).
__global__ void k_decay(int m, const double* __restrict__ mult, int64_t mode_stride, int64_t sum_stride,
                        const double* __restrict__ sn, double* __restrict__ out) {
  const int J = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (J >= m - 1) return;
  const double* mk = mult + k * mode_stride;
  double s = 0.0;
  int a = 0;  // (l+1)(J+1) mod 2m
  for (int l = 0; l < m - 1; ++l) {
    a += J + 1;
    if (a >= 2 * m) a -= 2 * m;
    s = fma(mk[l * sum_stride] * sn[l + 1], sn[a], s);
  }
  out[(int64_t)k * (m - 1) + J] = 0.25 * s;
}

// St of one axis of n cells: 2 sin(pi (k+1) (i+1) / n), i < n - 1; sn: sin(pi i / n), i < 2 n
__global__ void k_modes(int n, const double* __restrict__ sn, double* __restrict__ St) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (i < n - 1) St[(int64_t)k * (n - 1) + i] = 2.0 * sn[(int)((int64_t)(k + 1) * (i + 1) % (2 * n))];
}

// AringT[j][idx]: harmonic response of ring entry idx (one or two nodes of the level above) to
// coefficient j; gx [k][J]: bottom-side mode k at row J, hy [k][I]: left-side mode k at column I.
// On the host these nbc nK sums were most of the tables' time.
__global__ void k_ring_response(Geometry g, const int4* __restrict__ pts, const double* __restrict__ St, int Kx, int Ky,
                                const double* __restrict__ gx, const double* __restrict__ hy,
                                double* __restrict__ AringT) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  if (idx >= g.nbc) return;
  const int ncol = g.nx - 1, nrow = g.ny - 1;
  const int4 p = pts[idx];
  auto node = [&](int at, double wt) {
    const int J = at / ncol, I = at - J * ncol;
    if (j < 2 * Kx) {
      const int k = j < Kx ? j : j - Kx;
      return wt * St[(int64_t)k * ncol + I] * gx[(int64_t)k * nrow + (j < Kx ? J : nrow - 1 - J)];
    }
    const int k = j - 2 * Kx < Ky ? j - 2 * Kx : j - 2 * Kx - Ky;
    return wt * St[(int64_t)Kx * ncol + (int64_t)k * nrow + J] *
           hy[(int64_t)k * ncol + (j - 2 * Kx < Ky ? I : ncol - 1 - I)];
  };
  AringT[(int64_t)j * g.nbc + idx] = p.z < 0 ? node(p.x, 0.25) : node(p.x, 0.125) + node(p.z, 0.125);
}

// modes kept for a side along an axis of n cells whose nearest quarter-line node is d cells
// away: the smallest K with 2 sum_{k >= K} exp(-th_k d) below 1e-17
int modes_kept(int n, int d) {
  std::vector<double> e(n - 1);
  for (int k = 0; k < n - 1; ++k) e[k] = std::exp(-decay_rate(k + 1, n) * d);
  double tail = 0.0;
  int K = n - 1;
  for (int k = n - 2; k >= 0; --k) {
    tail += 2.0 * e[k];
    if (tail >= 1e-17) break;
    K = k;
  }
  return K;
}

}  // namespace

#define CE_V(x)                      \
  do {                               \
    cudaError_t e_ = (x);            \
    if (e_ != cudaSuccess) return e_; \
  } while (0)

template <int P>
static cudaError_t launch_lines_p(const DstAxis<float>& ax, const float* in, int64_t in_b, int64_t in_s, float* out,
                                  int64_t out_b, int64_t out_s, int nlines, cudaStream_t s) {
  const size_t smem = line_smem<P>();
  cudaError_t e = set_smem_limit((const void*)k_lines<P>, smem);
  if (e != cudaSuccess) return e;
  CE_V(launch_k(k_lines<P>, dim3((nlines + kLines - 1) / kLines), dim3(kLines * 32), smem, s, ax, in, in_b, in_s, out, out_b, out_s, nlines));
  return cudaGetLastError();
}

// one-warp (wNL = 32) axes only
#define IB_V2F_P(X) X(1) X(2) X(3) X(4) X(6) X(8) X(12) X(16) X(24) X(32)

cudaError_t v2f_lines(const DstAxis<float>& ax, const float* in, int64_t in_b, int64_t in_s, float* out,
                      int64_t out_b, int64_t out_s, int nlines, cudaStream_t s) {
  if (nlines <= 0) return cudaSuccess;
  if (ax.wNL != 32) return cudaErrorInvalidValue;
  switch (ax.wP) {
#define IB_C(P) \
  case P: return launch_lines_p<P>(ax, in, in_b, in_s, out, out_b, out_s, nlines, s);
    IB_V2F_P(IB_C)
#undef IB_C
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t v2f_yspec(const Geometry& g, const DstAxis<float>& ax, float* w, const float* m, int batch, float* vrow,
                      cudaStream_t s) {
  if (ax.wNL != 32 || ax.n != g.ny) return cudaErrorInvalidValue;
  ProfScope prof(kClassYPass, s);
  const int blocks = (batch * (g.nx - 1) + kLines - 1) / kLines;
  switch (ax.wP) {
#define IB_C(P)                                                                          \
  case P: {                                                                              \
    const size_t smem = line_smem<P>();                                                  \
    cudaError_t e = set_smem_limit((const void*)k_wy_spec<P>, smem);                     \
    if (e != cudaSuccess) return e;                                                      \
    CE_V(launch_k(k_wy_spec<P>, dim3(blocks), dim3(kLines * 32), smem, s, g, ax, w, m, batch, vrow));            \
    return cudaGetLastError();                                                           \
  }
    IB_V2F_P(IB_C)
#undef IB_C
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t v2f_yring(const Geometry& g, const DstAxis<float>& axy, const DstAxis<float>& axx, float* w,
                      const float* m, int batch, const float* sidex, const float* sidey, cudaStream_t s) {
  if (axy.wNL != 32 || axy.n != g.ny || axx.n != g.nx) return cudaErrorInvalidValue;
  ProfScope prof(kClassYPass, s);
  const int blocks = (batch * (g.nx - 1) + kLines - 1) / kLines;
  switch (axy.wP) {
#define IB_C(P)                                                                                           \
  case P: {                                                                                               \
    const size_t smem = line_smem<P>();                                                                   \
    cudaError_t e = set_smem_limit((const void*)k_wy_ring<P>, smem);                                      \
    if (e != cudaSuccess) return e;                                                                       \
    CE_V(launch_k(k_wy_ring<P>, dim3(blocks), dim3(kLines * 32), smem, s, g, axy, w, m, batch, sidex, sidey, axx.sintab, axy.sintab)); \
    return cudaGetLastError();                                                                            \
  }
    IB_V2F_P(IB_C)
#undef IB_C
    default: return cudaErrorInvalidValue;
  }
}
#undef IB_V2F_P

cudaError_t v2f_colsum(const Geometry& g, const RingPlan& rp, const float* w, int batch, cudaStream_t s) {
  const int nrow = g.ny - 1;
  dim3 grid((nrow + 127) / 128, batch * rp.nchunk);
  CE_V(launch_k(k_colsum, grid, dim3(128), 0, s, g, w, batch, rp.nchunk, rp.ucolp));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int64_t n = (int64_t)2 * batch * nrow;
  CE_V(launch_k(k_colred, dim3((int)((n + 255) / 256)), dim3(256), 0, s, 2 * batch, rp.nchunk, nrow, rp.ucolp, rp.ucol));
  return cudaGetLastError();
}

cudaError_t v2f_ring_eval(const Geometry& g, const RingPlan& rp, int l, const df64* xp_up, const float* x0_up,
                          df64* ring_l, cudaStream_t s) {
  const int up = l + 1;
  const double* coef = (up < g.nlev - 1) ? rp.coef + (int64_t)up * rp.nK : nullptr;
  return launch_k(k_ring_eval, dim3((g.nbc + 31) / 32), dim3(kEvalWarps * 32), 0, s, g, (const int4*)rp.pts, xp_up,
                  x0_up, (const float*)(rp.qline + (int64_t)up * rp.qls), (const double*)rp.Aring, coef, rp.nK,
                  rp.ringd + (int64_t)l * g.nbc, reinterpret_cast<df64*>(rp.dring) + (int64_t)l * g.nbc, ring_l,
                  rp.sidex + (int64_t)l * 2 * (g.nx - 1), rp.sidey + (int64_t)l * 2 * (g.ny - 1));
}

cudaError_t v2f_ring_coef(const Geometry& g, const RingPlan& rp, int l, cudaStream_t s) {
  return launch_k(k_ring_coef, dim3(rp.nK), dim3(kCoefThreads), 0, s, g, (const double*)(rp.ringd + (int64_t)l * g.nbc),
                  (const double*)rp.St, rp.Kx, rp.Ky, rp.coef + (int64_t)l * rp.nK);
}

cudaError_t v2f_fx_colsum(const Geometry& g, const RingPlan& rp, const double* w, cudaStream_t s) {
  return launch_k(k_spec_colsum, dim3((g.ny - 1 + kSumRows - 1) / kSumRows, g.nlev - 1), dim3(kSumRows * kSumGroups), 0,
                  s, g, w, rp.qfx + 2 * (g.nx - 1), rp.qls);
}

template <typename S>
cudaError_t v2f_fx_rings(const Geometry& g, const RingPlan& rp, S* rings, cudaStream_t s) {
  if (g.nlev > 2)
    CE_V(launch_k(k_fx_coef, dim3(rp.nK, g.nlev - 2), dim3(kCoefThreads), 0, s, g, (const int4*)rp.pts,
                  (const double*)rp.qfx, rp.qls, (const double*)rp.St, rp.Kx, rp.Ky, rp.coef));
  const int N = g.nbc <= 6144 ? 8 : 16;
  return launch_k(N == 8 ? k_fx_rings<S, 8> : k_fx_rings<S, 16>, dim3((g.nbc + N - 1) / N, g.nlev),
                  dim3(kRingWarps * 32), 0, s, g, (const int4*)rp.pts, (const double*)rp.qfx, rp.qls,
                  (const double*)rp.Apow, (const double*)rp.coef, rp.nK, rings, rp.side);
}
template cudaError_t v2f_fx_rings<double>(const Geometry&, const RingPlan&, double*, cudaStream_t);
template cudaError_t v2f_fx_rings<df64>(const Geometry&, const RingPlan&, df64*, cudaStream_t);

template <typename T>
cudaError_t RingPlan::get(T*& p, int64_t n) {
  const cudaError_t e = cudaMalloc(&p, sizeof(T) * n);
  if (e == cudaSuccess) bytes += (int64_t)sizeof(T) * n;
  else p = nullptr;
  return e;
}

// Everything is ordered by s, which does not wait for the legacy stream; a failed call leaves nothing
// behind, so that the next one starts again.
cudaError_t RingPlan::build_fx(const Geometry& g, cudaStream_t s) {
  if (Apow) return cudaSuccess;
  const int L = g.nlev;
  const int64_t one = (int64_t)nK * g.nbc, bytes0 = bytes;
  double* T = nullptr;
  const cudaError_t e = [&]() -> cudaError_t {
    auto zero = [&](double*& dst, int64_t n) -> cudaError_t {
      CE_V(get(dst, n));
      return cudaMemsetAsync(dst, 0, sizeof(double) * n, s);
    };
    auto sines = [&](double*& dst, int n) -> cudaError_t {
      std::vector<double> sn(n - 1);
      for (int i = 1; i < n; ++i) sn[i - 1] = sin_pi(i, n);
      CE_V(get(dst, n - 1));
      return cudaMemcpyAsync(dst, sn.data(), sizeof(double) * (n - 1), cudaMemcpyHostToDevice, s);  // (staged: sn may go)
    };
    CE_V(zero(qfx, (L - 1) * qls));
    CE_V(zero(side, (L - 1) * qls));
    CE_V(sines(sinx, g.nx));
    CE_V(sines(siny, g.ny));
    CE_V(zero(Apow, std::max(L - 2, 1) * one));
    if (L < 3) return cudaStreamSynchronize(s);
    CE_V(cudaMemcpyAsync(Apow, Aring, sizeof(double) * one, cudaMemcpyDeviceToDevice, s));
    CE_V(cudaMalloc(&T, sizeof(double) * nK * nK));
    k_coef_map<<<dim3(nK, nK), kCoefThreads, 0, s>>>(g, Aring, St, Kx, Ky, T);
    for (int d = 1; d < L - 2; ++d)
      k_coef_next<<<dim3((g.nbc + 127) / 128, nK), 128, 0, s>>>(g.nbc, nK, T, Apow + (d - 1) * one, Apow + d * one);
    CE_V(cudaGetLastError());
    return cudaStreamSynchronize(s);
  }();
  if (e != cudaSuccess) cudaStreamSynchronize(s);
  if (T) cudaFree(T);
  if (e != cudaSuccess) {
    for (double** p : {&qfx, &side, &sinx, &siny, &Apow}) {
      if (*p) cudaFree(*p);
      *p = nullptr;
    }
    bytes = bytes0;
  }
  return e;
}

int64_t v2f_ring_work(const Geometry& g) {
  const int64_t nK = 2 * (modes_kept(g.nx, g.ny / 4) + modes_kept(g.ny, g.nx / 4)), L = g.nlev;
  return nK * g.nbc * (L - 1) * (L - 2) / 2;
}

cudaError_t RingPlan::build(const Geometry& g, const double* mult) {
  const int nx = g.nx, ny = g.ny, ncol = nx - 1, nrow = ny - 1, L = g.nlev;
  const int nx4 = nx / 4, ny4 = ny / 4;
  Kx = modes_kept(nx, ny4);  // bottom / top modes, nearest quarter-line node ny/4 cells away
  Ky = modes_kept(ny, nx4);
  nK = 2 * Kx + 2 * Ky;
  qls = 2 * (int64_t)ncol + 2 * (int64_t)nrow;
  nchunk = (ncol + kColChunk - 1) / kColChunk;
  std::vector<int4> P(g.nbc);
  for (int idx = 0; idx < g.nbc; ++idx) {
    // the nodes get_bc! reads (fluid-ops.jl:210-239): column nx/4-1 or 3nx/4-1 (left / right
    // blocks) or row ny/4-1 or 3ny/4-1 (bottom / top), averaged pairs at odd ring entries
    int J1, I1, J2 = -1, I2 = -1, q1, q2 = -1;
    if (idx < g.B) {
      const bool right = idx >= g.R;
      const int jb = idx - (right ? g.R : g.L);
      const int I = right ? 3 * nx4 - 1 : nx4 - 1;
      const int qb = 2 * ncol + (right ? nrow : 0);
      const int t = (jb + 1) >> 1;
      J1 = ny4 - 1 + ((jb & 1) ? t : jb >> 1);
      I1 = I;
      q1 = qb + J1;
      if (jb & 1) { J2 = ny4 - 2 + t; I2 = I; q2 = qb + J2; }
    } else {
      const bool top = idx >= g.T;
      const int ib = idx - (top ? g.T : g.B);
      const int J = top ? 3 * ny4 - 1 : ny4 - 1;
      const int qb = top ? ncol : 0;
      const int t = (ib + 1) >> 1;
      J1 = J;
      I1 = nx4 - 1 + ((ib & 1) ? t : ib >> 1);
      q1 = qb + I1;
      if (ib & 1) { J2 = J; I2 = nx4 - 2 + t; q2 = qb + I2; }
    }
    P[idx] = J2 < 0 ? make_int4(J1 * ncol + I1, q1, -1, -1) : make_int4(J1 * ncol + I1, q1, J2 * ncol + I2, q2);
  }
  auto up = [&](auto*& dst, const auto& src) -> cudaError_t {
    cudaError_t e = get(dst, (int64_t)src.size());
    if (e == cudaSuccess) e = cudaMemcpy(dst, src.data(), src.size() * sizeof(src[0]), cudaMemcpyHostToDevice);
    return e;
  };
  cudaError_t e;
  if ((e = up(pts, P)) != cudaSuccess) return e;
  if ((e = get(St, (int64_t)Kx * ncol + (int64_t)Ky * nrow)) != cudaSuccess) return e;
  if ((e = get(Aring, (int64_t)nK * g.nbc)) != cudaSuccess) return e;
  {
    // sines and decay tables, for the length of this block
    std::vector<double> sn(2 * (size_t)(nx + ny));
    for (int i = 0; i < 2 * nx; ++i) sn[i] = sin_pi(i, nx);
    for (int i = 0; i < 2 * ny; ++i) sn[2 * nx + i] = sin_pi(i, ny);
    double* d = nullptr;
    const int64_t ngx = (int64_t)Kx * nrow, nhy = (int64_t)Ky * ncol;
    if ((e = cudaMalloc(&d, sizeof(double) * ((int64_t)sn.size() + ngx + nhy))) != cudaSuccess) return e;
    double *snx = d, *sny = d + 2 * nx, *gx = sny + 2 * ny, *hy = gx + ngx;
    e = cudaMemcpy(d, sn.data(), sizeof(double) * sn.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
      // (on a long, narrow grid no mode of the short sides reaches the quarter lines)
      if (Kx > 0) {
        k_modes<<<dim3((ncol + 127) / 128, Kx), 128>>>(nx, snx, St);
        k_decay<<<dim3((nrow + 63) / 64, Kx), 64>>>(ny, mult, nrow, 1, sny, gx);
      }
      if (Ky > 0) {
        k_modes<<<dim3((nrow + 127) / 128, Ky), 128>>>(ny, sny, St + (int64_t)Kx * ncol);
        k_decay<<<dim3((ncol + 63) / 64, Ky), 64>>>(nx, mult, 1, nrow, snx, hy);
      }
      k_ring_response<<<dim3((g.nbc + 127) / 128, nK), 128>>>(g, pts, St, Kx, Ky, gx, hy, Aring);
      e = cudaGetLastError();
    }
    const cudaError_t es = cudaStreamSynchronize(nullptr);  // the handle's stream does not wait for this one
    cudaFree(d);
    if (e == cudaSuccess) e = es;
    if (e != cudaSuccess) return e;
  }
  auto zero = [&](auto*& dst, int64_t n) -> cudaError_t {
    cudaError_t e2 = get(dst, n);
    if (e2 == cudaSuccess) e2 = cudaMemset(dst, 0, sizeof(*dst) * n);
    return e2;
  };
  if ((e = zero(vrow, (int64_t)L * 2 * ncol)) != cudaSuccess) return e;
  if ((e = zero(ucolp, (int64_t)L * 2 * nchunk * nrow)) != cudaSuccess) return e;
  if ((e = zero(ucol, (int64_t)L * 2 * nrow)) != cudaSuccess) return e;
  if ((e = zero(dring, (int64_t)L * g.nbc)) != cudaSuccess) return e;
  if ((e = zero(qline, (int64_t)L * qls)) != cudaSuccess) return e;
  if ((e = zero(sidex, (int64_t)L * 2 * ncol)) != cudaSuccess) return e;
  if ((e = zero(sidey, (int64_t)L * 2 * nrow)) != cudaSuccess) return e;
  if ((e = zero(ringd, (int64_t)L * g.nbc)) != cudaSuccess) return e;
  if ((e = zero(coef, (int64_t)L * nK)) != cudaSuccess) return e;
  return cudaStreamSynchronize(nullptr);
}

void RingPlan::release() {
  for (void* p : {(void*)St, (void*)Aring, (void*)pts, (void*)vrow, (void*)ucolp, (void*)ucol, (void*)qline,
                  (void*)sidex, (void*)sidey, (void*)ringd, (void*)dring, (void*)coef, (void*)qfx, (void*)side,
                  (void*)sinx, (void*)siny, (void*)Apow})
    if (p) cudaFree(p);
  St = nullptr; Aring = nullptr; pts = nullptr; vrow = nullptr; ucolp = nullptr; ucol = nullptr; qline = nullptr;
  sidex = nullptr; sidey = nullptr; ringd = nullptr; dring = nullptr; coef = nullptr;
  qfx = side = sinx = siny = Apow = nullptr;
  bytes = 0;
}

}  // namespace ib
