// Stencil kernels of the stream-function discretisation.
//
// Each kernel restates one operator of src/streamfcn/fluid-ops.jl (cited per kernel) on the
// reference's own column-major layouts.  Grid-stride loops, one thread per output value.
#include "ib_common.cuh"

namespace ib {

namespace {

constexpr int kThreads = 256;

inline int blocks_for(int64_t n) {
  int64_t b = (n + kThreads - 1) / kThreads;
  if (b > 65535LL * 8) b = 65535LL * 8;
  return (int)(b < 1 ? 1 : b);
}

// x * s for a power of two s: exact, so a float-float value scales part by part (the general
// float-float product would spend ~7 FP32 operations on it)
template <typename T>
__device__ __forceinline__ T xscale(T x, float s) {
  return x * T(s);
}
template <>
__device__ __forceinline__ df64 xscale<df64>(df64 x, float s) {
  return df64(x.hi * s, x.lo * s);
}

// get_bc! value at ring index idx (fluid-ops.jl:210-239), including the final *0.25.
template <typename T>
__device__ __forceinline__ T ring_value(const Geometry& g, const T* __restrict__ r, int idx) {
  const int nx = g.nx, ny = g.ny, ncol = nx - 1;
  const int nx4 = nx / 4, ny4 = ny / 4;
  T v;
  if (idx < g.B) {  // left (idx < R) or right block, node along y
    const bool right = idx >= g.R;
    const int jb = idx - (right ? g.R : g.L);
    const int col = right ? 3 * nx4 - 1 : nx4 - 1;
    if ((jb & 1) == 0) {
      const int t = jb >> 1;
      v = r[(ny4 - 1 + t) * ncol + col];
    } else {
      const int t = (jb + 1) >> 1;
      v = xscale(r[(ny4 - 1 + t) * ncol + col] + r[(ny4 - 2 + t) * ncol + col], 0.5f);
    }
  } else {  // bottom (idx < T) or top block, node along x
    const bool top = idx >= g.T;
    const int ib = idx - (top ? g.T : g.B);
    const int row = top ? 3 * ny4 - 1 : ny4 - 1;
    if ((ib & 1) == 0) {
      const int t = ib >> 1;
      v = r[row * ncol + nx4 - 1 + t];
    } else {
      const int t = (ib + 1) >> 1;
      v = xscale(r[row * ncol + nx4 - 1 + t] + r[row * ncol + nx4 - 2 + t], 0.5f);
    }
  }
  return xscale(v, 0.25f);
}

template <typename T>
__global__ void k_get_bc(Geometry g, const T* __restrict__ r, T* __restrict__ bc, int batch, T extra) {
  pdl_begin();
  const int64_t total = (int64_t)batch * g.nbc;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int b = (int)(t / g.nbc), idx = (int)(t - (int64_t)b * g.nbc);
    bc[t] = ring_value(g, r + (int64_t)b * g.nG, idx) * extra;
  }
}

// apply_bc! (fluid-ops.jl:249-275): rows first, then columns (same order as the reference).
template <typename T>
__global__ void k_apply_bc_rows(Geometry g, T* __restrict__ r, const T* __restrict__ bc, T fac, int batch) {
  pdl_begin();
  const int ncol = g.nx - 1, nrow = g.ny - 1;
  const int64_t total = (int64_t)batch * ncol;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int b = (int)(t / ncol), I = (int)(t - (int64_t)b * ncol);
    T* rr = r + (int64_t)b * g.nG;
    const T* bb = bc + (int64_t)b * g.nbc;
    rr[I] += fac * bb[g.B + 1 + I];
    rr[(nrow - 1) * ncol + I] += fac * bb[g.T + 1 + I];
  }
}
template <typename T>
__global__ void k_apply_bc_cols(Geometry g, T* __restrict__ r, const T* __restrict__ bc, T fac, int batch) {
  pdl_begin();
  const int ncol = g.nx - 1, nrow = g.ny - 1;
  const int64_t total = (int64_t)batch * nrow;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int b = (int)(t / nrow), J = (int)(t - (int64_t)b * nrow);
    T* rr = r + (int64_t)b * g.nG;
    const T* bb = bc + (int64_t)b * g.nbc;
    rr[J * ncol] += fac * bb[g.L + 1 + J];
    rr[J * ncol + ncol - 1] += fac * bb[g.R + 1 + J];
  }
}

// coarsify! (fluid-ops.jl:184-202)
template <typename T>
__global__ void k_coarsify(Geometry g, T* __restrict__ gc, const T* __restrict__ gf, int batch, int64_t stride) {
  pdl_begin();
  const int ncol = g.nx - 1;
  const int ct = g.nx / 2 - 1, cs = g.ny / 2 - 1;  // coarse centre extent
  const int per = ct * cs;  // batch * per < 2^31 (batch <= 64 slots of at most 4095^2 / 4 values)
  const int total = batch * per;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const int b = t / per;
    const int rem = t - b * per;
    const int s = rem / ct, tt = rem - s * ct;
    const T* f = gf + (int64_t)b * stride;
    const int J = 2 * s + 1, I = 2 * tt + 1;
    const int c = J * ncol + I;
    const T v = f[c]
                + xscale(f[c + 1] + f[c + ncol] + f[c - 1] + f[c - ncol], 0.5f)
                + xscale(f[c + ncol + 1] + f[c - ncol + 1] + f[c - ncol - 1] + f[c + ncol - 1], 0.25f);
    gc[(int64_t)b * stride + (int64_t)(g.ny / 4 + s) * ncol + g.nx / 4 + tt] = v;
  }
}

// Multilevel curl! (fluid-ops.jl:138-182); bc == nullptr means a zero ring.  A thread takes kCurlRows
// rows of one column of nodes and the column to its right: its own column's values make the qx of the
// column and, against the right one (which its neighbour loads too), the qy.  The thread of the last
// column also has qx of the boundary to its right, the last strip the top row of qy.
//
// Bound by memory (24 bytes a node), in FP64 also by its two operations a node.  Measured against one
// thread per flux value: 1024^2 x 4 levels, FP64 45 -> 24 us, float-float 46 -> 16.5; 2048^2 x 5 199 -> 77.
// (2 rows a thread: 23, 21, 88; 8: 25, 17, 76 and more on small grids.)
constexpr int kCurlX = 128, kCurlRows = 4;
template <typename T>
__global__ void __launch_bounds__(kCurlX)
k_curl(Geometry g, const T* __restrict__ psi, const T* __restrict__ bc, T* __restrict__ q) {
  pdl_begin();
  const int nx = g.nx, ny = g.ny, ncol = nx - 1;
  const int I = blockIdx.x * kCurlX + threadIdx.x, J0 = blockIdx.y * kCurlRows, b = blockIdx.z;
  if (I >= nx) return;
  const T* p = psi + (int64_t)b * g.nG;
  const T* c = bc ? bc + (int64_t)b * g.nbc : nullptr;
  T* qx = q + (int64_t)b * g.nq + (int64_t)J0 * (nx + 1) + I;
  T* qy = q + (int64_t)b * g.nq + g.nu + (int64_t)J0 * nx + I;
  auto ring = [&](int i) -> T { return c ? c[i] : T(0); };
  T l[kCurlRows + 1], r[kCurlRows + 1];  // nodes (J0 + u, I), (J0 + u, I + 1)
  if (I > 0 && I < nx - 1 && J0 > 0 && J0 + kCurlRows < ny) {
    const T* n = p + (J0 - 1) * ncol + I - 1;
#pragma unroll
    for (int u = 0; u <= kCurlRows; ++u) l[u] = n[u * ncol];
#pragma unroll
    for (int u = 0; u < kCurlRows; ++u) r[u] = n[u * ncol + 1];
#pragma unroll
    for (int u = 0; u < kCurlRows; ++u) {
      qx[u * (nx + 1)] = l[u + 1] - l[u];
      qy[u * nx] = l[u] - r[u];
    }
    return;
  }
  auto node = [&](int j, int i) -> T {
    if (i == 0) return ring(g.L + j);
    if (i == nx) return ring(g.R + j);
    if (j == 0) return ring(g.B + i);
    if (j == ny) return ring(g.T + i);
    return p[(j - 1) * ncol + i - 1];
  };
#pragma unroll
  for (int u = 0; u <= kCurlRows; ++u) {
    l[u] = r[u] = T(0);
    if (J0 + u <= ny) {
      l[u] = node(J0 + u, I);
      r[u] = node(J0 + u, I + 1);
    }
  }
#pragma unroll
  for (int u = 0; u < kCurlRows; ++u) {
    if (J0 + u >= ny) break;
    qx[u * (nx + 1)] = l[u + 1] - l[u];
    if (I == nx - 1) qx[u * (nx + 1) + 1] = r[u + 1] - r[u];
    // (the ring's corners belong to its rows here)
    qy[u * nx] = J0 + u == 0 ? ring(g.B + I) - ring(g.B + I + 1) : l[u] - r[u];
  }
  if (J0 + kCurlRows >= ny) qy[(ny - J0) * nx] = ring(g.T + I) - ring(g.T + I + 1);
}

// rot! = C^T (fluid-ops.jl:117-129)
template <typename T>
__global__ void k_rot(Geometry g, const T* __restrict__ q, T* __restrict__ gam, int batch) {
  const int nx = g.nx, ncol = nx - 1;
  const int64_t total = (int64_t)batch * g.nG;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int b = (int)(t / g.nG), e = (int)(t - (int64_t)b * g.nG);
    const int J = e / ncol, I = e - J * ncol;
    const T* qx = q + (int64_t)b * g.nq;
    const T* qy = qx + g.nu;
    gam[t] = (qx[J * (nx + 1) + I + 1] - qx[(J + 1) * (nx + 1) + I + 1])
             + (qy[(J + 1) * nx + I + 1] - qy[(J + 1) * nx + I]);
  }
}

// ---- nonlinear term + explicit right-hand side (cnab/ops.jl:151-167, fluid-ops.jl:277-401,
//      cnab/timestepping.jl:54-67) ----------------------------------------------------------
// Nonlinear term and CN right-hand side of every level (Nonlinear/RhsForce, timestepping.jl:
// 31-66; avg_flux! fluid-ops.jl:276-301, direct_product! :303-398, rot!).  With Qx, Qy the fluxes
// averaged to the nodes and G the circulation at the nodes (the ring on the boundary), the face
// products are fqx(j) = (Qy G)(j+1) + (Qy G)(j) and -fqy(i) = (Qx G)(i+1) + (Qx G)(i), up to exact
// factors; in rot the node's own products drop out, so that
//   N(j, i) = ((Qy G)(j-1) - (Qy G)(j+1) + (Qx G)(i-1) - (Qx G)(i+1)) / (4 hc^2).
// One block per tile of kNTY x kNTX cells: the products its cells share are formed once into shared
// memory, then each cell combines its four.
//
// FP64 is bound by its pipe (19 operations a cell; one takes 7 us at 1024^2 x 4 levels; 84% busy),
// float-float by instruction issue.  Measured there: FP64 325 us (averages, face products and combination,
// 30 operations a cell) -> 191 us -> 157 with the ring's edge terms under one branch of the block and the
// viscous term as two multiply-adds (predicated off, an FP64 instruction still takes its turn), float-float
// 111 -> 94 -> 92 us.  (4 rows a tile of 64: 164 and 94; 16 rows of 32: 156 and 98.)  A warp walking up its
// columns with the products in registers has fewer operations but waits for each row's loads.
constexpr int kNTX = 32, kNTY = 8;
template <typename T>
__global__ void __launch_bounds__(kNTX * kNTY) k_nonlin_rhs(Geometry g, NonlinArgs<T> a) {
  pdl_begin();
  __shared__ T sM[kNTY + 2][kNTX];  // 2 Qy G at nodes (J0 + r, I0 + 1 + c)
  __shared__ T sN[kNTY][kNTX + 2];  // 2 Qx G at nodes (J0 + 1 + r, I0 + c)
  __shared__ T sK[7];               // the level's 2 q0x, 2 q0y, 1/(4 hc^2), alpha; dt beta0, dt beta1; 1 - 4 alpha
  const int nx = g.nx, ny = g.ny, ncol = nx - 1, nrow = ny - 1, l = blockIdx.z;
  const int J0 = blockIdx.y * kNTY, I0 = blockIdx.x * kNTX, tid = threadIdx.x;
  const T* __restrict__ qx = a.q + (int64_t)l * g.nq;
  const T* __restrict__ qy = qx + g.nu;
  const T* __restrict__ G = a.gamma + (int64_t)l * g.nG;
  const T* __restrict__ bc = a.bcn + (int64_t)l * g.nbc;
  // the level's constants, converted once per block (a double-to-float-float conversion costs
  // FP64 operations, which GB300 runs at 1/64 of its FP32 rate)
  if (tid < 7) {
    sK[tid] = (T)(tid == 0 ? 2.0 * a.q0[2 * l]
                : tid == 1 ? 2.0 * a.q0[2 * l + 1]
                : tid == 2 ? 0.25 * a.inv_hc2[l]
                : tid == 3 ? (a.alpha ? a.alpha[l] : 0.0)
                : tid == 4 ? a.dtb0
                : tid == 5 ? a.dtb1 : (a.alpha ? 1.0 - 4.0 * a.alpha[l] : 1.0));
  }
  __syncthreads();
  // circulation at node (j, i) next to the interior, the ring on the boundary
  auto node = [&](int j, int i) -> T {
    if (j == 0) return bc[g.B + i];
    if (j == ny) return bc[g.T + i];
    if (i == 0) return bc[g.L + j];
    if (i == nx) return bc[g.R + j];
    return G[(j - 1) * ncol + i - 1];
  };
  for (int k = tid; k < (kNTY + 2) * kNTX; k += kNTX * kNTY) {
    const int r = k / kNTX, c = k % kNTX, j = J0 + r, i = I0 + 1 + c;
    if (j <= ny && i <= nx - 1) sM[r][c] = ((qy[j * nx + i] + qy[j * nx + i - 1]) + sK[1]) * node(j, i);
  }
  for (int k = tid; k < kNTY * (kNTX + 2); k += kNTX * kNTY) {
    const int r = k / (kNTX + 2), c = k % (kNTX + 2), j = J0 + 1 + r, i = I0 + c;
    if (j <= ny - 1 && i <= nx) sN[r][c] = ((qx[j * (nx + 1) + i] + qx[(j - 1) * (nx + 1) + i]) + sK[0]) * node(j, i);
  }
  __syncthreads();
  const int cr = tid / kNTX, cc = tid % kNTX, J = J0 + cr, I = I0 + cc;
  if (J >= nrow || I >= ncol) return;
  const int64_t t = (int64_t)l * g.nG + (int64_t)J * ncol + I;
  const T nl = ((sM[cr][cc] - sM[cr + 2][cc]) + (sN[cr][cc] - sN[cr][cc + 2])) * sK[2];
  a.nl_new[t] = nl;
  T r = sK[4] * nl + sK[5] * a.nl_old[t];
  if (a.alpha) {
    // A_l gamma = gamma - alpha_l (4 gamma - neighbours), zero outside the array
    const T* p = G + J * ncol + I;
    const T gc = *p;
    const T gl = I > 0 ? p[-1] : T(0), gr = I < ncol - 1 ? p[1] : T(0);
    const T gd = J > 0 ? p[-ncol] : T(0), gu = J < nrow - 1 ? p[ncol] : T(0);
    const T nb = (gl + gr) + (gd + gu);
    if constexpr (std::is_same<T, double>::value) r = fma(sK[3], nb, fma(sK[6], gc, r));
    else r = (gc - sK[3] * (xscale(gc, 4.0f) - nb)) + r;
  }
  // (one branch of the whole block: four predicated additions would cost every warp their issue)
  if (J0 == 0 || J0 + kNTY >= nrow || I0 == 0 || I0 + kNTX >= ncol) {
    const T* ed = a.edges + (int64_t)l * (2 * ncol + 2 * nrow);
    if (J == 0) r += ed[I];
    if (J == nrow - 1) r += ed[ncol + I];
    if (I == 0) r += ed[2 * ncol + J];
    if (I == ncol - 1) r += ed[2 * ncol + nrow + J];
  }
  a.rhs[t] = r;
}

// Rings of the trial step (cnab/timestepping.jl:42-57): bcn[l] = 0.25 * get_bc(gamma[l+1]) for
// l < nlev-1 (zero on the coarsest level) and the accumulated rhsbc edge vectors
// edges[l] = sum_{l' = l}^{nlev-2} fac[l'] * get_bc(gamma[l'+1]) on the four edges.
template <typename T>
__global__ void k_trial_rings(Geometry g, const T* __restrict__ gamma, T* __restrict__ bcn, T* __restrict__ edges,
                              const double* __restrict__ fac, int accumulate) {
  pdl_begin();
  const int ncol = g.nx - 1, nrow = g.ny - 1;
  const int ne = 2 * ncol + 2 * nrow;
  const int nl = g.nlev;
  const int64_t nb_total = (int64_t)nl * g.nbc;
  const int64_t total = nb_total + (int64_t)nl * ne;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    if (t < nb_total) {
      const int l = (int)(t / g.nbc), idx = (int)(t - (int64_t)l * g.nbc);
      bcn[t] = (l < nl - 1) ? xscale(ring_value(g, gamma + (int64_t)(l + 1) * g.nG, idx), 0.25f) : T(0);
    } else {
      const int64_t u = t - nb_total;
      const int l = (int)(u / ne), e = (int)(u - (int64_t)l * ne);
      int ridx;
      if (e < ncol) ridx = g.B + 1 + e;
      else if (e < 2 * ncol) ridx = g.T + 1 + (e - ncol);
      else if (e < 2 * ncol + nrow) ridx = g.L + 1 + (e - 2 * ncol);
      else ridx = g.R + 1 + (e - 2 * ncol - nrow);
      T acc = T(0);
      if (accumulate) {
        for (int lp = nl - 2; lp >= l; --lp) acc += (T)fac[lp] * ring_value(g, gamma + (int64_t)(lp + 1) * g.nG, ridx);
      } else if (l < nl - 1) {
        acc = (T)fac[l] * ring_value(g, gamma + (int64_t)(l + 1) * g.nG, ridx);
      }
      edges[u] = acc;
    }
  }
}

// One Runge-Kutta-Chebyshev stage, elementwise over n values:
//   Y = a0 Y0 + a1 Ym1 + a2 Ym2 + c1 (G - Ym1) + c0 F0,   G = Ym1 + F(Ym1)
// (Ym2 may be null when a2 = 0; Y may alias Ym2).  With store_f0, F0 = G - Ym1 is also written.
__global__ void k_rkc_stage(int64_t n, double* __restrict__ Y, const double* __restrict__ Y0, const double* Ym1,
                            const double* Ym2, const double* __restrict__ G, double* F0, double a0, double a1,
                            double a2, double c1, double c0, int store_f0) {
  pdl_begin();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double ym1 = Ym1[i];
    const double f = G[i] - ym1;
    if (store_f0) F0[i] = f;
    double y = a0 * Y0[i] + a1 * ym1 + c1 * f;
    if (Ym2) y += a2 * Ym2[i];
    if (!store_f0) y += c0 * F0[i];
    Y[i] = y;
  }
}

template <typename T>
__global__ void k_fill(T* p, T v, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) p[t] = v;
}
template <typename T>
__global__ void k_axpby(T* y, const T* x, T a, T b, int64_t n) {
  pdl_begin();
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    y[t] = a * x[t] + b * y[t];
}

}  // namespace

template <typename T>
cudaError_t get_bc(const Geometry& g, const T* r, T* bc, int batch, T extra, cudaStream_t s) {
  return launch_k(k_get_bc<T>, dim3(blocks_for((int64_t)batch * g.nbc)), dim3(kThreads), 0, s, g, r, bc, batch, extra);
}
template <typename T>
cudaError_t apply_bc(const Geometry& g, T* r, const T* bc, T fac, int batch, cudaStream_t s) {
  cudaError_t e = launch_k(k_apply_bc_rows<T>, dim3(blocks_for((int64_t)batch * (g.nx - 1))), dim3(kThreads), 0, s, g, r, bc, fac, batch);
  if (e != cudaSuccess) return e;
  return launch_k(k_apply_bc_cols<T>, dim3(blocks_for((int64_t)batch * (g.ny - 1))), dim3(kThreads), 0, s, g, r, bc, fac, batch);
}
template <typename T>
cudaError_t coarsify(const Geometry& g, T* gc, const T* gf, int batch, int64_t stride, cudaStream_t s) {
  return launch_k(k_coarsify<T>, dim3(blocks_for((int64_t)batch * (g.nx / 2 - 1) * (g.ny / 2 - 1))), dim3(kThreads), 0, s, g, gc, gf, batch, stride);
}
template <typename T>
cudaError_t curl(const Geometry& g, const T* psi, const T* bc, T* q, int batch, cudaStream_t s) {
  for (int b = 0; b < batch; b += 65535) {
    const dim3 grid((g.nx + kCurlX - 1) / kCurlX, (g.ny + kCurlRows - 1) / kCurlRows, std::min(batch - b, 65535));
    const cudaError_t e = launch_k(k_curl<T>, grid, dim3(kCurlX), 0, s, g, psi + (int64_t)b * g.nG,
                                   bc ? bc + (int64_t)b * g.nbc : nullptr, q + (int64_t)b * g.nq);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
template <typename T>
cudaError_t rot(const Geometry& g, const T* q, T* gam, int batch, cudaStream_t s) {
  k_rot<T><<<blocks_for((int64_t)batch * g.nG), kThreads, 0, s>>>(g, q, gam, batch);
  return cudaGetLastError();
}
template <typename T>
cudaError_t nonlin_rhs(const Geometry& g, const NonlinArgs<T>& a, cudaStream_t s) {
  ProfScope prof(kClassNonlin, s);
  const dim3 grid((g.nx - 1 + kNTX - 1) / kNTX, (g.ny - 1 + kNTY - 1) / kNTY, g.nlev);
  return launch_k(k_nonlin_rhs<T>, grid, dim3(kNTX * kNTY), 0, s, g, a);
}
template <typename T>
cudaError_t trial_rings(const Geometry& g, const T* gamma, T* bcn, T* edges, const double* fac, cudaStream_t s,
                        bool accumulate) {
  const int64_t n = (int64_t)g.nlev * g.nbc + (int64_t)g.nlev * (2 * (g.nx - 1) + 2 * (g.ny - 1));
  return launch_k(k_trial_rings<T>, dim3(blocks_for(n)), dim3(kThreads), 0, s, g, gamma, bcn, edges, fac,
                  accumulate ? 1 : 0);
}
cudaError_t rkc_stage(int64_t n, double* Y, const double* Y0, const double* Ym1, const double* Ym2, const double* G,
                      double* F0, double a0, double a1, double a2, double c1, double c0, bool store_f0, cudaStream_t s) {
  return launch_k(k_rkc_stage, dim3(blocks_for(n)), dim3(kThreads), 0, s, n, Y, Y0, Ym1, Ym2, G, F0, a0, a1, a2, c1, c0,
                  store_f0 ? 1 : 0);
}

template <typename T>
cudaError_t fill(T* p, T v, int64_t n, cudaStream_t s) {
  k_fill<T><<<blocks_for(n), kThreads, 0, s>>>(p, v, n);
  return cudaGetLastError();
}
template <typename T>
cudaError_t axpby(T* y, const T* x, T a, T b, int64_t n, cudaStream_t s) {
  return launch_k(k_axpby<T>, dim3(blocks_for(n)), dim3(kThreads), 0, s, y, x, a, b, n);
}

#define IB_INST(T)                                                                                   \
  template cudaError_t get_bc<T>(const Geometry&, const T*, T*, int, T, cudaStream_t);               \
  template cudaError_t apply_bc<T>(const Geometry&, T*, const T*, T, int, cudaStream_t);             \
  template cudaError_t coarsify<T>(const Geometry&, T*, const T*, int, int64_t, cudaStream_t);       \
  template cudaError_t curl<T>(const Geometry&, const T*, const T*, T*, int, cudaStream_t);          \
  template cudaError_t rot<T>(const Geometry&, const T*, T*, int, cudaStream_t);                     \
  template cudaError_t nonlin_rhs<T>(const Geometry&, const NonlinArgs<T>&, cudaStream_t);           \
  template cudaError_t trial_rings<T>(const Geometry&, const T*, T*, T*, const double*, cudaStream_t, bool); \
  template cudaError_t fill<T>(T*, T, int64_t, cudaStream_t);                                        \
  template cudaError_t axpby<T>(T*, const T*, T, T, int64_t, cudaStream_t);
IB_INST(double)
IB_INST(df64)
#undef IB_INST

}  // namespace ib
