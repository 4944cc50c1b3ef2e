// The fixed-point sine-transform passes (FP64 and float-float lines): tables and entry points (kernels in
// dstfx.cuh, compiled by length in dstfx_1.cu ... dstfx_8.cu).
#include "dstfx.cuh"

#include <cmath>
#include <vector>

namespace ib {

namespace fxp {
#define IB_FX_EXTERN(M) IB_FX_RUN(extern, M)
IB_FX_LENGTHS(IB_FX_EXTERN)
}  // namespace fxp

cudaError_t FxTables::build(int n) {
  release();
  if (!dst_axis_supported(n)) return cudaErrorInvalidValue;
  const int M = n / 2;
  d = FxAxis{};
  d.n = n;
  d.M = M;
  const fxp::Radices p = fxp::radices(M);
  const long double pi = 3.141592653589793238462643383279502884L;
  auto split = [](long double w) {
    const long long v = llrintl(w * (long double)(1LL << 60));
    const int h = (int)((v + (1LL << 29)) >> 30);
    return fx::wgt{h, (int)(v - h * (1LL << 30))};
  };
  auto cis = [&](long double num, long double den) {  // e^{-2 pi i num / den}
    const long double ang = -2.0L * pi * num / den;
    const fx::wgt c = split(cosl(ang)), s = split(sinl(ang));
    return fx::cwgt{c.h, c.l, s.h, s.l};
  };
  std::vector<fx::cwgt> tw, post(M / 2 + 1);
  std::vector<fx::wgt> sn(M + 1);
  int Ns = 1;
  for (int st = 0; st < p.n; ++st) {
    const int R = p.r[st];
    d.twoff[st] = (int)tw.size();
    if (st > 0)
      for (int r = 1; r < R; ++r)
        for (int k = 0; k < Ns; ++k) tw.push_back(cis((long double)(r * k), (long double)(Ns * R)));
    Ns *= R;
  }
  for (int k = 0; k <= M / 2; ++k) post[k] = cis((long double)k, (long double)n);
  // 2 sin(pi j / n) < 2 for j < M
  for (int j = 0; j < M; ++j) sn[j] = split(2.0L * sinl(pi * (long double)j / (long double)n));
  const size_t btw = tw.size() * sizeof(fx::cwgt), bpost = post.size() * sizeof(fx::cwgt), bsn = sn.size() * sizeof(fx::wgt);
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  cudaError_t e = cudaMalloc(&mem, up(btw) + up(bpost) + up(bsn) + 256);
  if (e != cudaSuccess) { mem = nullptr; return e; }
  char* base = static_cast<char*>(mem);
  if (btw && (e = cudaMemcpy(base, tw.data(), btw, cudaMemcpyHostToDevice)) != cudaSuccess) return e;
  if ((e = cudaMemcpy(base + up(btw), post.data(), bpost, cudaMemcpyHostToDevice)) != cudaSuccess) return e;
  if ((e = cudaMemcpy(base + up(btw) + up(bpost), sn.data(), bsn, cudaMemcpyHostToDevice)) != cudaSuccess) return e;
  d.tw = reinterpret_cast<const fx::cwgt*>(base);
  d.post = reinterpret_cast<const fx::cwgt*>(base + up(btw));
  d.sin2 = reinterpret_cast<const fx::wgt*>(base + up(btw) + up(bpost));
  return cudaSuccess;
}

void FxTables::release() {
  if (mem) cudaFree(mem);
  mem = nullptr;
}

template <typename T>
cudaError_t fx_fwd(const Geometry& g, const FxAxis& ax, const T* in, double* out, int batch, const T* bc,
                   cudaStream_t s) {
  if (ax.n != g.nx) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassXPass, s);
  switch (ax.M) {
#define IB_FX_CASE(M) \
  case M: return fxp::run_fwd<M, T>(g, ax, in, out, batch, bc, s);
    IB_FX_LENGTHS(IB_FX_CASE)
#undef IB_FX_CASE
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t fx_ypass(const Geometry& g, const FxAxis& ay, const double* in, double* out, int batch, const double* mult,
                     int64_t mstride, int log2scale, cudaStream_t s) {
  if (ay.n != g.ny) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassYPass, s);
  switch (ay.M) {
#define IB_FX_CASE(M) \
  case M: return fxp::run_y<M>(g, ay, in, out, batch, mult, mstride, log2scale, s);
    IB_FX_LENGTHS(IB_FX_CASE)
#undef IB_FX_CASE
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t fx_yspec(const Geometry& g, const FxAxis& ay, double* w, int batch, const double* mult, double* qrow,
                     int64_t qls, cudaStream_t s) {
  if (ay.n != g.ny) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassYPass, s);
  switch (ay.M) {
#define IB_FX_CASE(M) \
  case M: return fxp::run_yspec<M>(g, ay, w, batch, mult, qrow, qls, s);
    IB_FX_LENGTHS(IB_FX_CASE)
#undef IB_FX_CASE
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t fx_yring(const Geometry& g, const FxAxis& ay, const double* w, double* out, int batch, const double* mult,
                     const FxRings& r, cudaStream_t s) {
  if (ay.n != g.ny) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassYPass, s);
  switch (ay.M) {
#define IB_FX_CASE(M) \
  case M: return fxp::run_yring<M>(g, ay, w, out, batch, mult, r, s);
    IB_FX_LENGTHS(IB_FX_CASE)
#undef IB_FX_CASE
    default: return cudaErrorInvalidValue;
  }
}

template <typename T>
cudaError_t fx_inv(const Geometry& g, const FxAxis& ax, const double* in, T* out, int batch, const T* sub_from,
                   cudaStream_t s) {
  if (ax.n != g.nx) return cudaErrorInvalidValue;
  if (batch <= 0) return cudaSuccess;
  ProfScope prof(kClassXPass, s);
  switch (ax.M) {
#define IB_FX_CASE(M) \
  case M: return fxp::run_inv<M, T>(g, ax, in, out, batch, sub_from, s);
    IB_FX_LENGTHS(IB_FX_CASE)
#undef IB_FX_CASE
    default: return cudaErrorInvalidValue;
  }
}

template cudaError_t fx_fwd<double>(const Geometry&, const FxAxis&, const double*, double*, int, const double*, cudaStream_t);
template cudaError_t fx_fwd<df64>(const Geometry&, const FxAxis&, const df64*, double*, int, const df64*, cudaStream_t);
template cudaError_t fx_inv<double>(const Geometry&, const FxAxis&, const double*, double*, int, const double*, cudaStream_t);
template cudaError_t fx_inv<df64>(const Geometry&, const FxAxis&, const double*, df64*, int, const df64*, cudaStream_t);

}  // namespace ib
