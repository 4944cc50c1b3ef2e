// The fixed-point passes of every eighth length (kernels in dstfx.cuh).
#include "dstfx.cuh"

namespace ib::fxp {
#define IB_FX_HERE(M) IB_FX_RUN(, M)
IB_FX_GROUP_7(IB_FX_HERE)
}  // namespace ib::fxp
