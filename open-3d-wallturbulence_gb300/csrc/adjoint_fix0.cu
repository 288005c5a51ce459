// The Lamb vector's adjoint in fixed point: the kernels of plan class 0 (see adjoint_fix.cuh).
#include "adjoint_fix.cuh"

namespace owt {
FxAdjKernels fx_adj_kernels0(int L) { return fx_adj_kernels_of_class<0>(L); }
}  // namespace owt
