// The Lamb vector's adjoint in fixed point: the kernels of plan class 1 (see adjoint_fix.cuh).
#include "adjoint_fix.cuh"

namespace owt {
FxAdjKernels fx_adj_kernels1(int L) { return fx_adj_kernels_of_class<1>(L); }
}  // namespace owt
