// The Lamb vector's adjoint in fixed point: the kernels of plan class 2 (see adjoint_fix.cuh).
#include "adjoint_fix.cuh"

namespace owt {
FxAdjKernels fx_adj_kernels2(int L) { return fx_adj_kernels_of_class<2>(L); }
}  // namespace owt
