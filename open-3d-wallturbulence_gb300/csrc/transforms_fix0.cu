// FP64 transforms in fixed point: the kernels of plan class 0 (see transforms_fix.cuh).
#include "transforms_fix.cuh"

namespace owt {
FxXformKernels fx_xform_kernels0(int L) { return fx_kernels_of_class<0>(L); }
}  // namespace owt
