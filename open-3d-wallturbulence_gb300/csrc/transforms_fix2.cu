// FP64 transforms in fixed point: the kernels of plan class 2 (see transforms_fix.cuh).
#include "transforms_fix.cuh"

namespace owt {
FxXformKernels fx_xform_kernels2(int L) { return fx_kernels_of_class<2>(L); }
}  // namespace owt
