// FP64 transforms in fixed point: the kernels of plan class 1 (see transforms_fix.cuh).
#include "transforms_fix.cuh"

namespace owt {
FxXformKernels fx_xform_kernels1(int L) { return fx_kernels_of_class<1>(L); }
}  // namespace owt
