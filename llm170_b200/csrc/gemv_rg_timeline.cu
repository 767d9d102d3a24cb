// The row-group GEMV kernels that stamp the diagnostic timeline.
#define RG_TIMELINE true
#include "gemv_rg_kernel.cuh"

namespace w4 {

const RgKernel* rg_timeline_kernels() { return rg_kernels; }

}  // namespace w4
