// ckt_batch_exact_few.cu -- persistent batched kernels, EXACT arithmetic,
// circuits of fewer than kFreeSteps steps.
#include "ckt_batch_inst.cuh"

namespace ckt {
BatchKernelFn batch_kernel_exact_few(int block, int wpt, int dcs) {
  CKT_BATCH_TABLE(CKT_MODE_EXACT, false)
}
}  // namespace ckt
