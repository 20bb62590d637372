// The FP64 kernels with 64 threads a CTA (bse_kernels.cuh).
#include "bse_kernels.cuh"

namespace dga {

DGA_FP64_KERNELS(template, 64)

}  // namespace dga
