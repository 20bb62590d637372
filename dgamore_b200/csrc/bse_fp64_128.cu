// The FP64 kernels with 128 threads a CTA (bse_kernels.cuh).
#include "bse_kernels.cuh"

namespace dga {

DGA_FP64_KERNELS(template, 128)

}  // namespace dga
