// Internal interface between the C-ABI layer and the resident-cluster kernel (see resident.cu).
#pragma once

#include <cuda_runtime.h>

#include "../../include/dlr_b200.h"

namespace dlr {

bool resident_supported(int d, int r);
// Estimated time of a forward of M rows, from measured times per layer, and (optionally) how it would be launched; 1e30
// where the kernel does not apply.  `terms`: with operands of 24 bits instead of bf16 ones.
double resident_estimate_us(int M, int d, int r, int L, bool terms, int smem_optin, dlrb200_plan* plan);
int resident_forward(void* encode_fn_ptr, const void* x, void* y, const void* Vp, const void* Up, int M, int d, int r,
                     int L, float eps, bool terms, int* status_dev, cudaStream_t stream, int smem_optin,
                     unsigned int spin_limit);

}  // namespace dlr
