// Internal interface between the C-ABI layer and the weight-folding kernel (see fold.cu).
#pragma once

#include <cuda_runtime.h>

namespace dlr {

// V' = V * gain, U' = alpha * U for L layers whose tensors lie anywhere (arrays of L device addresses, in host memory) into
// the stacks Vp (L, r, d) and Up (L, d, r).  matrices_f32: V, U and the gains are fp32 (and rounded to bf16 first), else
// bf16.  alpha_f32: the scales are fp32, else bf16.  round_alpha: fp32 scales are rounded to bf16 first.
bool fold_layers(const void* const* V, const void* const* U, const void* const* gain, const void* const* alpha,
                 bool matrices_f32, bool alpha_f32, bool round_alpha, void* Vp, void* Up, int d, int r, int L,
                 cudaStream_t stream);

}  // namespace dlr
