// Entry points of the tensor-core forward (ndc_tc.cu) for the ABI unit.
#pragma once

#include "ndc_common.cuh"

namespace ndc {
namespace tc {

// Whether the tensor-core kernels take this geometry and are the faster ones for it: for `forward`, or for `backward_ratio`.
bool covers(const Geo& g, bool ratio);
cudaError_t forward(const Geo& g, const __nv_bfloat16* x, const __nv_bfloat16* z, const float* h, const float* bias,
                    __nv_bfloat16* out, __nv_bfloat16* t1, cudaStream_t st);
// First step of the backward: gnum, gden (two tensors, or (gden, gnum) pairs at `gnum`) and the direct term,
// as ratio_kernel writes them.
cudaError_t backward_ratio(const Geo& g, const __nv_bfloat16* x, const __nv_bfloat16* z, const __nv_bfloat16* t1, const float* h,
                           const float* bias, const __nv_bfloat16* gout, float* gnum, float* gden, __nv_bfloat16* direct,
                           bool pairs, cudaStream_t st);
// Non-zero once a kernel's bounded wait has run out on the current device (synchronises).
unsigned wait_expired();
// The same for launches that are known to have run by now, without synchronising; true once for each.
bool take_expired();
// Launches one wait that runs out after `limit_us` (up to a second).
cudaError_t probe_wait(unsigned limit_us, cudaStream_t st);

}  // namespace tc
}  // namespace ndc
