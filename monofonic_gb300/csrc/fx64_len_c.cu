// Fixed-point transforms of the lengths 288, 384, 512 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template cudaError_t launch_len<288>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<384>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<512>(FxOp, const void *, dim3, cudaStream_t);
}  // namespace fx
