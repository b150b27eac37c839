// Fixed-point transforms of the lengths 576, 768, 1152 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template cudaError_t launch_len<576>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<768>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<1152>(FxOp, const void *, dim3, cudaStream_t);
}  // namespace fx
