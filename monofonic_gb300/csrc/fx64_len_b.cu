// Fixed-point transforms of the lengths 128, 144, 192, 256 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template cudaError_t launch_len<128>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<144>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<192>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<256>(FxOp, const void *, dim3, cudaStream_t);
}  // namespace fx
