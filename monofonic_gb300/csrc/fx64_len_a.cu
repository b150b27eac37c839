// Fixed-point transforms of the lengths 16, 24, 32, 48, 64, 72, 96 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template cudaError_t launch_len<16>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<24>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<32>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<48>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<64>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<72>(FxOp, const void *, dim3, cudaStream_t);
template cudaError_t launch_len<96>(FxOp, const void *, dim3, cudaStream_t);
}  // namespace fx
