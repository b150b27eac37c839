// Launches of the pipeline's kernels with programmatic stream serialisation: the
// next kernel of the stream is set up, and its prologue runs, while the previous
// one drains.  A kernel launched so calls pdl_begin() (or load_tw of fused.cuh)
// before it touches anything that an earlier kernel writes or reads: every one
// of its threads waits there until all earlier kernels of the stream have
// completed, so the order of memory accesses is that of a plain launch.
// On small grids the gap between two dependent kernels was 2.7 us, half as long as
// a kernel: a 32^3 2LPT pass of nine launches went from 70 to 59 us, a 64^3 3LPT
// one of 35 from 301 to 226 us.  When it is used: pdl_rule in engine.cu.
#pragma once
#include <cuda_runtime.h>

namespace mfx {

// lets the next kernel start its prologue
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }
// waits for the earlier kernels of the stream
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_trigger();
  pdl_wait();
}

// whether the calling thread's launches may overlap their predecessors' ends
inline bool &pdl_enabled() {
  static thread_local bool on = true;
  return on;
}

// Inside a stream capture the launch is a plain one: a graph's own edges have a
// gap of 0.6 us already.
template <class... P, class... A>
inline void launch_pdl(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A &&...args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (pdl_enabled() && cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
    c.attrs = &at;
    c.numAttrs = 1;
  }
  cudaLaunchKernelEx(&c, kernel, static_cast<A &&>(args)...);
}

}  // namespace mfx
