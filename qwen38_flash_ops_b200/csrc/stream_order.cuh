// Stream order of kernels that are launched before the kernel ahead of them in the stream has quite ended.
//
// A call of this library is 5 to 20 us, and an ordinary launch waits until its predecessor's end has travelled through the
// front end: back to back, calls ended on multiples of 2.05 us.  With the attribute that allows programmatic launches, and no
// trigger in the predecessor, blocks are placed when the last block of the predecessor leaves, set themselves up, and wait for
// its writes in GridDependencyWait.  Eager calls back to back on one B200, ordinary launch -> this: BF16 5120 x 5120, one row,
// 12.3 -> 10.6 us; NVFP4 17408 x 5120, four rows, 18.4 -> 16.3; shared expert 640 x 2560 8.2 -> 6.8; argmax 64 x 151936 8.2 -> 5.1.
// A call that finds the GPU idle gains nothing by it, and loses nothing (gate and up 43.5 us until the host has waited, 43.5 to 44.0; the head 108.4, 107.8).
// No gain, not done: fetching the first weights to L2 before the wait (BF16 10.6 -> 10.8 to 12.0 us, the more the slower),
// releasing the next kernel behind the K loop without being asked to (10.6 -> 12.3).
#pragma once

#include <cuda_runtime.h>

namespace qfg {

// Every thread of such a kernel comes here before its first access to global memory, whatever it is launched with: the
// predecessor may be writing anything the call reads, its weights included.  Two things are read earlier, by the few-row kernel: w_scale,
// which a node uploads when it is created and no kernel writes, and with pdl_wait, which says that they may be, the first
// weights.  Without the attribute it returns at once.
__device__ __forceinline__ void GridDependencyWait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void GridLaunchDependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// An address for loads behind that wait.  Non-coherent loads (__ldg) count as loads of constants, which a compiler may move
// past it; through this address they come after it.
template <typename T>
__device__ __forceinline__ const T* BehindWait(const T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}

// Not while the stream is being captured: the edges of a graph stay the plain ones that every call on graphs takes, and its
// kernels follow one another that closely anyway (30 calls in a graph, BF16 5120 x 5120: 10.75 us each either way).
inline bool MayOverlapPredecessor(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusActive;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
    cudaGetLastError();  // the launch itself meets the error, if there is one
    return false;
  }
  return status == cudaStreamCaptureStatusNone;
}

inline cudaLaunchAttribute OverlapAttribute() {
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

}  // namespace qfg
