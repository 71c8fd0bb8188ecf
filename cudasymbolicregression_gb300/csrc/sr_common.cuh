// sr_common.cuh -- host-side helpers shared by the C-ABI translation units.
#pragma once
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>

#include "../../include/sr_gb300.h"

namespace sr {

// Thread-local text of the last API-level failure (sr_last_error()).
void set_error(const char* fmt, ...);

inline int cuda_check(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return SR_OK;
  set_error("%s: %s", what, cudaGetErrorString(e));
  return SR_ERR_CUDA;
}

inline int launch_check(const char* what) { return cuda_check(cudaGetLastError(), what); }

// CTAs of a kernel that fit on an SM with this many threads and this much dynamic shared
// memory (cudaOccupancyMaxActiveBlocksPerMultiprocessor; 0 for an error).  The answers, facts
// of the kernel and the device, are kept in a table of fixed size: asking for the handful of
// shapes that a launch chooses from took longer than a small launch.
int resident_ctas(const void* kern, int threads, size_t smem);

int max_dyn_smem();  // dynamic shared memory that a block can have

// Lets a kernel be launched with `bytes` of dynamic shared memory: a kernel that needs more than
// it may take unasked is allowed all that a block can have beside static arrays of up to 1 KB.
// Never just `bytes`: the limit belongs to the kernel, and a call that set it to its own size
// could lower it under the launch of a larger call in another thread.
inline int allow_dynamic_smem(const void* kern, size_t bytes) {
  if (bytes <= 46 * 1024) return SR_OK;
  return cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem() - 1024),
                    "shared memory attribute");
}

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

__device__ __forceinline__ void report(int* status, int code) {
  if (code) atomicCAS(status, 0, code);
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace sr
