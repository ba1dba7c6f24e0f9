// gfe_internal.cuh -- shared host/device helpers of libgfe (status codes, error text, scratch).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "../../include/gfe.h"

namespace gfe {

// Record the message of a failure for gfe_last_error() on this host thread and return `code`.
int set_error(int code, const char* fmt, ...);

// Device-resident error word of the current device (lazily allocated once per device), or the
// word this host thread routed its kernels to (gfe_set_thread_error_word).
unsigned* device_error_word();
// The calling thread's override of the error word (nullptr: the per-device word), and its reset.
unsigned* thread_error_word();
void set_thread_error_word(unsigned* w);

// Stream-ordered scratch allocation; returns GFE_ERR_NOMEM with a message on failure.
int scratch_alloc(void** p, size_t bytes, cudaStream_t s, const char* what);
void scratch_free(void* p, cudaStream_t s);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Number of SMs of the current device (cached).
int sm_count();

// Stage timing (gfe_profile_enable): token = stage_begin(...); launch kernels; stage_end(...).
bool profiling();
void* stage_begin(int stage, cudaStream_t s);
void stage_end(int stage, void* token, cudaStream_t s, int launches);

}  // namespace gfe

#define GFE_CUDA_TRY(call)                                                                        \
  do {                                                                                            \
    cudaError_t e__ = (call);                                                                     \
    if (e__ != cudaSuccess)                                                                       \
      return gfe::set_error(GFE_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e__), \
                            __FILE__, __LINE__);                                                  \
  } while (0)

#define GFE_LAUNCH_CHECK(what)                                                                     \
  do {                                                                                             \
    cudaError_t e__ = cudaGetLastError();                                                          \
    if (e__ != cudaSuccess)                                                                        \
      return gfe::set_error(GFE_ERR_CUDA, "launch of %s failed: %s", what, cudaGetErrorString(e__)); \
  } while (0)

// Chains of small kernels, each adding one colour's entries: with `overlap` a launch may start once every CTA of the
// kernel before it has called chain_release (or has ended), so its launch and first loads run under that kernel's end;
// what the kernels before it wrote may be read (past the L1: __ldcg) or written after chain_wait only.  A kernel calls
// chain_wait before chain_release: what precedes the whole chain is then complete when the next one starts.
namespace gfe {
template <typename... Params, typename... Args>
cudaError_t launch_chained(bool overlap, void (*kernel)(Params...), int grid, int block, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
}  // namespace gfe
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Device-side error reporting: kernels never trap; they set bits in the error word.
__device__ __forceinline__ void gfe_raise(unsigned* err, unsigned bit) {
  if (err) atomicOr(err, bit);
}
