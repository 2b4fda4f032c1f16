// Programmatic dependent launch for chains of small kernels (decode): a kernel launched with the stream-serialization
// attribute may start while its predecessor in the stream is still running. Everything it does before pdl_wait() must
// be independent of the predecessor's output (reading weights, prefetching them into L2); pdl_wait() returns once the
// predecessor has completed and its writes are visible. Every kernel of a chain calls pdl_launch_dependents() at its
// top so that its successor can be scheduled as soon as all of this kernel's CTAs are resident. In a kernel launched the ordinary way
// only pdl_wait() is a no-op: its pdl_launch_dependents() still lets an attributed successor start early. What a kernel reads before
// pdl_wait() must therefore be older than the whole chain, attributed or not. launch_pdl sets the launch attribute inside a PdlScope (the chains of
// layer_stack.cu) or with PMETAL_PDL=1.
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>

namespace pm {

__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Bulk prefetch of `bytes` (multiple of 16, 16-byte aligned) into L2; no data is returned to the SM.
__device__ __forceinline__ void l2_prefetch_bulk(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

inline bool pdl_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("PMETAL_PDL");
    v = e ? (atoi(e) != 0) : 0;
  }
  return v != 0;
}

// While one is alive, launch_pdl calls of this thread carry the attribute.
inline thread_local int pdl_scope_depth = 0;
struct PdlScope {
  const int on;
  explicit PdlScope(bool enable) : on(enable ? 1 : 0) { pdl_scope_depth += on; }
  ~PdlScope() { pdl_scope_depth -= on; }
  PdlScope(const PdlScope&) = delete;
};

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = pdl_scope_depth > 0 || pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace pm
