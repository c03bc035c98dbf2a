// Kernel launch with programmatic dependent launch (PDL).
//
// A decode step is ~260 short kernels in one stream. Launched the plain way, kernel N+1 is only handed to
// the GPU when kernel N has drained; with the programmatic-stream-serialization attribute its CTAs are
// scheduled as soon as every CTA of kernel N has executed pdl_trigger() (ptx.cuh), they run their
// prologue (barrier set-up, TMEM allocation, descriptor prefetch) and then block in pdl_wait() until
// kernel N has completed and its memory is visible. Every kernel launched through launch_pdl() therefore
// calls pdl_wait() before its first access to memory that an earlier kernel may have written, and before
// its first write to memory that an earlier kernel may still read. The attribute is recorded by stream
// capture, so the overlap is kept inside CUDA graphs.
//
// A kernel with tensor memory triggers after its allocation, behind a barrier of the CTA. Triggered before it, a CTA of kernel N + 1 on the
// same SM could take the columns first and hold them until kernel N has completed, which could then not allocate its own: neither would end.
//
// Products that may fetch their weights early (gemm_ws.cuh: early_w) are launched like that unless SKEIN_EARLY_WEIGHTS=0: behind a norm or the
// attention, whose CTAs leave room for theirs (~200 KB of shared memory), the streaming GEMM's stages fill while the kernel before ends (4096 x
// 4096 in a chain 13.3 -> 11.7 us). For everything else it is off unless SKEIN_PDL=1: on the decode step of the flagship model it measured 1-2 %
// slower than plain serialization (132.6 -> 135.1 us per layer at the 8-way tensor-parallel shard shapes), as a product cannot become resident behind
// another one and the other kernels have no prologue worth overlapping.
#pragma once
#include "per_device.h"
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>
#include <utility>

namespace skein {

// Read once per process (RuntimeConfig: pdl, early_weights).
inline bool pdl_enabled() {
  static const bool on = [] { const char* e = getenv("SKEIN_PDL"); return e != nullptr && strcmp(e, "1") == 0; }();
  return on;
}
inline bool early_weights_enabled() {
  static const bool on = [] { const char* e = getenv("SKEIN_EARLY_WEIGHTS"); return e == nullptr || strcmp(e, "0") != 0; }();
  return on;
}

// Wait budgets of the kernels that wait on other CTAs of their own launch, in milliseconds, from the environment
// (set as a group through RuntimeConfig: grid_barrier_ms, gemm_wait_ms). Read once per process.
inline int env_ms(const char* name, int fallback) {
  const char* e = getenv(name);
  if (e == nullptr || *e == 0) return fallback;
  const long v = strtol(e, nullptr, 10);
  return (v > 0 && v < 3600000) ? (int)v : fallback;
}
inline int grid_barrier_budget_ms() { static int v = env_ms("SKEIN_GRID_BARRIER_MS", 2000); return v; }
inline int gemm_wait_budget_ms() { static int v = env_ms("SKEIN_GEMM_WAIT_MS", 2000); return v; }

// Shared memory beyond 48 KB for a kernel, allowed once on every device that launches it (`done`: static, one per kernel).
inline cudaError_t allow_smem(PerDevice& done, const void* kernel, int bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int got = done.get(dev, [&] {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e == cudaSuccess ? 1 : -1;
  });
  return got > 0 ? cudaSuccess : e != cudaSuccess ? e : cudaErrorInvalidDevice;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_if(bool on, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = on ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  return launch_pdl_if(pdl_enabled(), kernel, grid, block, smem, stream, std::forward<Args>(args)...);
}

}  // namespace skein
