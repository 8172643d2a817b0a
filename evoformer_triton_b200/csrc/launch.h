// Host-side launch entry points of the kernel families (internal to the library).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>

#include <atomic>
#include <mutex>
#include <unordered_map>
#include <utility>

#include "common.cuh"

namespace evo {

// Per (device, kernel) facts that cost a driver call each: the dynamic shared memory limit that has
// been set for the kernel and its launch-time register count.  Looked up on every launch, asked of
// the driver once (the limit again only when a launch needs more than any before it).
struct KernelFacts {
  int smem_limit = 0;
  int num_regs = 0;
};
inline bool kernel_ready(const void* kern, int smem_bytes, int* num_regs) {
  static std::mutex mu;
  static std::unordered_map<const void*, KernelFacts> facts[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  std::lock_guard<std::mutex> lock(mu);
  KernelFacts& f = facts[dev][kern];
  if (f.num_regs == 0) {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return false;
    f.num_regs = fa.numRegs;
  }
  if (smem_bytes > f.smem_limit) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess) return false;
    f.smem_limit = smem_bytes;
  }
  if (num_regs) *num_regs = f.num_regs;
  return true;
}

// SM count of the current device, or 0 (asked of the driver once per device).
inline int sm_count() {
  static std::atomic<int> table[64];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if ((n = table[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 0;
  table[dev].store(n, std::memory_order_relaxed);
  return n;
}

// Launches a kernel that may be scheduled while the one before it on the stream is still draining
// (programmatic dependent launch).  The kernel calls ptx::grid_dependency_wait() before it touches
// global memory, which waits for that one to have completed, and ptx::grid_launch_dependents() to let the
// next one in.  Saves the gap between the kernels of a call, about a microsecond each.
template <class K, class... A>
inline cudaError_t launch_dependent(K kern, dim3 grid, int threads, size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// CUDA-core kernels (generic_kernels.cu).  Backward needs generic_bwd_workspace_bytes() of scratch at a.delta
// (asked for with a.dbias set if and only if d(pair_bias) is wanted).
size_t generic_bwd_workspace_bytes(const Args& a);
cudaError_t launch_generic_fwd(int dtype, const Args& a, cudaStream_t st, int* launches);
cudaError_t launch_generic_bwd(int dtype, const Args& a, cudaStream_t st, int* launches);

// tcgen05 / TMEM / TMA kernels (fwd_sm100.cu, bwd_sm100.cu).  The *_supported
// predicates say whether a request is covered; the launchers return an EVOATTN_* status.
bool sm100_fwd_supported(int dtype, const Args& a);
int launch_sm100_fwd(int dtype, const Args& a, cudaStream_t st, int* launches);
bool sm100_bwd_supported(int dtype, const Args& a);
size_t sm100_bwd_workspace_bytes(int dtype, const Args& a);
int launch_sm100_bwd(int dtype, const Args& a, void* workspace, size_t workspace_bytes, cudaStream_t st,
                     int* launches);

// The exchange of d(pair_bias) between the GPUs of a node (peer_reduce.cu), and the side stream
// with its fork / join events on which a backward call runs it next to its last kernel.
int launch_peer_allreduce(const evoattn_peer_allreduce_params* p, cudaStream_t st);
bool exchange_lane(cudaStream_t* side, cudaEvent_t* fork, cudaEvent_t* join);

// d(pair_bias) from the fp32 buffer it was summed in to a.dbias_out, in its type and layout (extras.cu).
int launch_dbias_out(const Args& a, cudaStream_t st, int* launches);

// From here on `a` reads the effective dO of a gated output (contiguous, in scratch).
inline void use_effective_d_o(Args* a) {
  a->d_o = a->d_o_eff;
  a->sdo = Str4{(long long)a->H * a->S * a->R * a->D, (long long)a->S * a->R * a->D, (long long)a->R * a->D, (long long)a->D};
}

}  // namespace evo
