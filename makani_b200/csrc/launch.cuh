// Launches that follow one another in a stream without the gap in between.
//
// A kernel launched by `launch_chained` may begin while the one before it in the stream ends: its blocks take the SMs that become free,
// set up what is theirs (barriers, tensor memory) and wait in `chain_begin` until that kernel is complete and its writes are visible.
// `chain_begin` also lets the next kernel of the chain begin in the same way.  Every kernel launched like this calls it, in all its threads,
// before its first access to global memory; a complete kernel has then seen all kernels before it complete.  Kernels that wait for other
// devices are launched in the ordinary way, and the next one begins when they are complete: blocks that wait behind a wait would hold
// shared memory that kernels of other streams may need.
//
// What it saves is the time between two launches (some 2 us) and the set-up: the AFNO filter of 90 x 180 tokens, 14 products of 6 - 20 us, 256 -> 236 us
// a training pass, the token MLP (16200 x 768 -> 3072) 525 -> 511, the MLP of 240 x 480 tokens 600 -> 590.  Kernels of several waves gain as well
// (cast of 4096 x 4096 weights between two products, seven waves, 31.2 -> 30.9 us; weights of 8 x 512 AFNO channels, 3.5 waves, 29.7 -> 29.2).
// Launched in the ordinary way:
// - what spreads few blocks evenly, several to an SM: begun early these crowd on the SMs that are free (column sums, 127 us become 160);
// - the re-layout of the spectral weights (18432 blocks, 70 -> 90 and 99 -> 134 us);
// - long products (CHAINED_SLABS in gemm_tcgen05.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <atomic>
#include <utility>

namespace mk {

// Lets `kernel` take up to `bytes` of dynamic shared memory on the current device.  The attribute belongs to kernel and device: `devices` (one per
// kernel) holds those that have it, and none that refused.
inline cudaError_t allow_shared_memory(std::atomic<uint64_t>& devices, const void* kernel, int bytes) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  const uint64_t bit = device < 64 ? uint64_t{1} << device : 0;
  if (devices.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) devices.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

#ifdef __CUDACC__
// `next` false: the next kernel does not begin before this one is complete.  `p`: pointers whose loads the compiler may take for constant during the
// kernel (const __restrict__) and could move in front of the wait; they come out of it as new values.
template <typename... P>
__device__ __forceinline__ void chain_begin(bool next, P&... p) {
  if (next) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  auto renew = [](auto& q) { asm volatile("" : "+l"(q)::"memory"); };
  (renew(p), ...);
}

// `cluster`: blocks of a cluster (1: none); `chained` false: an ordinary launch
template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, bool chained,
                           Args&&... args) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (chained) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
#endif  // __CUDACC__

}  // namespace mk
