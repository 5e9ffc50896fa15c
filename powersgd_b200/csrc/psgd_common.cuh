// Shared device / host helpers for the PowerSGD sm_100a kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <tuple>
#include "psgd_types.h"

#define PSGD_API extern "C" __attribute__((visibility("default")))

// ---- host-side error plumbing -------------------------------------------------------------
void psgd_set_error(const char* fmt, ...);
#define PSGD_CUDA_OK(expr)                                                          \
  do {                                                                              \
    cudaError_t _e = (expr);                                                        \
    if (_e != cudaSuccess) {                                                        \
      psgd_set_error("%s:%d %s -> %s", __FILE__, __LINE__, #expr, cudaGetErrorString(_e)); \
      return (int)_e;                                                               \
    }                                                                               \
  } while (0)

// Status word written by kernels whose waits ran out. 0 = fine.
enum PsgdStatus : int {
  PSGD_OK = 0,
  PSGD_TIMEOUT_PEER_BARRIER = 2,
  PSGD_TIMEOUT_MBARRIER = 3,
  PSGD_BAD_ARGUMENT = 4,
};

// ---- device helpers -----------------------------------------------------------------------
__device__ __forceinline__ uint64_t psgd_globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ float psgd_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double psgd_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Partial sums of a split tile: element e of partial p lies at first[p * tile_elems + e]. Writes the sums
// over the `n` partials, in split order (fixed, so the result does not depend on which tile arrived last),
// to out[0 .. TILE_ELEMS). One CTA does this at the end of a product while the rest of the GPU has
// nothing left to do, and a tall matrix has tens of partials per block, so what counts is how many loads
// are under way: every thread takes four elements and eight partials at a time (tensor-core tiles, M^T P on CUDA
// cores above rank 2), or, where that would leave more than half of the threads without work, one element
// and sixteen partials (M^T P at rank 1 and 2, M Q on CUDA cores: at most 256 elements, one per thread).
template <int TILE_ELEMS, int THREADS>
__device__ __forceinline__ void psgd_sum_partials(const float* first, int n, float* out) {
  constexpr int W = TILE_ELEMS >= 2 * THREADS ? 4 : 1;   // floats per thread and load
  constexpr int B = W == 4 ? 8 : 16;                     // loads under way
  static_assert(TILE_ELEMS % W == 0, "whole vectors");
  for (int e = threadIdx.x * W; e < TILE_ELEMS; e += THREADS * W) {
    float s[W];
#pragma unroll
    for (int i = 0; i < W; ++i) s[i] = 0.f;
    for (int p = 0; p < n; p += B) {
      float v[B][W];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        if (p + j < n) {
          const float* src = first + (long long)(p + j) * TILE_ELEMS + e;
          if (W == 4) {
            const float4 q = __ldcg(reinterpret_cast<const float4*>(src));
            v[j][0] = q.x; v[j][1 % W] = q.y; v[j][2 % W] = q.z; v[j][3 % W] = q.w;
          } else {
            v[j][0] = __ldcg(src);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < B; ++j) {
        if (p + j < n) {
#pragma unroll
          for (int i = 0; i < W; ++i) s[i] += v[j][i];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < W; ++i) out[e + i] = s[i];
  }
}

__device__ __forceinline__ int psgd_atom_add_acqrel_gpu(int* p, int v) {
  int old;
  asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

// ---- launches that overlap the end of their predecessor ----------------------------------------
// A chain of short launches pays for each start: the grid is set up, descriptors are fetched, the
// first loads take their latency. With programmatic dependent launch a kernel may start while its
// predecessor in the stream still runs: the predecessor says so (psgd_launch_dependents, at its
// very beginning here), and the successor does what does not depend on any launch of the chain
// before it waits (psgd_wait_for_predecessor) for the predecessor to COMPLETE, memory included.
// Every kernel launched with `early` != 0 executes that wait in every thread before it reads or
// writes anything another launch of the chain writes; so completion stays transitive, and the
// launch that opens a chain (`early` == 0) still waits for everything before it.
__device__ __forceinline__ void psgd_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void psgd_wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Asks for the 128-byte line of L2 that holds *p. Only for addresses inside live allocations.
__device__ __forceinline__ void psgd_prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// More than 48 KiB of dynamic shared memory for a kernel: asked once per device, whose copy of the kernel the attribute belongs
// to. `devices`: those that have it (one bit each), a static variable of the caller.
static inline int psgd_allow_shared(const void* kernel, size_t bytes, unsigned long long& devices) {
  int device = 0;
  PSGD_CUDA_OK(cudaGetDevice(&device));
  const unsigned long long bit = 1ull << (device & 63);
  if (device < 64 && (devices & bit) != 0) return 0;
  PSGD_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  if (device < 64) __atomic_fetch_or(&devices, bit, __ATOMIC_RELAXED);
  return 0;
}

// Launches of the calling thread are written down here while it is not null, besides being made (psgd_host.cpp, psgd_tape_begin).
struct PsgdTape;
extern thread_local PsgdTape* psgd_tape_now;
void psgd_tape_add(const void* kernel, int grid, int block, size_t smem, int early, int cluster, int count, const void* const* args,
                   const size_t* sizes);

// `early` != 0: the kernel contains the wait above and the launch directly before it in `stream` is
// one of this library's.
static inline void psgd_launch_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attrs, int grid, int block, size_t smem, cudaStream_t stream,
                                      int early, int cluster) {
  cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  int n = 0;
  if (early) {
    attrs[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attrs[n].id = cudaLaunchAttributeClusterDimension;
    attrs[n].val.clusterDim.x = (unsigned)cluster;
    attrs[n].val.clusterDim.y = attrs[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = n;
}
template <typename... Params, typename... Args>
static inline int psgd_launch_clusters(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t stream, int early,
                                       int cluster, Args&&... args) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attrs[2];
  psgd_launch_config(cfg, attrs, grid, block, smem, stream, early, cluster);
  PSGD_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
  if (psgd_tape_now != nullptr) {
    const std::tuple<Params...> held(static_cast<Params>(args)...);
    std::apply([&](const auto&... arg) {
      const void* at[] = {(const void*)&arg...};
      const size_t sizes[] = {sizeof(arg)...};
      psgd_tape_add((const void*)kernel, grid, block, smem, early, cluster, (int)sizeof...(arg), at, sizes);
    }, held);
  }
  return 0;
}
template <typename... Params, typename... Args>
static inline int psgd_launch(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t stream, int early,
                              Args&&... args) {
  return psgd_launch_clusters(kernel, grid, block, smem, stream, early, 1, static_cast<Args&&>(args)...);
}

static inline int psgd_ceil_div(int a, int b) { return (a + b - 1) / b; }
