// common.cuh -- shared device helpers for libufvm (sm_100a).
//
// Floating-point contract: every FP64 kernel in this library is compiled with
// --fmad=false and evaluates each expression in the left-to-right order of the MATLAB
// source it restates, so results are reproducible bit for bit against a sequential
// evaluation of the same expression. Reductions over many rows (sums of |r|, r^2) use a
// fixed two-stage tree and are deterministic run to run.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <string>
#include <vector>

#include "../../include/ufvm.h"

namespace ufvm {

constexpr int kBlock = 256;

// error state (thread-local message for ufvm_last_error)
void set_error(const std::string& msg);
const char* get_error();
void trim_scratch_pool();  // gives the stand-alone functions' idle scratch back to the device

#define UFVM_CUDA(call)                                                                   \
  do {                                                                                    \
    cudaError_t _e = (call);                                                              \
    if (_e != cudaSuccess) {                                                              \
      ::ufvm::set_error(std::string(#call) + ": " + cudaGetErrorString(_e));             \
      return UFVM_E_CUDA;                                                                 \
    }                                                                                     \
  } while (0)

#define UFVM_CHECK(expr)                 \
  do {                                   \
    int _s = (expr);                     \
    if (_s != UFVM_OK) return _s;        \
  } while (0)

#define UFVM_LAUNCH_CHECK() UFVM_CUDA(cudaGetLastError())

inline int nblocks(long long n, int bs = kBlock) { return (int)((n + bs - 1) / bs); }

__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double dot3(double a0, double a1, double a2, double b0, double b1, double b2) {
  return (a0 * b0 + a1 * b1) + a2 * b2;
}

// Bytes of device memory this host thread holds through dalloc (freed by dfree). The batched
// service takes differences of it around each case's allocations to learn the case's HBM
// footprint.
inline thread_local long long t_dev_bytes = 0;
// Host time (ms) this thread has spent inside device allocation and free calls.
inline thread_local double t_alloc_ms = 0.0;

// Stream-ordered allocation. A thread inside an AllocStreamScope allocates from the device's
// default memory pool on the scope's stream (cudaMallocAsync) and frees there (cudaFreeAsync):
// neither call waits for the device, while cudaFree waits for the whole device and cudaMalloc
// goes through the driver's allocator. The batched service builds hundreds of cases' meshes and
// AMG hierarchies on several host threads at once (hundreds of allocations per case), so it
// allocates this way; everything else uses cudaMalloc. An array remembers how it was allocated.
// An allocation is ordered on the scope's stream: work on another stream that uses it first
// waits for that stream (the service's builders synchronise their streams before the service
// stream uses what they made).
// With a pool of its own a scope allocates from that instead (the stand-alone matrix functions: their
// scratch lives for one call), but for arrays of kPoolArray bytes and more: what a pool does not keep it
// maps and unmaps in small pieces. Allocation and free, ms, cudaMalloc / pool: 128 MB 0.7 / 0.4 (kept),
// 512 MB 1.3 / 3.4, 2 GB 2.2 / 22, 4.8 GB 7 / 180 and more.
constexpr size_t kPoolArray = 128ull << 20;
struct AllocScopeState {
  bool on = false;
  cudaStream_t stream = nullptr;
  cudaMemPool_t pool = nullptr;
};
inline thread_local AllocScopeState t_alloc;
struct AllocStreamScope {
  AllocScopeState prev;
  explicit AllocStreamScope(cudaStream_t s, cudaMemPool_t pool = nullptr) : prev(t_alloc) { t_alloc = {true, s, pool}; }
  ~AllocStreamScope() { t_alloc = prev; }
  AllocStreamScope(const AllocStreamScope&) = delete;
  AllocStreamScope& operator=(const AllocStreamScope&) = delete;
};
// Whether this thread allocates on its scope's stream now; not while that stream is being captured into a
// graph, where an asynchronous allocation would become a graph node.
inline bool alloc_async_now() {
  if (!t_alloc.on) return false;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(t_alloc.stream, &cs) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return cs == cudaStreamCaptureStatusNone;
}
double host_ms_now();

// Device array owned by a case; freed by its owner.
template <typename T>
struct DArr {
  T* p = nullptr;
  size_t n = 0;
  bool async = false;  // stream-ordered allocation, else cudaMalloc
};

template <typename T>
void dfree(DArr<T>& a) {
  if (a.p) {
    const double t0 = host_ms_now();
    if (!a.async) {
      cudaFree(a.p);
    } else if (alloc_async_now()) {
      cudaFreeAsync(a.p, t_alloc.stream);
    } else {
      // outside a scope nothing orders the free after the array's last use: wait for it
      cudaDeviceSynchronize();
      cudaFree(a.p);
    }
    t_alloc_ms += host_ms_now() - t0;
    t_dev_bytes -= (long long)(a.n * sizeof(T));
  }
  a.p = nullptr;
  a.n = 0;
  a.async = false;
}

// At least n elements. An array that has to grow gets a quarter more than asked for: the coarse levels
// of a hierarchy that is rebuilt at every solve change by a few rows each time. Where that does not fit
// on the device, the stand-alone functions' idle scratch is given back and the array gets what was asked
// for.
template <typename T>
int dalloc(DArr<T>& a, size_t n) {
  if (a.p && a.n >= n) return UFVM_OK;
  if (n == 0) n = 1;
  size_t cap = a.p ? n + n / 4 : n;
  dfree(a);
  const double t0 = host_ms_now();
  const bool scope = alloc_async_now();
  bool async = scope;
  auto get = [&]() {
    const size_t bytes = cap * sizeof(T);
    async = scope && !(t_alloc.pool && bytes >= kPoolArray);
    return !async ? cudaMalloc((void**)&a.p, bytes)
           : t_alloc.pool ? cudaMallocFromPoolAsync((void**)&a.p, bytes, t_alloc.pool, t_alloc.stream)
                          : cudaMallocAsync((void**)&a.p, bytes, t_alloc.stream);
  };
  cudaError_t e = get();
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();  // an out-of-memory report is not sticky: clear it for later checks
    trim_scratch_pool();
    cap = n;
    e = get();
  }
  t_alloc_ms += host_ms_now() - t0;
  if (e != cudaSuccess) {
    a.p = nullptr;
    cudaGetLastError();
    set_error(std::string(async ? "cudaMallocAsync: " : "cudaMalloc: ") + cudaGetErrorString(e));
    return UFVM_E_OOM;
  }
  a.n = cap;
  a.async = async;
  t_dev_bytes += (long long)(cap * sizeof(T));
  return UFVM_OK;
}

// Programmatic dependent launch. A kernel launched with programmatic stream serialization may
// start once every block of the kernel before it has executed pdl_trigger; pdl_wait then blocks
// until that kernel has completed and its writes are visible. Without the launch attribute both
// are no-ops. A kernel that waits before touching memory any earlier kernel writes behaves as
// an ordinary launch, minus the launch gap.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Kernels whose blocks wait for one another's results: a flag is read and written past the L1, and a
// wait gives up after kFlagClocks SM clocks (seconds), which the host reports.
constexpr long long kFlagClocks = 1ll << 33;
__device__ __forceinline__ int ld_flag(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_flag(int* p, int v) {
  asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ---- block reductions (fixed shape => deterministic) ----
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = dmax(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_min(double v) {
  for (int o = 16; o > 0; o >>= 1) v = dmin(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// reduce over the block; result valid in thread 0. sh must hold blockDim/32 doubles.
template <int OP>  // 0 sum, 1 max, 2 min
__device__ __forceinline__ double block_reduce(double v, double* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = OP == 0 ? warp_sum(v) : (OP == 1 ? warp_max(v) : warp_min(v));
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  if (w == 0) {
    double x = lane < nw ? sh[lane] : (OP == 0 ? 0.0 : (OP == 1 ? -INFINITY : INFINITY));
    x = OP == 0 ? warp_sum(x) : (OP == 1 ? warp_max(x) : warp_min(x));
    v = x;
  }
  return v;
}

}  // namespace ufvm
