// common.cuh -- shared host/device helpers of libvcpcuda (status, errors,
// stream-ordered scratch, launch accounting).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cstddef>
#include <cstdio>
#include <string>
#include <atomic>

#include "../../include/vcpcuda.h"

namespace vcpcu {

// ---- error reporting (thread-local text, read by vcpcu_last_error_string) ---
void set_error(const char* fmt, ...);
void clear_error();

// Record a launch of one of this library's kernels.
void count_launch(long long n = 1);

// Turn a CUDA error into VCPCU_ERR_CUDA with a message.
int cuda_fail(cudaError_t e, const char* what);

#define VCPCU_CUDA_TRY(expr)                                         \
  do {                                                               \
    cudaError_t _e = (expr);                                         \
    if (_e != cudaSuccess) return ::vcpcu::cuda_fail(_e, #expr);     \
  } while (0)

#define VCPCU_LAUNCH_CHECK(what)                                     \
  do {                                                               \
    cudaError_t _e = cudaGetLastError();                             \
    if (_e != cudaSuccess) return ::vcpcu::cuda_fail(_e, what);      \
    ::vcpcu::count_launch();                                         \
  } while (0)

// The device must be an sm_103 part (the only code this library carries).
int check_device();

// Stream-ordered scratch: a buffer from the current device's default memory
// pool (cudaMallocAsync), freed stream-ordered when the guard goes away.
struct Scratch {
  void* ptr = nullptr;
  size_t bytes = 0;
  cudaStream_t stream = nullptr;
  Scratch() = default;
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  int alloc(size_t nbytes, cudaStream_t s);
  ~Scratch();
};

// Chains of kernels: with `chained` the kernel may start while its
// predecessor on the stream, a kernel of the same call that ends its own
// prologue with dep_ready(), still runs, and begins with dep_wait(), which
// returns when that one has completed and its writes are visible (every kernel
// of a chain waits, so all earlier ones have completed too).  Takes the launch
// latency out of the gap between two kernels: the product 61 x 48 x 97 34.8 ->
// 28.9 us, the eigenvalue verification at n = 1225 897 -> 873 us.  Not
// for the chunks of a batch: on their two streams the waiting blocks hold
// places that the other stream's kernels would take (1743 -> 1874 us).
// Without `chained`, an ordinary launch (and dep_wait() returns at once).
// A chained kernel lives while its predecessors write, so it must not take what
// they write through __restrict__ pointers to const or __ldg: the read-only path
// that these allow is only for data constant during the kernel's whole life.
#ifdef __CUDACC__
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_ready() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class T>
struct SameType {
  using type = T;
};
template <class... P>
cudaError_t launch_dep(bool chained, int cluster, void (*kernel)(P...), dim3 grid, dim3 block,
                       size_t smem, cudaStream_t s, typename SameType<P>::type... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  unsigned n = 0;
  if (chained) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = (unsigned)cluster;
    at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
#endif

inline size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace vcpcu
