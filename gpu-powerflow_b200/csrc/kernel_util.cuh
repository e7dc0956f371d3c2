// kernel_util.cuh -- device and launch helpers shared by the factor kernels.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <stdexcept>
#include <string>
#include <utility>

#include "kernels.hpp"

namespace cupf_b200 {
namespace {

template <typename T>
__device__ __forceinline__ T guarded_pivot(T piv, bool static_pivot, double eps, bool& shifted) {
  if (piv == T(0)) {
    shifted = true;
    if (!static_pivot) return T(1);
  }
  if (static_pivot && (piv < T(0) ? -piv : piv) <= static_cast<T>(eps)) {
    shifted = true;
    return piv < T(0) ? static_cast<T>(-eps) : static_cast<T>(eps);
  }
  return piv;
}

// Opt a kernel into the full 227 KB of dynamic shared memory, once per
// (device, kernel); the attribute is per device and per function.
inline void allow_full_smem(const void* fn) {
  static std::mutex mu;
  static std::set<std::pair<int, const void*>> done;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) throw std::runtime_error("cudaGetDevice failed");
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({dev, fn})) return;
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
  if (e != cudaSuccess) throw std::runtime_error(std::string("shared-memory attribute: ") + cudaGetErrorString(e));
  done.insert({dev, fn});
}

inline void check_launch(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + " launch: " + cudaGetErrorString(e));
}

// ---------------------------------------------------------------------------
// Programmatic dependent launch between consecutive level kernels: a level
// kernel lets the next one be scheduled as soon as all of its own blocks are
// running (launch_dependents), and the next one runs the part of its work
// that reads only the static plan (launch record, assembly list, zeroing its
// shared-memory front) before it waits for the previous grid to finish and
// its writes to be visible (griddepcontrol.wait, a hardware wait that ends
// when that grid completes).  Launched without the attribute, both are
// no-ops.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void chain_allow_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void chain_wait_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Launch with programmatic stream serialization (the kernel's prologue may
// overlap the tail of the kernel before it on the stream).
template <typename... KArgs, typename... Args>
void launch_chained(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const char* what,
                    Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + " launch: " + cudaGetErrorString(e));
}

// ---------------------------------------------------------------------------
// Asynchronous global -> shared copies (cp.async, sm_80+ form; the copy
// completes in the background and cp.async.wait_group is a hardware wait, so
// no software spin is involved).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

}  // namespace
}  // namespace cupf_b200
