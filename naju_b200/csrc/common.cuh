// Shared device helpers for the sm_100a gated-scan kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "naju_b200.h"

namespace naju {

constexpr int kDT = 128;        // channels per tile

// Spin budget of every device-side wait: iterations of (poll + nanosleep).  About 0.2 s in
// the worst case, after which the waiter records NAJU_ST_LOOKBACK_TIMEOUT and carries on
// with whatever it has, so a kernel can never hang the device.
constexpr int kSpinLimit = 1 << 20;

// ---------------------------------------------------------------- dtype conversion
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat162float(v);
}
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

__host__ __device__ __forceinline__ int dtype_size(int dt) { return dt == NAJU_F32 ? 4 : 2; }

// runtime-typed scalar access (used only for the small B/C tiles and the finalize kernels)
__device__ __forceinline__ float load_dyn(const void* p, int dt, int64_t idx) {
  if (dt == NAJU_F32) return reinterpret_cast<const float*>(p)[idx];
  if (dt == NAJU_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[idx]);
  return __half2float(reinterpret_cast<const __half*>(p)[idx]);
}
__device__ __forceinline__ void store_dyn(void* p, int dt, int64_t idx, float v) {
  if (dt == NAJU_F32) reinterpret_cast<float*>(p)[idx] = v;
  else if (dt == NAJU_BF16) reinterpret_cast<__nv_bfloat16*>(p)[idx] = __float2bfloat16_rn(v);
  else reinterpret_cast<__half*>(p)[idx] = __float2half_rn(v);
}

// ---------------------------------------------------------------- gates
// sigmoid(x) and 1 - sigmoid(x) without cancellation: a = e^-x, f = 1/(1+a), 1-f = a f.
// ex2.approx + a fast reciprocal keep the relative error near 2 ulp, which matters because
// retention gates multiply up over hundreds of steps.
struct Gate { float s; float one_minus; };
__device__ __forceinline__ Gate gate(float x) {
  x = fmaxf(x, -80.f);  // e^80 is finite in fp32; sigmoid(-80) ~ 1.8e-35 either way
  const float a = __expf(-x);
  const float s = __fdividef(1.f, 1.f + a);
  return Gate{s, a * s};
}
__device__ __forceinline__ float sigmoid_f(float x) { return gate(x).s; }

// ---------------------------------------------------------------- memory ordering
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ---------------------------------------------------------------- programmatic dependent launch
// A kernel started with launch_pdl() may begin while the kernel before it in the stream is still
// running: pdl_wait() returns once that one has completed and its writes are visible, and nothing that
// touches global memory may come before it.  pdl_launch_dependents() lets the next such kernel's
// blocks start as soon as every block of this one has called it (or ended).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// (`cluster` CTAs in a row form a thread-block cluster)
template <typename... P, typename... A>
inline int launch_cluster(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, int cluster, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}
template <typename... P, typename... A>
inline int launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  return launch_cluster(kernel, grid, block, smem, 1, st, static_cast<A&&>(args)...);
}

// Raises a kernel's dynamic shared-memory limit once per device (`done`: a bit per device ordinal, one
// word per kernel).
template <typename K>
inline int allow_smem(K* kernel, size_t bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev < 64 && (done.load(std::memory_order_relaxed) & bit)) return 0;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return static_cast<int>(e);
}

}  // namespace naju
