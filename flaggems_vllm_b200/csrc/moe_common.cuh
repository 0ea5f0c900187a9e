// Shared helpers for the sm_100a MoE kernels: error reporting for the C ABI,
// dtype tags, small device utilities.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/moe_sm100.h"

namespace moe {

// Records a host-side failure text for moe_last_error(); returns `code`.
int fail(int code, const char* fmt, ...);
// Checks the launch error of the kernel just enqueued; returns 0 or the cudaError_t.  Called once per kernel: it counts
// the launches that were accepted (moe_launch_count).
int check_launch(const char* what);
// Limit, in nanoseconds, of every bounded barrier wait of the kernels launched from now on
// (moe_set_wait_limit_ns; 2 s unless changed).
unsigned long long wait_limit_ns();
// Lets `kernel` use `bytes` of dynamic shared memory (and clusters of more than 8 CTAs) on the current device (set once
// per device, remembered).
int allow_smem(const void* kernel, int bytes, bool large_cluster = false);
// Multiprocessors of the current device (remembered).
int sm_count();
// Clusters of `ctas` CTAs of this kernel that the device, or the part of it this context has, runs at once: 0 = such a
// cluster never starts (a partition without a GPC that holds it), -1 = there is no device to ask.  Asked on every
// call, 0.2 us: what a context has of a device can change.
int max_clusters(const void* kernel, int ctas, int threads, size_t smem);

// Programmatic dependent launch.  The kernels of a layer are launched so that each may start while its predecessor
// drains: what it does before pdl_wait() touches nothing the predecessor writes (barriers, TMEM, weights, and the
// route plan, which is two kernels old for a GEMM; read past L1).  pdl_wait() returns when the predecessor has
// completed and is visible; only then does a kernel let its own successor start, so whatever is older than the
// predecessor is complete too.  Both are no-ops in a kernel launched the ordinary way.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch with a cluster size (1 = none) and the programmatic dependency on what precedes it in the stream.
template <typename Kernel, typename... Args>
int launch_pdl(Kernel kern, dim3 grid, int threads, size_t smem, int cluster, cudaStream_t st, const char* what, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t ce = cudaLaunchKernelEx(&cfg, kern, args...);
  if (ce != cudaSuccess) return fail((int)ce, "%s: %s", what, cudaGetErrorString(ce));
  return check_launch(what);
}

// The same for many small blocks that one wave holds.  A kernel that starts while its predecessor still fills most multiprocessors
// finds room on the few that are free, and its blocks crowd there (router_gemm, then grouped_topk of 2000 tokens: 500 blocks on 20
// of 148).  So a block asks for the share of the shared memory that lets no multiprocessor take more than its part.  us in a graph,
// elementwise kernel + router_gemm + grouped_topk, nothing started early / crowding / so: 1000 tokens 21.8 / 22.6 / 19.9, 2000
// 31.8 / 33.2 / 26.9, 4000 56.8 / 50.7 / 45.8; with 128 experts and topk_softmax 19.1 / 21.1 / 18.5, 25.4 / 26.8 / 24.7, 40.2 / 43.4 / 39.0.
template <typename Kernel, typename... Args>
int launch_pdl_spread(Kernel kern, dim3 grid, int threads, size_t static_smem, cudaStream_t st, const char* what, Args... args) {
  constexpr size_t kSm = 228 * 1024, kBlock = 227 * 1024;  // of a multiprocessor (1 KB of it the system's per block), of a block
  const int rc = allow_smem((const void*)kern, (int)(kBlock - static_smem));
  if (rc) return rc;
  const size_t per_sm = ((size_t)grid.x * grid.y + sm_count() - 1) / sm_count();
  size_t smem = 0;
  if (per_sm > 1 && per_sm < 2048u / threads) smem = (kSm / per_sm - 1024 - static_smem) / 128 * 128;
  return launch_pdl(kern, grid, threads, smem, 1, st, what, args...);
}

template <typename T> struct ToF32;
template <> struct ToF32<float> {
  static __device__ __forceinline__ float get(float v) { return v; }
};
template <> struct ToF32<__half> {
  static __device__ __forceinline__ float get(__half v) { return __half2float(v); }
};
template <> struct ToF32<__nv_bfloat16> {
  static __device__ __forceinline__ float get(__nv_bfloat16 v) { return __bfloat162float(v); }
};

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

__device__ __forceinline__ float fp8e4m3_to_f32(uint8_t v) {
  __half_raw h = __nv_cvt_fp8_to_halfraw(v, __NV_E4M3);
  return __half2float(*reinterpret_cast<__half*>(&h));
}
__device__ __forceinline__ uint8_t f32_to_fp8e4m3(float v) {
  return (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}

// SiLU(g) * u with the sigmoid written as the reference kernel does,
// g / (1 + exp(-g)) in fp32 (src/flaggems_vllm/ops/fused_moe.py:1795).
__device__ __forceinline__ float silu_mul(float g, float u) {
  return (g / (1.0f + expf(-g))) * u;
}

__device__ __forceinline__ void set_status(int32_t* status, int bit) {
  if (status != nullptr) atomicOr(status, bit);
}

// Eight consecutive elements as fp32 (one or two 16-byte loads).
template <typename T>
__device__ __forceinline__ void load8(const T* p, float (&v)[8]);
template <>
__device__ __forceinline__ void load8<float>(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <>
__device__ __forceinline__ void load8<__half>(const __half* p, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(h[i]);
    v[2 * i] = f.x; v[2 * i + 1] = f.y;
  }
}
template <>
__device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x; v[2 * i + 1] = f.y;
  }
}

constexpr float kFp8Max = 448.0f;
constexpr float kQuantEps = 1e-10f;

}  // namespace moe
