// Row movement on both sides of the grouped GEMMs of gemm_wt.cu: tokens into expert-sorted order (quantised on
// the way where the mode wants it), route rows back into tokens.
//
//   scatter   every token row is read ONCE and written to the sorted rows of its k routes (row_index of the route
//             plan; -1 = no row).  Quantising per route instead of per token costs k times the divisions, and
//             quantising first and gathering afterwards reads the quantised rows k times.
//   combine   out[token] = sum over its routes, in slot order, of weight * y[row], fp32.
// Bound: HBM / L2 bandwidth.
#include "moe_common.cuh"

namespace moe {
namespace {

constexpr int kThreads = 256;

// Zeroes the padding rows of the plan's tiles, one block per (tile, eighth of its padding rows).  At prefill sizes the
// GEMMs multiply those rows, and zeros cost the power-limited board less than stale bytes (DSV3 FP8, 8192 tokens:
// 5430 -> 5050 us per layer).
constexpr int kPadParts = 8;
__global__ void __launch_bounds__(kThreads) zero_padding_kernel(const int4* __restrict__ tiles, const int32_t* __restrict__ counts,
                                                                int row_vec, uint4* __restrict__ rows) {
  pdl_wait();
  pdl_trigger();
  if ((int)blockIdx.x >= counts[0]) return;
  const int4 d = tiles[blockIdx.x];
  for (int r = (d.y >> 16) + blockIdx.y; r < (d.y & 0xFFFF); r += kPadParts) {
    uint4* p = rows + (int64_t)(d.x + r) * row_vec;
    for (int i = threadIdx.x; i < row_vec; i += kThreads) p[i] = make_uint4(0, 0, 0, 0);
  }
}

// Block (c, m): 2048 columns of token m, a warp per two neighbouring 128-groups, 8 elements per lane.  The arithmetic
// is that of the stand-alone quantiser (quant.cu), bit for bit.
template <typename T>
__global__ void __launch_bounds__(kThreads) scatter_quant_group_kernel(const T* __restrict__ x, int groups, int k,
                                                                       const int32_t* __restrict__ row_index,
                                                                       int64_t rows_cap, uint8_t* __restrict__ q,
                                                                       float* __restrict__ scales_t) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int64_t m = blockIdx.y;
  const int g = (blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * 2 + (lane >> 4);
  const int row = lane < k ? row_index[m * k + lane] : -1;
  if (__ballot_sync(0xFFFFFFFFu, row >= 0) == 0) return;  // no route of this token is local
  const int64_t K = (int64_t)groups * 128;
  const bool in = g < groups;
  uint4 raw = make_uint4(0, 0, 0, 0);
  if (in) raw = *reinterpret_cast<const uint4*>(x + m * K + (int64_t)g * 128 + (lane & 15) * 8);
  const T* pv = reinterpret_cast<const T*>(&raw);
  float v[8], amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = ToF32<T>::get(pv[i]);
    amax = fmaxf(amax, fabsf(v[i]));
  }
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, off));
  const float s = fmaxf(amax, kQuantEps) * (1.0f / kFp8Max);
  uint32_t lo = 0, hi = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    lo |= (uint32_t)f32_to_fp8e4m3(fminf(fmaxf(v[i] / s, -kFp8Max), kFp8Max)) << (8 * i);
    hi |= (uint32_t)f32_to_fp8e4m3(fminf(fmaxf(v[4 + i] / s, -kFp8Max), kFp8Max)) << (8 * i);
  }
  for (int j = 0; j < k; ++j) {
    const int r = __shfl_sync(0xFFFFFFFFu, row, j);
    if (r < 0 || !in) continue;
    *reinterpret_cast<uint2*>(q + (int64_t)r * K + (int64_t)g * 128 + (lane & 15) * 8) = make_uint2(lo, hi);
    if ((lane & 15) == 0) scales_t[(int64_t)g * rows_cap + r] = s;
  }
}

// Rows of `vec` 16-byte pieces copied as they are; block (c, m): 512 pieces of token m, two per thread.
__global__ void __launch_bounds__(kThreads) scatter_rows_kernel(const uint4* __restrict__ x, int vec, int k,
                                                                const int32_t* __restrict__ row_index,
                                                                uint4* __restrict__ out) {
  pdl_wait();
  pdl_trigger();
  const int64_t m = blockIdx.y;
  const int c = blockIdx.x * 2 * kThreads + threadIdx.x;
  uint4 v[2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (c + i * kThreads < vec) v[i] = x[m * vec + c + i * kThreads];
  for (int j = 0; j < k; ++j) {
    const int64_t r = row_index[m * k + j];
    if (r < 0) continue;
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (c + i * kThreads < vec) out[r * vec + c + i * kThreads] = v[i];
  }
}

// dst[row_index[i]] = src[i / div] (one float per route: route weights, or a token's activation scale)
__global__ void scatter_floats_kernel(const float* __restrict__ src, int64_t numel, int div,
                                      const int32_t* __restrict__ row_index, float* __restrict__ dst) {
  pdl_wait();
  pdl_trigger();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < numel; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = row_index[i];
    if (r >= 0) dst[r] = src[i / div];
  }
}

// Block (c, m): 256 16-byte pieces of token m's output row, one per thread, eight route rows in flight.  No loop over
// tokens and no division: the loads of enough blocks are in flight to fill HBM whatever k is.
template <typename T, bool WEIGHTED>
__global__ void __launch_bounds__(kThreads) combine_kernel(const T* __restrict__ y, const float* __restrict__ weight,
                                                           const int32_t* __restrict__ row_index, int k, int vec,
                                                           T* __restrict__ out) {
  pdl_wait();
  pdl_trigger();
  constexpr int V = 16 / sizeof(T);
  const int64_t m = blockIdx.y;
  const int c = blockIdx.x * kThreads + threadIdx.x;
  if (c >= vec) return;
  const int32_t* rows = row_index + m * k;
  const float* w = weight + m * k;
  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.0f;
  for (int j0 = 0; j0 < k; j0 += 8) {
    uint4 raw[8];
    int r[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      r[u] = j0 + u < k ? rows[j0 + u] : -1;
      if (r[u] >= 0) raw[u] = reinterpret_cast<const uint4*>(y)[(int64_t)r[u] * vec + c];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (r[u] >= 0) {
        const float wj = WEIGHTED ? w[j0 + u] : 1.0f;
        const T* p = reinterpret_cast<const T*>(&raw[u]);
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] = WEIGHTED ? fmaf(wj, ToF32<T>::get(p[i]), acc[i]) : acc[i] + ToF32<T>::get(p[i]);
      }
    }
  }
  uint4 o;
  T* p = reinterpret_cast<T*>(&o);
#pragma unroll
  for (int i = 0; i < V; ++i) p[i] = from_f32<T>(acc[i]);
  reinterpret_cast<uint4*>(out)[m * vec + c] = o;
}
}  // namespace

// M <= 65535 for all of these (the second grid dimension): the layer call checks it.
int zero_padding(const void* tiles, int64_t tiles_cap, const int32_t* counts, int64_t row_bytes, void* rows, cudaStream_t st) {
  return launch_pdl(zero_padding_kernel, dim3((unsigned)tiles_cap, kPadParts), kThreads, 0, 1, st, "zero padding rows",
                    (const int4*)tiles, counts, (int)(row_bytes / 16), (uint4*)rows);
}

int scatter_quant_group(const void* x, int dtype, int64_t M, int H, int k, const int32_t* row_index, int64_t rows_cap, void* q,
                        float* scales_t, cudaStream_t st) {
  const int groups = H / 128;
  const dim3 grid((unsigned)((groups + 15) / 16), (unsigned)M);
  if (dtype == MOE_BF16)
    return launch_pdl(scatter_quant_group_kernel<__nv_bfloat16>, grid, kThreads, 0, 1, st, "scatter (1x128 quantised)",
                      (const __nv_bfloat16*)x, groups, k, row_index, rows_cap, (uint8_t*)q, scales_t);
  return launch_pdl(scatter_quant_group_kernel<__half>, grid, kThreads, 0, 1, st, "scatter (1x128 quantised)", (const __half*)x,
                    groups, k, row_index, rows_cap, (uint8_t*)q, scales_t);
}

int scatter_rows(const void* x, int64_t M, int64_t row_bytes, int k, const int32_t* row_index, void* out, cudaStream_t st) {
  const int vec = (int)(row_bytes / 16);
  return launch_pdl(scatter_rows_kernel, dim3((unsigned)((vec + 2 * kThreads - 1) / (2 * kThreads)), (unsigned)M), kThreads, 0, 1, st,
                    "scatter", (const uint4*)x, vec, k, row_index, (uint4*)out);
}

int scatter_floats(const float* src, int64_t numel, int div, const int32_t* row_index, float* dst, cudaStream_t st) {
  const int64_t blocks = (numel + 255) / 256;
  return launch_pdl(scatter_floats_kernel, dim3((unsigned)(blocks < 1024 ? blocks : 1024)), 256, 0, 1, st, "scatter (floats)", src,
                    numel, div, row_index, dst);
}

int combine_rows(const void* y, int dtype, const float* weight, const int32_t* row_index, int64_t M, int k, int64_t H, void* out,
                 cudaStream_t st) {
  const int vec = (int)(H / 8);
  const dim3 grid((unsigned)((vec + kThreads - 1) / kThreads), (unsigned)M);
#define MOE_COMBINE(T, W) \
  launch_pdl(combine_kernel<T, W>, grid, kThreads, 0, 1, st, "combine", (const T*)y, weight, row_index, k, vec, (T*)out)
  if (dtype == MOE_BF16) return weight != nullptr ? MOE_COMBINE(__nv_bfloat16, true) : MOE_COMBINE(__nv_bfloat16, false);
  return weight != nullptr ? MOE_COMBINE(__half, true) : MOE_COMBINE(__half, false);
#undef MOE_COMBINE
}

}  // namespace moe
