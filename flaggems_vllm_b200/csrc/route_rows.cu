// Row movement on both sides of the grouped GEMMs of the layer call: tokens into expert-sorted order (quantised on
// the way where the mode wants it), route rows back into tokens.
//
//   scatter   every token row is read ONCE and written to the sorted rows of its k routes (row_index of the route
//             plan; -1 = no row).  Quantising per route instead of per token costs k times the divisions, and
//             quantising first and gathering afterwards reads the quantised rows k times.
//   combine   out[token] = sum over its routes, in slot order, of weight * y[row], fp32.
// Bound: memory only where a launch is long; else the chain of a block (row index, rows, store) with too few bytes in flight.
// DSV3 FP8, 8192 tokens: combine 179 us for 1.06 GB (5.9 TB/s; a copy runs at 6.5), clearing the padding 23 us, the
// quantising scatter 125 us for 0.60 GB while it divided every element (issue slots 65 % busy).  Qwen3 shape, 4096 tokens, 151 MB
// each: scatter 25 us, combine 29 us (5.2 TB/s; registers let 23 % of an SM's warps in, and 7 of 10 wait for a load).
// 1024 tokens of DSV3 width: combine 29 us for 125 MB (4.3 TB/s).
#include "moe_common.cuh"

namespace moe {
namespace {

constexpr int kThreads = 256;

// Zeroes the padding rows of the plan's tiles and (1x128 scaled rows) their scales, one block per (tile, eighth of its
// padding).  At prefill sizes the GEMMs multiply those rows, and the tensor cores' clock there is what power leaves: DSV3
// FP8, 8192 tokens, 5390 us per layer with zeros in them and 5590 with pseudo-random e4m3 (a workspace that happens to
// hold zeros already: the same either way; fetching occupied rows only: 4826 us where whole blocks took 4796).
constexpr int kPadParts = 8;
__global__ void __launch_bounds__(kThreads) zero_padding_kernel(const int4* __restrict__ tiles, const int32_t* __restrict__ counts,
                                                                int row_vec, uint4* __restrict__ rows, int groups,
                                                                int64_t scale_ld, float* __restrict__ scales_t) {
  pdl_wait();
  pdl_trigger();
  if ((int)blockIdx.x >= counts[0]) return;
  const int4 d = tiles[blockIdx.x];
  const int occupied = d.y >> 16, padding = (d.y & 0xFFFF) - occupied;
  for (int r = blockIdx.y; r < padding; r += kPadParts) {
    uint4* p = rows + (int64_t)(d.x + occupied + r) * row_vec;
    for (int i = threadIdx.x; i < row_vec; i += kThreads) p[i] = make_uint4(0, 0, 0, 0);
  }
  if (scales_t == nullptr) return;
  // zero times a stale scale is NaN where the workspace happened to hold one
  for (int i = blockIdx.y * kThreads + threadIdx.x; i < padding * groups; i += kPadParts * kThreads)
    scales_t[(int64_t)(i / padding) * scale_ld + d.x + occupied + i % padding] = 0.0f;
}

// v / s, correctly rounded, for |v| <= 448 s (1 + ulp) from the rounded reciprocal of s: one correction step by the exact
// remainder (P. Markstein, Computation of elementary functions on the IBM RISC System/6000, 1990).  Where the quotient is
// so small that the remainder is not exact it rounds to zero in e4m3 all the same: over every pair of finite bf16 or f16
// values (amax, |v| <= amax) the e4m3 bytes are those of the division.  The sign is v's, of a zero too.
__device__ __forceinline__ float div_by_scale(float v, float s, float inv) {
  const float q = v * inv;
  return copysignf(fmaf(fmaf(-q, s, v), inv, q), v);
}

// EARLY (below): the token is read and quantised while the route plan is still being made.
// Block (c, m): P x blockDim.x / 8 128-groups of token m, eight lanes per group, 16 elements per lane.  The bytes and scales
// are those of the stand-alone quantiser (quant.cu).  With a division per element the kernel was bound by its instructions.
template <typename T, int P, bool EARLY>
__global__ void __launch_bounds__(kThreads) scatter_quant_group_kernel(const T* __restrict__ x, int groups, int k,
                                                                       const int32_t* __restrict__ row_index,
                                                                       int64_t rows_cap, uint8_t* __restrict__ q,
                                                                       float* __restrict__ scales_t) {
  const int lane = threadIdx.x & 31;
  const int64_t m = blockIdx.y;
  int row = -1;
  uint32_t rows = 0;
  auto fetch_rows = [&] {
    pdl_wait();
    pdl_trigger();
    if (lane < k) row = row_index[m * k + lane];
    rows = __ballot_sync(0xFFFFFFFFu, row >= 0);
  };
  if constexpr (!EARLY) {
    fetch_rows();
    if (rows == 0) return;  // no route of this token is local
  }
  const int64_t K = (int64_t)groups * 128;
  const int step = blockDim.x / 8;  // groups of one pass of the block
  const int g0 = blockIdx.x * P * step + (threadIdx.x >> 3);
  uint4 raw[P][2];
#pragma unroll
  for (int u = 0; u < P; ++u) {
    raw[u][0] = raw[u][1] = make_uint4(0, 0, 0, 0);
    if (g0 + u * step < groups) {
      const uint4* src = reinterpret_cast<const uint4*>(x + m * K + (int64_t)(g0 + u * step) * 128 + (lane & 7) * 16);
      raw[u][0] = EARLY ? __ldcg(src) : src[0];
      raw[u][1] = EARLY ? __ldcg(src + 1) : src[1];
    }
  }
  uint4 packed[P];
  float scale[P];
#pragma unroll
  for (int u = 0; u < P; ++u) {
    const T* pv = reinterpret_cast<const T*>(&raw[u][0]);
    float v[16], amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      v[i] = ToF32<T>::get(pv[i]);
      amax = fmaxf(amax, fabsf(v[i]));
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, off));
    const float s = fmaxf(amax, kQuantEps) * (1.0f / kFp8Max), inv = 1.0f / s;
    const bool finite = s < INFINITY;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float d[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        d[j] = finite ? div_by_scale(v[4 * i + j], s, inv) : v[4 * i + j] / s;
        d[j] = fminf(fmaxf(d[j], -kFp8Max), kFp8Max);
      }
      w[i] = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(d[0], d[1]), __NV_SATFINITE, __NV_E4M3) |
             (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(d[2], d[3]), __NV_SATFINITE, __NV_E4M3) << 16;
    }
    packed[u] = make_uint4(w[0], w[1], w[2], w[3]);
    scale[u] = s;
  }
  if constexpr (EARLY) fetch_rows();
  while (rows != 0) {
    const int64_t r = __shfl_sync(0xFFFFFFFFu, row, __ffs(rows) - 1);
    rows &= rows - 1;
#pragma unroll
    for (int u = 0; u < P; ++u) {
      const int g = g0 + u * step;
      if (g < groups) {
        *reinterpret_cast<uint4*>(q + r * K + (int64_t)g * 128 + (lane & 7) * 16) = packed[u];
        if ((lane & 7) == 0) scales_t[(int64_t)g * rows_cap + r] = scale[u];
      }
    }
  }
}

// Rows of `vec` 16-byte pieces copied as they are; block (c, m): 512 pieces of token m, two per thread.
template <bool EARLY>
__global__ void __launch_bounds__(kThreads) scatter_rows_kernel(const uint4* __restrict__ x, int vec, int k,
                                                                const int32_t* __restrict__ row_index,
                                                                uint4* __restrict__ out) {
  if constexpr (!EARLY) pdl_wait();
  const int64_t m = blockIdx.y;
  const int c = blockIdx.x * 2 * kThreads + threadIdx.x;
  uint4 v[2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (c + i * kThreads < vec) v[i] = __ldcg(x + m * vec + c + i * kThreads);
  if constexpr (EARLY) pdl_wait();
  pdl_trigger();
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

// Block (c, m): blockDim x P 16-byte pieces of token m's output row, P per thread, P x U route rows in flight.  The slots
// without a row are skipped before the loads, so a token with one local route of eight costs one round.
template <typename T, bool WEIGHTED, int P, int U, bool EARLY>
__global__ void __launch_bounds__(kThreads) combine_kernel(const T* __restrict__ y, const float* __restrict__ weight,
                                                           const int32_t* __restrict__ row_index, int k, int vec,
                                                           T* __restrict__ out) {
  if constexpr (!EARLY) pdl_wait();
  constexpr int V = 16 / sizeof(T);
  const int64_t m = blockIdx.y;
  const int lane = threadIdx.x & 31, c0 = blockIdx.x * P * blockDim.x + threadIdx.x;
  const int row = lane < k ? __ldcg(row_index + m * k + lane) : -1;
  const float wl = WEIGHTED && lane < k ? __ldcg(weight + m * k + lane) : 1.0f;
  if constexpr (EARLY) pdl_wait();
  pdl_trigger();
  uint32_t left = __ballot_sync(0xFFFFFFFFu, row >= 0);
  float acc[P][V];
#pragma unroll
  for (int u = 0; u < P; ++u)
#pragma unroll
    for (int i = 0; i < V; ++i) acc[u][i] = 0.0f;
  while (left != 0) {  // slots in order
    uint4 raw[U][P];
    float w[U];
    int n = 0;
#pragma unroll
    for (int s = 0; s < U; ++s) {
      if (left != 0) {
        const int j = __ffs(left) - 1;
        left &= left - 1;
        w[s] = __shfl_sync(0xFFFFFFFFu, wl, j);
        const uint4* src = reinterpret_cast<const uint4*>(y) + (int64_t)__shfl_sync(0xFFFFFFFFu, row, j) * vec;
#pragma unroll
        for (int u = 0; u < P; ++u)
          if (c0 + u * (int)blockDim.x < vec) raw[s][u] = src[c0 + u * blockDim.x];
        n = s + 1;
      }
    }
#pragma unroll
    for (int s = 0; s < U; ++s) {
      if (s < n) {
#pragma unroll
        for (int u = 0; u < P; ++u) {
          const T* p = reinterpret_cast<const T*>(&raw[s][u]);
#pragma unroll
          for (int i = 0; i < V; ++i)
            acc[u][i] = WEIGHTED ? fmaf(w[s], ToF32<T>::get(p[i]), acc[u][i]) : acc[u][i] + ToF32<T>::get(p[i]);
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < P; ++u) {
    if (c0 + u * (int)blockDim.x < vec) {
      uint4 o;
      T* p = reinterpret_cast<T*>(&o);
#pragma unroll
      for (int i = 0; i < V; ++i) p[i] = from_f32<T>(acc[u][i]);
      reinterpret_cast<uint4*>(out)[m * vec + c0 + u * blockDim.x] = o;
    }
  }
}

// What a kernel may read before pdl_wait().  A kernel of the layer call starts when its predecessor has passed its own wait, so
// what is older than the predecessor is complete: for the scatter behind the route plan the tokens, for the combine behind
// GEMM2 the plan and the route weights.  All of it is read past L1.  `early` says that the predecessor is the one of the same
// layer call; the scatters take it below four tokens per SM only: beyond, few blocks fit beside the plan, and a token without a
// local route would be read for nothing.
// us per call, before and with it: DSV3 FP8, 1 token 79.6, 78.6; Qwen3 e4m3 per channel, 500 tokens 135.9, 134.6; from a
// few hundred us of weights on nothing either way.
//
// From four tokens per SM on, a block takes a whole row: its dependent chain (row index, rows, store) is walked once per
// token instead of once per quarter of it (DSV3 FP8, one of 8 ranks, 2000 tokens: layer 308 -> 300 us; 8192 tokens: the
// same).  Below, quarters spread a token over more SMs.
bool whole_rows(int64_t M) { return M >= 4 * sm_count(); }
}  // namespace

// M <= 65535 for all of these (the second grid dimension): the layer call checks it.
int zero_padding(const void* tiles, int64_t tiles_cap, const int32_t* counts, int64_t row_bytes, void* rows, int groups,
                 int64_t rows_cap, float* scales_t, cudaStream_t st) {
  return launch_pdl(zero_padding_kernel, dim3((unsigned)tiles_cap, kPadParts), kThreads, 0, 1, st, "zero padding rows",
                    (const int4*)tiles, counts, (int)(row_bytes / 16), (uint4*)rows, groups, rows_cap, scales_t);
}

int scatter_quant_group(const void* x, int dtype, int64_t M, int H, int k, const int32_t* row_index, int64_t rows_cap, void* q,
                        float* scales_t, bool early, cudaStream_t st) {
  const int groups = H / 128;
  const bool whole = whole_rows(M);
  const int threads = whole ? kThreads : kThreads / 2, per_block = whole ? 64 : 16;
  const dim3 grid((unsigned)((groups + per_block - 1) / per_block), (unsigned)M);
#define MOE_SCATTER(T, P, E)                                                                                                   \
  launch_pdl(scatter_quant_group_kernel<T, P, E>, grid, threads, 0, 1, st, "scatter (1x128 quantised)", (const T*)x, groups, k, \
             row_index, rows_cap, (uint8_t*)q, scales_t)
#define MOE_SCATTER_T(T) (whole ? MOE_SCATTER(T, 2, false) : early ? MOE_SCATTER(T, 1, true) : MOE_SCATTER(T, 1, false))
  return dtype == MOE_BF16 ? MOE_SCATTER_T(__nv_bfloat16) : MOE_SCATTER_T(__half);
#undef MOE_SCATTER_T
#undef MOE_SCATTER
}

int scatter_rows(const void* x, int64_t M, int64_t row_bytes, int k, const int32_t* row_index, void* out, bool early,
                 cudaStream_t st) {
  const int vec = (int)(row_bytes / 16);
  const dim3 grid((unsigned)((vec + 2 * kThreads - 1) / (2 * kThreads)), (unsigned)M);
  return launch_pdl(early ? scatter_rows_kernel<true> : scatter_rows_kernel<false>, grid, kThreads, 0, 1, st, "scatter",
                    (const uint4*)x, vec, k, row_index, (uint4*)out);
}

int scatter_floats(const float* src, int64_t numel, int div, const int32_t* row_index, float* dst, cudaStream_t st) {
  const int64_t blocks = (numel + 255) / 256;
  return launch_pdl(scatter_floats_kernel, dim3((unsigned)(blocks < 1024 ? blocks : 1024)), 256, 0, 1, st, "scatter (floats)", src,
                    numel, div, row_index, dst);
}

int combine_rows(const void* y, int dtype, const float* weight, const int32_t* row_index, int64_t M, int k, int64_t H, void* out,
                 bool early, cudaStream_t st) {
  const int vec = (int)(H / 8);
  const int P = whole_rows(M) ? 4 : 1;
  // equal blocks of whole warps: H = 7168 is 4 x 224 pieces, not 3.5 x 256
  const int blocks = (vec + P * kThreads - 1) / (P * kThreads);
  const int threads = ((vec + P * blocks - 1) / (P * blocks) + 31) / 32 * 32;
  const dim3 grid((unsigned)blocks, (unsigned)M);
#define MOE_COMBINE_P(T, W, P, U, E) \
  launch_pdl(combine_kernel<T, W, P, U, E>, grid, threads, 0, 1, st, "combine", (const T*)y, weight, row_index, k, vec, (T*)out)
#define MOE_COMBINE(T, W)                                                                    \
  (P == 4 ? (early ? MOE_COMBINE_P(T, W, 4, 4, true) : MOE_COMBINE_P(T, W, 4, 4, false))     \
          : (early ? MOE_COMBINE_P(T, W, 1, 8, true) : MOE_COMBINE_P(T, W, 1, 8, false)))
  if (dtype == MOE_BF16) return weight != nullptr ? MOE_COMBINE(__nv_bfloat16, true) : MOE_COMBINE(__nv_bfloat16, false);
  return weight != nullptr ? MOE_COMBINE(__half, true) : MOE_COMBINE(__half, false);
#undef MOE_COMBINE_P
#undef MOE_COMBINE
}

}  // namespace moe
