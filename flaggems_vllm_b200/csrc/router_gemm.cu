// Router GEMM in front of the routers: logits[M, N] = x[M, K] . w[N, K]^T, fp32 accumulate and
// fp32 output, for decode-sized M.  Stands in for router_gemm (bf16 x bf16 -> fp32,
// src/flaggems_vllm/ops/router_gemm.py:207-237) and fp32_router_gemm (bf16/fp32 x fp32 -> fp32,
// src/flaggems_vllm/ops/fp32_router_gemm.py:108-145).
//
// One CTA of 128 threads per tile of token rows and router columns: the weight rows are read once
// per CTA (16-byte loads, each thread a strided set of 8-element chunks), the token rows come from
// L2, every product is formed in fp32 and the reduction order is fixed (lane partial sums ->
// warp shuffle tree -> four warp sums added in warp order), so the result is run-to-run
// deterministic: no split-K atomics.  Bound: latency and L2 bandwidth; algorithmic bytes
// N*K*b_w + M*K*b_x + 4*M*N.
#include <cooperative_groups.h>

#include <type_traits>

#include "tc_common.cuh"

namespace cg = cooperative_groups;

namespace moe {
namespace {

constexpr int kThreads = 128;
constexpr int kRows = 8;
constexpr int kRowStreamMax = 4;

// ROWS tokens x COLS router columns per CTA.  Every (token, column) sum is formed in the same order whatever the
// tile, so the choice below never changes a bit of the result.
template <typename XT, typename WT, int ROWS, int COLS>
__global__ void __launch_bounds__(kThreads) router_gemm_kernel(const XT* __restrict__ x, int64_t x_ld,
                                                                const WT* __restrict__ w, int64_t M, int N, int K,
                                                                float* __restrict__ out) {
  pdl_wait();
  pdl_trigger();
  const int n0 = blockIdx.x * COLS;
  const int64_t m0 = (int64_t)blockIdx.y * ROWS;
  const int rows = (int)min((int64_t)ROWS, M - m0);
  const WT* wr[COLS];
#pragma unroll
  for (int c = 0; c < COLS; ++c) wr[c] = w + (int64_t)min(n0 + c, N - 1) * K;
  float acc[ROWS][COLS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int c = 0; c < COLS; ++c) acc[r][c] = 0.0f;
#pragma unroll(ROWS <= 2 ? 4 : (ROWS <= 4 ? 2 : 1))
  for (int k = threadIdx.x * 8; k < K; k += kThreads * 8) {
    float wv[COLS][8];
#pragma unroll
    for (int c = 0; c < COLS; ++c) load8<WT>(wr[c] + k, wv[c]);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      if (ROWS == 1 || r < rows) {
        float xv[8];
        load8<XT>(x + (m0 + r) * x_ld + k, xv);
#pragma unroll
        for (int c = 0; c < COLS; ++c)
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[r][c] = fmaf(xv[i], wv[c][i], acc[r][c]);
      }
    }
  }
  __shared__ float part[kThreads / 32][ROWS * COLS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
      float v = acc[r][c];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
      if (lane == 0) part[warp][r * COLS + c] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < ROWS * COLS) {
    const int r = threadIdx.x / COLS, n = n0 + threadIdx.x % COLS;
    if (r < rows && n < N) {
      float v = part[0][threadIdx.x];
#pragma unroll
      for (int wi = 1; wi < kThreads / 32; ++wi) v += part[wi][threadIdx.x];
      out[(m0 + r) * N + n] = v;
    }
  }
}

// Batches above the decode sizes: tcgen05 (kind::f16, fp32 accumulators in TMEM), f16 / bf16 operands of
// one type.  A CTA multiplies 128 token rows by BN router columns over K / S elements; the S CTAs of a
// cluster share one output tile, leave their fp32 partial tiles in shared memory and each adds a
// 1/S slice of the rows over the cluster in rank order (distributed shared memory), so the sums are
// run-to-run deterministic and no partial ever goes to memory.  The product is small (256 x 7168
// weights): what bounds it is how many SMs pull operands from L2 at once and the latency of one CTA's
// K loop, hence the split.  Rows and columns beyond the matrix are zero-filled by TMA.
// Launched so that its set-up (barriers, TMEM, the launch itself) overlaps the end of the kernel in front.  What that is worth
// depends on the neighbours; us per call, K = 7168, N = 256, bf16, ordinary launch : this one (neighbour subtracted):
//                                               64 rows     200 rows     1000 rows    2000 rows    8192 rows
//   back to back, stream                        8.3 : 6.0   10.3 : 7.1   12.4 : 10.2  14.7 : 12.3  39.0 : 35.4
//   behind an elementwise kernel, stream        8.2 : 6.2   10.3 : 8.2   13.0 : 11.4  14.4 : 13.2  39.6 : 36.9
//   back to back, graph                         6.5 : 5.4    8.5 : 6.5   10.6 : 9.2   12.5 : 11.8  36.2 : 33.9
//   behind an elementwise kernel, graph         7.0 : 6.5    8.4 : 8.7   10.8 : 11.1  12.8 : 12.7  39.5 : 38.9
constexpr int RBM = 128, RTHREADS = 192;
template <int BN> struct RCfg {
  static constexpr int STAGE = (RBM + BN) * 128;
  // narrow tiles leave room for a second CTA on the SM: clusters of 8 with one CTA per SM do not reach every SM
  static constexpr int STAGES = BN <= 64 ? (BN == 32 ? 5 : 4) : 196608 / STAGE;
  // partial tile: rows of BN + 4 floats (a thread writes its own row: the pad spreads the banks)
  static constexpr int PART = RBM * (BN + 4) * 4;
  static constexpr int RING = STAGES * STAGE > PART ? STAGES * STAGE : PART;
  static constexpr size_t SMEM = (size_t)RING + 1024 + 256;
};
struct RAux {
  uint64_t full[8], empty[8], done;
  uint32_t tmem_base;
};

template <typename T, int BN>
__global__ void __launch_bounds__(RTHREADS, 1) router_tc_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                const __grid_constant__ CUtensorMap map_w, int64_t M,
                                                                int N, int KB, int split, float* __restrict__ out,
                                                                int32_t* status, unsigned long long wait_ns) {
  using namespace tc;
  using C = RCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_1024(smem_raw);
  RAux* aux = reinterpret_cast<RAux*>(smem + C::RING);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = ((int)blockIdx.x / split) * BN;
  const int64_t m0 = (int64_t)blockIdx.y * RBM;
  const int kb0 = (int)((int64_t)KB * rank / split), kb1 = (int)((int64_t)KB * (rank + 1) / split);
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(&aux->full[s], 1); mbar_init(&aux->empty[s], 1); }
    mbar_init(&aux->done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&aux->tmem_base)), "r"(BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = aux->tmem_base;
  pdl_wait();  // the operands and the output may be the kernel's in front
  pdl_trigger();
  if (warp == 0) {
    const bool leader = elect_lane();
    for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
      const int s = it % C::STAGES;
      if (!mbar_wait(&aux->empty[s], ((it / C::STAGES) & 1) ^ 1, status, wait_ns)) break;
      if (!leader) continue;
      mbar_expect_tx(&aux->full[s], C::STAGE);
      tma_load_2d(&map_x, &aux->full[s], smem + (size_t)s * C::STAGE, kb * 64, (int)m0);
      tma_load_2d(&map_w, &aux->full[s], smem + (size_t)s * C::STAGE + RBM * 128, kb * 64, n0);
    }
  } else if (warp == 1) {
    const bool leader = elect_lane();
    constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
    constexpr uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(RBM >> 4) << 24);
    const uint64_t a0 = make_smem_desc(smem_u32(smem)), b0 = make_smem_desc(smem_u32(smem + RBM * 128));
    for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
      const int s = it % C::STAGES;
      if (!mbar_wait(&aux->full[s], (it / C::STAGES) & 1, status, wait_ns)) break;
      tc_fence_after();
      if (!leader) continue;
      const uint64_t ad = a0 + (uint64_t)(s * (C::STAGE >> 4)), bd = b0 + (uint64_t)(s * (C::STAGE >> 4));
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4)
        tc_mma<MMA_F16>(tmem, ad + (uint64_t)(k4 * 2), bd + (uint64_t)(k4 * 2), idesc, (it > 0 || k4 > 0) ? 1u : 0u);
      tc_commit(&aux->empty[s]);
    }
    if (leader) tc_commit(&aux->done);
  } else {
    // every MMA has finished reading the ring: it now holds the partial tile
    const bool ok = warp_agrees(mbar_wait(&aux->done, 0, status, wait_ns));
    tc_fence_after();
    const int row = ((warp & 3) << 5) + lane;
    const uint32_t t0 = tmem + ((uint32_t)((warp & 3) << 5) << 16);
    float* part = reinterpret_cast<float*>(smem) + (size_t)row * (BN + 4);
    const int64_t m = m0 + row;
    if (ok) {
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t r[32];
        tmem_ld32_sync(t0 + (uint32_t)c, r);
        if (split > 1) {
#pragma unroll
          for (int i = 0; i < 8; ++i) reinterpret_cast<uint4*>(part + c)[i] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
        } else if (m < M) {
          float* o = out + m * N + n0 + c;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (N % 4 == 0) {
              if (n0 + c + 4 * i < N) reinterpret_cast<uint4*>(o)[i] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (n0 + c + 4 * i + q < N) o[4 * i + q] = __uint_as_float(r[4 * i + q]);
            }
          }
        }
      }
    }
    tc_fence_before();
  }
  if (split > 1) {
    cluster.sync();
    const int rows = RBM / split, r0 = rank * rows;
    for (int idx = threadIdx.x; idx < rows * (BN / 4); idx += RTHREADS) {
      const int row = r0 + idx / (BN / 4), c = (idx % (BN / 4)) * 4;
      const int64_t m = m0 + row;
      if (m >= M || n0 + c >= N) continue;
      float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      auto add_all = [&](auto ranks) {  // all ranks' partial sums in flight, added in rank order
        constexpr int R = decltype(ranks)::value;
        float4 v[R];
#pragma unroll
        for (int j = 0; j < R; ++j)
          v[j] = *reinterpret_cast<const float4*>(
              cluster.map_shared_rank(reinterpret_cast<float*>(smem), j) + (size_t)row * (BN + 4) + c);
#pragma unroll
        for (int j = 0; j < R; ++j) { sum.x += v[j].x; sum.y += v[j].y; sum.z += v[j].z; sum.w += v[j].w; }
      };
      // a loop for each split: one for eight with a test per rank took 0.7 us more at 2000 rows (split 4)
      if (split == 8) add_all(std::integral_constant<int, 8>());
      else if (split == 4) add_all(std::integral_constant<int, 4>());
      else add_all(std::integral_constant<int, 2>());
      float* o = out + m * N + n0 + c;
      if (N % 4 == 0) {
        *reinterpret_cast<float4*>(o) = sum;
      } else {
        o[0] = sum.x;
        if (n0 + c + 1 < N) o[1] = sum.y;
        if (n0 + c + 2 < N) o[2] = sum.z;
        if (n0 + c + 3 < N) o[3] = sum.w;
      }
    }
    cluster.sync();  // no CTA leaves while its partial tile may still be read
  } else {
    __syncthreads();
  }
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN));
  }
}

template <typename T, int BN>
int launch_tc(const void* x, int64_t x_ld, const void* w, int64_t M, int N, int K, int split, float* out, int32_t* status,
              cudaStream_t st) {
  using C = RCfg<BN>;
  const CUtensorMapDataType dt = std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap mx, mw;
  int rc = tc::make_map(&mx, x, dt, 2, (uint64_t)M, (uint64_t)K, RBM, false, 128, (uint64_t)x_ld);
  if (rc) return rc;
  rc = tc::make_map(&mw, w, dt, 2, (uint64_t)N, (uint64_t)K, BN, true);
  if (rc) return rc;
  auto kern = router_tc_kernel<T, BN>;
  rc = allow_smem((const void*)kern, (int)C::SMEM, split > 8);
  if (rc) return rc;
  const dim3 grid((unsigned)((N + BN - 1) / BN * split), (unsigned)((M + RBM - 1) / RBM));
  return launch_pdl(kern, grid, RTHREADS, C::SMEM, split, st, "router_gemm (tcgen05)", mx, mw, M, N, (K + 63) / 64, split, out, status,
                    wait_limit_ns());
}

// Column tile and K split.  A CTA's K loop advances by the larger of its operand bytes (an SM takes about 64 bytes
// per clock out of L2) and its tensor-core time per 64-element step; the fixed part stands for launch, pipeline
// fill, epilogue and (split) the cluster sum.  `reach` = SMs that clusters of that size fill before a second
// round starts (128 CTAs in clusters of 8, one per SM, took two rounds); narrow tiles run two CTAs per SM, which
// then share its bandwidth.  Of a whole GPU's 148 SMs it is 112 and 132 and not what the occupancy query gives (120 and
// 132 on one GPU; which SMs are fused off differs), so that the order of the sums is one on every B200; a
// partition has its share.  `largest`: most CTAs of a cluster.  N = 256, K = 7168, bf16, us back to back, with tiles of 256 columns :
// up to 128 : 128 with the split of the 256: 2600 rows 17.1 : 26.7 : 21.8, 4000 rows 18.2 : 19.4 : 23.5, 6000 rows 29.6 : 39.4 : 36.7,
// 8192 rows 36.4 : 33.6 : 39.6.  Where narrower tiles were ahead they divided K less, and one accumulator over all of K = 7168 is twice
// as far from 64-bit arithmetic as two (relative 7.9e-6 against 3.8e-6).
void pick_tc(int64_t M, int N, int K, int sms, int largest, int& bn, int& split) {
  const int kb = (K + 63) / 64;
  const int64_t mt = (M + RBM - 1) / RBM;
  double best = 0.0;
  bn = 0;
  for (int b = 32; b <= 256; b *= 2) {
    if (b > 32 && b / 2 >= N) break;
    for (int s = 1; s <= 8 && s <= kb && s <= largest; s *= 2) {
      const double reach = (s == 8 ? 112.0 : (s == 4 ? 132.0 : 148.0)) * sms / 148.0;
      double load = (double)(mt * ((N + b - 1) / b) * s) / reach;
      if (load < 1.0) load = 1.0;
      else if (b > 64 || load > 2.0) load = (double)(int64_t)(load + 0.999);
      const double step = (RBM + b) * 2.0;  // never below the 2 b clocks of the four instructions
      const double cost = load * (((kb + s - 1) / s) * step + 4.0 * b) + 3000.0 + (s > 1 ? 1500.0 + 2.0 * b : 0.0);
      if (bn == 0 || cost < best) { best = cost; bn = b; split = s; }
    }
  }
}

template <typename T, int BN>
bool split_fits(int split) {
  const void* kern = (const void*)router_tc_kernel<T, BN>;
  return allow_smem(kern, (int)RCfg<BN>::SMEM) != 0 || max_clusters(kern, split, RTHREADS, RCfg<BN>::SMEM) != 0;
}
template <typename T>
bool split_fits(int bn, int split) {
  switch (bn) {
    case 32: return split_fits<T, 32>(split);
    case 64: return split_fits<T, 64>(split);
    case 128: return split_fits<T, 128>(split);
    default: return split_fits<T, 256>(split);
  }
}

template <typename T>
int dispatch_tc(const void* x, int64_t x_ld, const void* w, int64_t M, int N, int K, float* out, int32_t* status, cudaStream_t st) {
  int bn = 0, split = 1;
  for (int largest = 8; largest >= 1; largest /= 2) {  // the largest cluster that a partition holds
    pick_tc(M, N, K, sm_count(), largest, bn, split);
    if (split == 1 || split_fits<T>(bn, split)) break;
  }
  switch (bn) {
    case 32: return launch_tc<T, 32>(x, x_ld, w, M, N, K, split, out, status, st);
    case 64: return launch_tc<T, 64>(x, x_ld, w, M, N, K, split, out, status, st);
    case 128: return launch_tc<T, 128>(x, x_ld, w, M, N, K, split, out, status, st);
    default: return launch_tc<T, 256>(x, x_ld, w, M, N, K, split, out, status, st);
  }
}

template <typename XT, typename WT>
int launch_rows(const void* x, int64_t x_ld, const void* w, int64_t M, int N, int K, float* out, cudaStream_t st) {
  // one token: its row and one weight row per CTA, several loads in flight; more tokens than fill one tile of
  // rows: four columns per CTA, so that a token row is fetched from L2 once per four columns
#define MOE_ROWS(ROWS, COLS)                                                                                              \
  launch_pdl(router_gemm_kernel<XT, WT, ROWS, COLS>, dim3((unsigned)((N + COLS - 1) / COLS), (unsigned)((M + ROWS - 1) / ROWS)), \
             kThreads, 0, 1, st, "router_gemm", (const XT*)x, x_ld, (const WT*)w, M, N, K, out)
  if (M == 1) return MOE_ROWS(1, 1);
  if (M == 2) return MOE_ROWS(2, 1);
  if (M <= kRowStreamMax) return MOE_ROWS(kRowStreamMax, 1);
  if (M <= 2 * kRows) return MOE_ROWS(kRows, 1);
  return MOE_ROWS(kRows, 4);
#undef MOE_ROWS
}

template <typename XT>
int launch_w(const void* x, int64_t x_ld, const void* w, int w_dtype, int64_t M, int N, int K, float* out,
             cudaStream_t st) {
  switch (w_dtype) {
    case MOE_F32: return launch_rows<XT, float>(x, x_ld, w, M, N, K, out, st);
    case MOE_F16: return launch_rows<XT, __half>(x, x_ld, w, M, N, K, out, st);
    case MOE_BF16: return launch_rows<XT, __nv_bfloat16>(x, x_ld, w, M, N, K, out, st);
    default: return fail(MOE_E_DTYPE, "router_gemm: unsupported weight dtype %d", w_dtype);
  }
}

}  // namespace
}  // namespace moe

extern "C" int moe_router_gemm_tile(int64_t M, int N, int K, int sms, int largest_cluster, int* columns, int* split) {
  using namespace moe;
  if (M <= 0 || N <= 0 || K <= 0 || sms <= 0 || largest_cluster <= 0 || !columns || !split)
    return fail(MOE_E_BADARG, "router_gemm_tile: bad extent");
  pick_tc(M, N, K, sms, largest_cluster, *columns, *split);
  return 0;
}

extern "C" int moe_router_gemm(const void* x, int x_dtype, int64_t x_ld, const void* w, int w_dtype, int64_t M, int N,
                               int K, float* out, void* stream) {
  return moe_router_gemm_ex(x, x_dtype, x_ld, w, w_dtype, M, N, K, out, nullptr, stream);
}

extern "C" int moe_router_gemm_ex(const void* x, int x_dtype, int64_t x_ld, const void* w, int w_dtype, int64_t M, int N,
                                  int K, float* out, int32_t* status, void* stream) {
  using namespace moe;
  if (M < 0 || N <= 0 || K <= 0) return fail(MOE_E_BADARG, "router_gemm: bad extent");
  if (M == 0) return 0;
  if (!x || !w || !out) return fail(MOE_E_BADARG, "router_gemm: null pointer");
  if (K % 8 != 0 || x_ld % 8 != 0 || x_ld < K) return fail(MOE_E_SHAPE, "router_gemm: K and the row pitch must be multiples of 8");
  if (((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return fail(MOE_E_BADARG, "router_gemm: operands must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  // Half-precision products run on tcgen05 from five rows on (K = 7168, N = 256, graph replay: 6.5-6.9 us for 8 to 128
  // rows, 7.7 for five; the row-streaming kernel 2.7 us for one row, 3.7 for two, 5.2 for four, 10 for eight, 19 for
  // 64).  Below, the row-streaming kernel's reduction order is shared by the fused router
  // (moe_router_gemm_grouped_topk) bit for bit.
  if (M > kRowStreamMax && x_dtype == w_dtype && (x_dtype == MOE_BF16 || x_dtype == MOE_F16) && M < (1ll << 31) - RBM && ((uintptr_t)out & 15) == 0) {
    if ((M + RBM - 1) / RBM > 65535) return fail(MOE_E_TOOBIG, "router_gemm: serves at most %d rows", 65535 * RBM);
    return x_dtype == MOE_BF16 ? dispatch_tc<__nv_bfloat16>(x, x_ld, w, M, N, K, out, status, st)
                               : dispatch_tc<__half>(x, x_ld, w, M, N, K, out, status, st);
  }
  if ((M + kRows - 1) / kRows > 65535) return fail(MOE_E_TOOBIG, "router_gemm: serves at most %d rows", 65535 * kRows);
  switch (x_dtype) {
    case MOE_F32: return launch_w<float>(x, x_ld, w, w_dtype, M, N, K, out, st);
    case MOE_F16: return launch_w<__half>(x, x_ld, w, w_dtype, M, N, K, out, st);
    case MOE_BF16: return launch_w<__nv_bfloat16>(x, x_ld, w, w_dtype, M, N, K, out, st);
    default: return fail(MOE_E_DTYPE, "router_gemm: unsupported input dtype %d", x_dtype);
  }
}
