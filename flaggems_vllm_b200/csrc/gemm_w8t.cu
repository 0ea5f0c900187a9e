// Weight-only int8 grouped GEMMs with the widened weights as the tensor-memory operand.
//
//     D[weight row, token] = (int8 W[row, :] widened exactly to f16 / bf16) . X[token, :],   channel scale at the end
//
// gemm_w8.cu widens the weights into shared memory, where every 128x256 tile moves 128 KB per 64 elements of K: raw
// bytes in and out, widened bytes in and out, activations in and out; 1400 cycles for 512 cycles of MMA.  Here the
// weights are the M operand, so their widened form can live in TENSOR MEMORY: converter warps read the raw bytes
// (each byte once), widen them in registers and write them with tcgen05.st, and the MMA takes A from there
// (tcgen05.mma with a TMEM A operand).  Shared memory only sees the raw bytes and the token rows.
//
// One CTA, 128 weight rows by up to 64 tokens (decode batches: deep rings, the weights stream) or by up to 160
// tokens (WIDE, prefill: the token rows are fetched and the weights widened for as many tokens as the accumulators
// hold twice).
// K is consumed 128 elements at a time: 16 KB of raw weights and two 64-element sub-tiles of the token rows.
//
// Warp roles (640 threads):
//   warp 0       TMA: raw weights
//   warp 1       MMA issuer
//   warp 2       TMEM allocation: two accumulators of 160 (64) columns, three (six) A buffers of 64 columns
//   warp 3       TMA: token rows
//   warps 4-7    epilogue (drain_tile)
//   warps 8-19   converters: three groups of four warps; group g owns every third A buffer and K block, warp quarter
//                q the 32 weight rows = TMEM lanes 32 q...  A thread widens one row of 128 bytes; the 128-byte
//                swizzle of the raw tile makes its 16-byte loads conflict-free.
// TMEM columns hold two elements of K each, so an MMA (16 elements) takes 8 columns of A.
//
// Bound.  Decode: HBM, less the last partial wave; before, the MMA warp's chain of a K block, two waits, eight
// instructions and two commits.  Now a K block is one wait, one statement of eight instructions and ONE commit (token rows and
// widened weights of a K block share a stage index), the loops carry their addresses, and an epilogue warp stages 16 tokens
// of its own rows instead of a tile of everybody's (no barriers, and room for twice the raw stages).  GEMM1 / GEMM2 back to
// back, Qwen3 shape, us: 33 tokens 64.7 / 37.7 -> 59.7 / 31.9, 500 tokens 89 / 50 -> 78 / 42, 4096 tokens 228 / 128 -> 218 /
// 122.  A second commit and wait per K block (token stages of half a K block, four blocks of them) measured 78.6 / 45.0 at 33
// tokens and 247 / 136 at 4096.  Prefill: no single part.  Copies that skip work, on a GPU where GEMM1 takes 208 us: without the
// token loads 162, with one of the eight MMAs 171, without raw loads 179, without widening 186, without epilogue 195.
// Against gemm_w8.cu: 33 tokens 191 -> 118 us per layer, 4096 tokens 591 -> 455.
#include "wt_common.cuh"

namespace moe {
namespace w8t {
using namespace wt;

constexpr int THREADS = 640, EPI_THREADS = 128, GROUPS = 3;
constexpr int RAW_BYTES = 128 * 128;
constexpr int LAUNCH_REGS = 96, PRODUCER_REGS = 40, EPI_REGS = 144;  // converters keep what they were launched with
static_assert(128 * PRODUCER_REGS + 128 * EPI_REGS + 384 * LAUNCH_REGS <= THREADS * LAUNCH_REGS, "register redistribution");

template <bool WIDE> struct Cfg {
  static constexpr int TILE = WIDE ? 160 : 64;     // most tokens of a tile
  static constexpr int SUB_BYTES = TILE * 128;     // 64 elements of K of the token rows
  static constexpr int TOK_BYTES = 2 * SUB_BYTES;
  // stages: a K block's token rows in shared memory and its widened weights in tensor memory; raw stages
  static constexpr int STAGES = WIDE ? 3 : 6, RSTAGES = 6;
  static constexpr int A_COLS = 64, A_BASE = 2 * TILE;  // TMEM: two accumulators, then the widened weights
  static_assert(A_BASE + STAGES * A_COLS <= 512, "TMEM columns");
  // Every stage belongs to ONE converter group, which has seen the use before the one it waits for.  With five raw
  // stages a group could wait two uses ahead of a late load: the parity wait lets it pass, it hands the stage back too
  // early, and the launch fails, about once in a thousand layers.
  static_assert(RSTAGES % GROUPS == 0 && STAGES % GROUPS == 0, "stages per converter group");
};
// What one K block costs the MMA warp is what bounds this kernel, so a K block has one barrier to wait for and one to
// commit to: ready[s] counts the token rows (bytes) and the four converter warps, done[s] frees both.
struct Aux {
  uint64_t r_full[6], r_empty[6];
  uint64_t ready[6], done[6];
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  uint32_t pad;
};
constexpr int OUT_TOKENS = 16, OUT_BYTES = OUT_TOKENS * (32 * 2 + 16);  // staging buffer of an epilogue warp (drain_tile)
template <bool WIDE> constexpr size_t smem_bytes() {
  using C = Cfg<WIDE>;
  return (size_t)C::RSTAGES * RAW_BYTES + (size_t)C::STAGES * C::TOK_BYTES + EPI_THREADS / 32 * OUT_BYTES + sizeof(Aux) + 1024;
}
static_assert(smem_bytes<true>() <= 232448 && smem_bytes<false>() <= 232448, "shared memory of one SM");

__device__ __forceinline__ void tma_load_5d(const CUtensorMap* map, uint64_t* bar, void* dst, int c0, int c1, int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
// A K block (128 elements, eight instructions) with A from tensor memory, and the commit to the stage's barrier, by the lane
// where `yes`, in one statement
template <int SUB_BYTES>
__device__ __forceinline__ void mma_ts_block(bool yes, uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool acc, uint32_t done) {
  asm volatile(
      "{\n\t.reg .pred l, p, t;\n\t.reg .b64 b1, b2, b3, b4, b5, b6, b7;\n\t.reg .b32 a1, a2, a3, a4, a5, a6, a7;\n\t"
      "setp.ne.b32 l, %0, 0;\n\tsetp.ne.b32 p, %5, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "add.s64 b1, %3, 2;\n\tadd.s64 b2, %3, 4;\n\tadd.s64 b3, %3, 6;\n\tadd.s64 b4, %3, %7;\n\t"
      "add.s64 b5, b4, 2;\n\tadd.s64 b6, b4, 4;\n\tadd.s64 b7, b4, 6;\n\t"
      "add.u32 a1, %2, 8;\n\tadd.u32 a2, %2, 16;\n\tadd.u32 a3, %2, 24;\n\tadd.u32 a4, %2, 32;\n\t"
      "add.u32 a5, %2, 40;\n\tadd.u32 a6, %2, 48;\n\tadd.u32 a7, %2, 56;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], %3, %4, p;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%1], [a1], b1, %4, t;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%1], [a2], b2, %4, t;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%1], [a3], b3, %4, t;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%1], [a4], b4, %4, t;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%1], [a5], b5, %4, t;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%1], [a6], b6, %4, t;\n\t"
      "@l tcgen05.mma.cta_group::1.kind::f16 [%1], [a7], b7, %4, t;\n\t"
      "@l tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t}"
      ::"r"((uint32_t)yes), "r"(d), "r"(a), "l"(b), "r"(idesc), "r"((uint32_t)acc), "r"(done), "n"(SUB_BYTES >> 4)
      : "memory");
}
#define MOE_S8(a, o) "r"(a[o]), "r"(a[o + 1]), "r"(a[o + 2]), "r"(a[o + 3]), "r"(a[o + 4]), "r"(a[o + 5]), "r"(a[o + 6]), "r"(a[o + 7])
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&a)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
      ::MOE_S8(a, 0), MOE_S8(a, 8), MOE_S8(a, 16), MOE_S8(a, 24), "r"(taddr)
      : "memory");
}
#undef MOE_S8

template <typename AT, bool GEMM1, bool WIDE>
__global__ void __launch_bounds__(THREADS, 1)
w8t_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_b64,
                const __grid_constant__ CUtensorMap map_b16, const __grid_constant__ CUtensorMap map_b8, const Params P) {
  using C = Cfg<WIDE>;
  constexpr int RSTAGES = C::RSTAGES, STAGES = C::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_1024(smem_raw);
  uint8_t* s_tok = smem + (size_t)RSTAGES * RAW_BYTES;
  uint8_t* s_out = s_tok + (size_t)STAGES * C::TOK_BYTES;
  Aux* aux = reinterpret_cast<Aux*>(s_out + EPI_THREADS / 32 * OUT_BYTES);

  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // the compiler sees that `warp` is uniform
  const int KB = (P.K + 127) / 128;
  const int item0 = blockIdx.x, step = gridDim.x;
  const int total = __ldcg(P.counts) * P.R;  // the route plan is older than the predecessor
  auto fetch = [&](int item) { return fetch_item(P, item); };

  if (threadIdx.x == 0) {
    for (int s = 0; s < RSTAGES; ++s) { mbar_init(&aux->r_full[s], 1); mbar_init(&aux->r_empty[s], 4); }
    for (int s = 0; s < STAGES; ++s) { mbar_init(&aux->ready[s], 1 + 4); mbar_init(&aux->done[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&aux->tmem_full[a], 1); mbar_init(&aux->tmem_empty[a], 4); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&aux->tmem_base)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = aux->tmem_base;

  // the weights, their widening and the tensor core do not wait for the kernel in front; the token rows and the
  // results do
  if (warp >= 3 && warp < 8) {
    pdl_wait();
    pdl_trigger();
  }
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGS));
    bool alive = true;
    Item nx = {};
    if (item0 < total) nx = fetch(item0);
    if (warp == 0) {
      // ------------------------------------------------------------ raw weights
      const bool leader = elect_lane();
      if (leader) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
      uint32_t s = 0, ph = 0;
      for (int item = item0; item < total && alive; item += step) {
        const Item it = nx;
        if (item + step < total) nx = fetch(item + step);
        const int wrow = GEMM1 ? it.rt * 8 : it.e * P.Nout + it.rt * 128;
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait_at(smem_u32(&aux->r_empty[s]), ph ^ 1, P.status, P.wait_ns)) { alive = false; break; }
          if (leader) {
            mbar_expect_tx(&aux->r_full[s], RAW_BYTES);
            if constexpr (GEMM1) tma_load_5d(&map_w, &aux->r_full[s], smem + (size_t)s * RAW_BYTES, kb * 128, 0, 0, wrow, it.e);
            else tma_load_2d(&map_w, &aux->r_full[s], smem + (size_t)s * RAW_BYTES, kb * 128, wrow);
          }
          if (++s == RSTAGES) { s = 0; ph ^= 1; }
        }
      }
    } else if (warp == 3) {
      // ------------------------------------------------------------ token rows
      const bool leader = elect_lane();
      if (leader) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b8) : "memory");
      uint32_t s = 0, ph = 0;
      for (int item = item0; item < total && alive; item += step) {
        const Item it = nx;
        if (item + step < total) nx = fetch(item + step);
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait_at(smem_u32(&aux->done[s]), ph ^ 1, P.status, P.wait_ns)) { alive = false; break; }
          if (leader) {
            mbar_expect_tx(&aux->ready[s], (uint32_t)it.n * 256);  // both sub-tiles
#pragma unroll
            for (int sub = 0; sub < 2; ++sub) {
              uint8_t* dst = s_tok + (size_t)s * C::TOK_BYTES + sub * C::SUB_BYTES;
              const int k0 = kb * 128 + sub * 64;
              int r = 0;
              for (; it.n - r >= 64; r += 64) tma_load_2d(&map_b64, &aux->ready[s], dst + r * 128, k0, it.row0 + r);
              for (; it.n - r >= 16; r += 16) tma_load_2d(&map_b16, &aux->ready[s], dst + r * 128, k0, it.row0 + r);
              if (r < it.n) tma_load_2d(&map_b8, &aux->ready[s], dst + r * 128, k0, it.row0 + r);
            }
          }
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------ MMA issuer
      const bool leader = elect_lane();
      constexpr uint32_t fmt = std::is_same<AT, __nv_bfloat16>::value ? 1u : 0u;
      constexpr uint32_t idesc0 = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(128 >> 4) << 24);
      const uint64_t b0 = make_smem_desc(smem_u32(s_tok));
      const uint32_t ready0 = smem_u32(&aux->ready[0]), a0 = tmem_base + C::A_BASE;
      constexpr uint32_t TO_DONE = (uint32_t)(offsetof(Aux, done) - offsetof(Aux, ready));
      uint32_t ready = ready0, ph = 0, ta = a0, acc_it = 0;
      uint64_t bd = b0;
      for (int item = item0; item < total && alive; item += step) {
        const Item it = nx;
        if (item + step < total) nx = fetch(item + step);
        const uint32_t idesc = idesc0 | ((uint32_t)(it.n >> 3) << 17);
        const uint32_t a = acc_it & 1, d = tmem_base + a * C::TILE;
        if (!mbar_wait(&aux->tmem_empty[a], ((acc_it >> 1) & 1) ^ 1, P.status, P.wait_ns)) { alive = false; break; }
#pragma unroll 1
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait_at(ready, ph, P.status, P.wait_ns)) { alive = false; break; }
          tc_fence_after();
          mma_ts_block<C::SUB_BYTES>(leader, d, ta, bd, idesc, kb > 0, ready + TO_DONE);
          ready += 8;
          ta += C::A_COLS;
          bd += (uint64_t)(C::TOK_BYTES >> 4);
          if (ready == ready0 + 8 * STAGES) { ready = ready0; ta = a0; bd = b0; ph ^= 1; }
        }
        if (leader && alive) tc_commit(&aux->tmem_full[a]);
        ++acc_it;
      }
    }
  } else if (warp < 8) {
    // -------------------------------------------------------------- epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EPI_REGS));
    const int wq = warp & 3;
    const uint32_t t_lane = tmem_base + ((uint32_t)(wq << 5) << 16);
    const uint32_t out_base = smem_u32(s_out) + wq * OUT_BYTES;
    uint32_t acc_it = 0;
    Item nx = {};
    if (item0 < total) nx = fetch(item0);
    for (int item = item0; item < total; item += step) {
      const Item it = nx;
      if (item + step < total) nx = fetch(item + step);
      const uint32_t a = acc_it & 1;
      if (!warp_agrees(mbar_wait_idle(&aux->tmem_full[a], (acc_it >> 1) & 1, P.status, P.wait_ns))) break;
      tc_fence_after();
      drain_tile<FMT_W8, AT, GEMM1, true, 1, 1, OUT_TOKENS>(P, it, 0, t_lane + a * C::TILE, 0, wq, lane, out_base, [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&aux->tmem_empty[a]);
      });
      ++acc_it;
    }
  } else {
    // -------------------------------------------------------------- converters
    const int grp = (warp - 8) >> 2, wq = warp & 3;
    const int row = wq * 32 + lane;
    const uint32_t t_lane = tmem_base + ((uint32_t)(wq << 5) << 16) + C::A_BASE;
    // K blocks of all tiles in one sequence; this group takes every third of them
    const int tiles = item0 < total ? (total - item0 + step - 1) / step : 0;
    const int64_t blocks = (int64_t)tiles * KB;
    uint32_t rs = grp, rph = 0, s = grp, ph = 1;
    for (int64_t j = grp; j < blocks; j += GROUPS) {
      if (!warp_agrees(mbar_wait_at(smem_u32(&aux->r_full[rs]), rph, P.status, P.wait_ns))) break;
      const uint8_t* src = smem + (size_t)rs * RAW_BYTES + row * 128;
      const uint32_t ta = t_lane + s * C::A_COLS;
      bool ok = true;
      uint4 raw[4];
      uint32_t w[32];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int c = 0; c < 4; ++c)  // 16-byte chunk XOR (row mod 8): TMA's 128-byte swizzle
          raw[c] = *reinterpret_cast<const uint4*>(src + (((half * 4 + c) ^ (row & 7)) << 4));
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          widen4<AT>(raw[c].x, w[c * 8 + 0], w[c * 8 + 1]);
          widen4<AT>(raw[c].y, w[c * 8 + 2], w[c * 8 + 3]);
          widen4<AT>(raw[c].z, w[c * 8 + 4], w[c * 8 + 5]);
          widen4<AT>(raw[c].w, w[c * 8 + 6], w[c * 8 + 7]);
        }
        if (half == 0) {
          // the buffer's last MMA is over (the wait comes after the first half is widened)
          ok = warp_agrees(mbar_wait_at(smem_u32(&aux->done[s]), ph, P.status, P.wait_ns));
          if (!ok) break;
          tc_fence_after();
        }
        tmem_st32(ta + half * 32, w);
      }
      if (!ok) break;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      mbar_arrive_at<0>(smem_u32(&aux->r_empty[rs]), lane == 0);
      mbar_arrive_at<0>(smem_u32(&aux->ready[s]), lane == 0);
      rs += GROUPS;
      if (rs >= RSTAGES) { rs -= RSTAGES; rph ^= 1; }
      s += GROUPS;
      if (s >= STAGES) { s -= STAGES; ph ^= 1; }
    }
  }

  // -------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
  }
}

// ------------------------------------------------------------------ host side
template <typename AT, bool GEMM1, bool WIDE>
static int launch(const CUtensorMap& mw, const CUtensorMap (&mb)[3], const Params& P, int64_t items, cudaStream_t st) {
  auto kern = w8t_gemm_kernel<AT, GEMM1, WIDE>;
  constexpr size_t smem = smem_bytes<WIDE>();
  static const int regs = [&] {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, kern) == cudaSuccess ? fa.numRegs : 0;
  }();
  // refuse to launch rather than let setmaxnreg.inc wait for registers that do not exist
  if (128 * PRODUCER_REGS + 128 * EPI_REGS > 256 * regs)
    return fail(MOE_E_DRIVER, "int8-weight GEMM: kernel was built with %d registers per thread, %d needed", regs, LAUNCH_REGS);
  const int rc = allow_smem((const void*)kern, (int)smem);
  if (rc) return rc;
  const int sms = sm_count();
  return launch_pdl(kern, dim3((unsigned)(items < sms ? items : sms)), THREADS, smem, 1, st,
                    GEMM1 ? "gemm1 (int8 weights, TMEM)" : "gemm2 (int8 weights, TMEM)", mw, mb[0], mb[1], mb[2], P);
}

}  // namespace w8t

bool w8t_serves(int act_dtype, int H, int I) {
  return (act_dtype == MOE_BF16 || act_dtype == MOE_F16) && H % 64 == 0 && I % 128 == 0;
}
// most rows of a tile of the two variants
int w8t_tile(bool wide) { return wide ? w8t::Cfg<true>::TILE : w8t::Cfg<false>::TILE; }

// a: [rows_cap, K] activation rows in the order of the route plan
int w8t_gemm(bool gemm1, bool wide, int act_dtype, const void* a, const void* w, const float* w_scale, const void* tiles,
             int64_t tiles_cap, const int32_t* counts, const float* row_weight, int64_t rows_cap, int E, int K, int Nout, void* out,
             int32_t* status, cudaStream_t st) {
  using namespace w8t;
  const int64_t rows_w = gemm1 ? 2 * (int64_t)Nout : Nout;
  if ((int64_t)E * rows_w >= (1ll << 31) || rows_cap >= (1ll << 31)) return fail(MOE_E_TOOBIG, "int8-weight GEMM: extent exceeds int32 coordinates");
  const CUtensorMapDataType dt = act_dtype == MOE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap mw, mb[3];
  int rc = gemm1 ? make_gate_up_map(&mw, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)E, (uint64_t)Nout, (uint64_t)K)
                 : make_map(&mw, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)E * rows_w, (uint64_t)K, 128, true);
  const uint32_t box[3] = {64, 16, 8};
  for (int i = 0; i < 3 && !rc; ++i) rc = make_map(&mb[i], a, dt, 2, (uint64_t)rows_cap, (uint64_t)K, box[i], false);
  if (rc) return rc;
  Params P = {};
  P.tiles = (const int4*)tiles; P.counts = counts; P.w_scale = w_scale; P.row_weight = row_weight; P.out = out; P.status = status;
  P.wait_ns = wait_limit_ns(); P.E = E; P.K = K; P.Nout = Nout;
  const int cols = gemm1 ? 64 : 128;
  P.R = (Nout + cols - 1) / cols;
  const int64_t items = tiles_cap * P.R;
#define MOE_W8T(T)                                                                                            \
  (gemm1 ? (wide ? launch<T, true, true>(mw, mb, P, items, st) : launch<T, true, false>(mw, mb, P, items, st)) \
         : (wide ? launch<T, false, true>(mw, mb, P, items, st) : launch<T, false, false>(mw, mb, P, items, st)))
  return act_dtype == MOE_BF16 ? MOE_W8T(__nv_bfloat16) : MOE_W8T(__half);
#undef MOE_W8T
}

}  // namespace moe
