// Expert grouped GEMMs with the weights as the M operand: a CTA pair (cta_group::2) multiplies 256 weight
// rows, 128 per CTA, by one tile of n <= 256 tokens of an expert, n a multiple of 16.
//
//     D[weight row, token] = W[row, :] . X[token, :]
//
// Why this way round.  With tokens as M (gemm_tc.cu) an expert's rows are padded to 128, a fifth of all rows at
// DeepSeek-V3's prefill sizes, and every CTA fetches 48 KB of operands per 128-byte K block of a 128x256 tile.
// Here the padding is to 16 (route plan, plan.cu), and the pair shares the token tile: each CTA fetches
// its 16 KB of weights and HALF of the tokens (<= 16 KB) and the tensor cores read the other half from the peer.
// Bound at prefill: the clock that power leaves.  Mixtral shape, 16384 tokens: GEMM1 6.73 million cycles, 94 % of them
// MMA, whether the clock in the kernel is 1.30 GHz (after a pause) or 1.10 (sustained); operands not moved and padding
// not multiplied are clock as well as cycles.
//
// Both operands arrive by TMA: token rows were put into sorted order by the scatter kernels (route_rows.cu, quant.cu).  Every load
// of both CTAs counts its bytes on the leader's barrier of the stage; the leader's MMA thread needs no other
// signal from its peer.
//
// Warp roles (384 threads):
//   warp 0      TMA producer (both CTAs; the whole warp runs the loop, one elected lane issues)
//   warp 1      MMA issuer (leader CTA; likewise)
//   warp 2      TMEM allocation: two accumulators of up to 256 columns, so that a tile's epilogue overlaps the next tile's
//               main loop (the whole K loop of a tile accumulates in TMEM)
//   warps 4-11  consumers: warp w owns accumulator lanes 32 (w mod 4)..., group h = (w - 4) / 4 the h-th half
//               of the tile's tokens
// The accumulators are read in the 16x256b shape (tmem_ld_frag32_async): a thread holds neighbouring tokens of lanes
// t/4 and t/4 + 8.  The GEMM1 weight tile is laid out as alternating groups of 8 gate and 8 up rows
// (make_gate_up_map), so those two lanes are gate and up of one output, and SiLU(gate) * up needs no exchange.
// Results are transposed on their way to shared memory by stmatrix.trans and leave as whole rows.
//
// Formats: half precision, and e4m3 / int8 with one scale per row and per output channel, which the epilogue applies
// to the finished sums.  FP8 with block scales stays with tokens as M: its sums leave the tensor core every
// 128 elements of K and are folded with one scale per token.  With tokens along the columns that is a scale per
// register (a shared-memory load each) and twice as many rounds between MMA and fold per byte of weights; it
// measured 1.3 to 1.5 times slower than gemm_tc.cu from one token to 8192.
#include "wt_common.cuh"

namespace moe {
namespace wt {
using namespace tc;

constexpr int WROWS = 128;   // weight rows per CTA
constexpr int A_BYTES = WROWS * 128;
constexpr int THREADS = 384;
constexpr int CONS_THREADS = 256;
// setmaxnreg moves registers inside the CTA's allocation: 128 x 56 + 256 x 224 = 384 x 168
constexpr int LAUNCH_REGS = 168, PRODUCER_REGS = 56, CONSUMER_REGS = 224;
static_assert(128 * PRODUCER_REGS + CONS_THREADS * CONSUMER_REGS <= THREADS * LAUNCH_REGS, "register redistribution");

// NTOK: most tokens of a tile.  With few rows per expert the weights stream, and what they need is bytes in flight: small tiles
// leave the ring to them, ten (64 tokens) or eight and seven (128) stages of 16 KB of weights instead of five and four.
// layer.cu has the figures.
template <bool GEMM1, int NTOK> struct Cfg {
  static constexpr int STAGE_BYTES = A_BYTES + NTOK / 2 * 128;
  static_assert(NTOK == 256 || NTOK == 128 || NTOK == 64, "tile");
  static constexpr int STAGES = NTOK <= 64 ? 10 : (NTOK <= 128 ? (GEMM1 ? 8 : 7) : (GEMM1 ? 5 : 4));
  static constexpr int OUT_BYTES = NTOK * ((GEMM1 ? 64 : 128) * 2 + 16);  // staged rows, see drain_tile
};
struct Aux {
  uint64_t full[10], empty[10];
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  uint32_t pad;
};
template <bool GEMM1, int NTOK> constexpr size_t smem_bytes() {
  using C = Cfg<GEMM1, NTOK>;
  return (size_t)C::STAGES * C::STAGE_BYTES + C::OUT_BYTES + sizeof(Aux) + 1024;
}
static_assert(smem_bytes<true, 256>() <= 232448 && smem_bytes<false, 256>() <= 232448, "shared memory of one SM");
static_assert(smem_bytes<true, 64>() <= 232448 && smem_bytes<false, 64>() <= 232448, "shared memory of one SM");
static_assert(smem_bytes<true, 128>() <= 232448 && smem_bytes<false, 128>() <= 232448, "shared memory of one SM");

// SILU: the activation of GEMM1 (false: swigluoai, which reads GEMM1's result rounded to the activation type)
template <int FMT, typename AT, bool GEMM1, bool SILU, int NTOK>
__global__ void __launch_bounds__(THREADS, 1)
wt_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_b64,
               const __grid_constant__ CUtensorMap map_b16, const __grid_constant__ CUtensorMap map_b8, const Params P) {
  constexpr int KIND = FMT == FMT_HALF ? MMA_F16 : (FMT == FMT_I8ROW ? MMA_I8 : MMA_F8);
  constexpr int KBE = FMT == FMT_HALF ? 64 : 128;  // elements of K per stage
  using C = Cfg<GEMM1, NTOK>;
  constexpr int STAGES = C::STAGES, STAGE_BYTES = C::STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_1024(smem_raw);
  uint8_t* s_out = smem + (size_t)STAGES * STAGE_BYTES;
  Aux* aux = reinterpret_cast<Aux*>(s_out + C::OUT_BYTES);

  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // the compiler sees that `warp` is uniform
  const int KB = (P.K + KBE - 1) / KBE;
  const int cr = (int)cluster_ctarank();  // 0 leads
  const int item0 = blockIdx.x / 2, step = gridDim.x / 2;
  const int total = __ldcg(P.counts) * P.R;  // the route plan is older than the predecessor
  auto fetch = [&](int item) { return fetch_item(P, item); };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&aux->full[s], 1); mbar_init(&aux->empty[s], 1); }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&aux->tmem_full[a], 1);
      mbar_init(&aux->tmem_empty[a], 2 * (CONS_THREADS / 32));  // the warps of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&aux->tmem_base)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anyone signals across
  tc_fence_after();
  const uint32_t tmem_base = aux->tmem_base;
  if (warp != 0) {
    pdl_wait();
    pdl_trigger();
  }

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGS));
    if (warp == 0) {
      // ------------------------------------------------------------ TMA producer
      const bool leader = elect_lane();
      if (leader) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b64) : "memory");
      }
      uint32_t s = 0, ph = 0;
      bool alive = true;
      Item nx = {};
      if (item0 < total) nx = fetch(item0);
      auto load_weights = [&](const Item& it, int kb, uint32_t st) {
        if (cr == 0) mbar_expect_tx(&aux->full[st], 2 * (A_BYTES + (uint32_t)(it.n >> 1) * 128));  // the peer's bytes may already have been counted
        uint8_t* sA = smem + (size_t)st * STAGE_BYTES;
        if constexpr (GEMM1) tma_load_5d_pair(&map_w, &aux->full[st], sA, kb * KBE, 0, 0, it.rt * 16 + cr * 8, it.e);
        else tma_load_2d_pair(&map_w, &aux->full[st], sA, kb * KBE, it.e * P.Nout + it.rt * 256 + cr * 128);
      };
      // the weights of the first stages do not wait for the kernel in front
      int early = 0;
      if (item0 < total) {
        for (; early < STAGES && early < KB; ++early)
          if (leader) load_weights(nx, early, (uint32_t)early);
      }
      pdl_wait();
      for (int item = item0; item < total && alive; item += step) {
        const Item it = nx;
        if (item + step < total) nx = fetch(item + step);
        const int nh = it.n >> 1;                 // this CTA's share of the token rows
        const int brow = it.row0 + cr * nh;
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait_at(smem_u32(&aux->empty[s]), ph ^ 1, P.status, P.wait_ns)) { alive = false; break; }
          if (leader) {
            if (early > 0) --early;
            else load_weights(it, kb, s);
            uint8_t* sB = smem + (size_t)s * STAGE_BYTES + A_BYTES;
            int r = 0;
            for (; nh - r >= 64; r += 64) tma_load_2d_pair(&map_b64, &aux->full[s], sB + r * 128, kb * KBE, brow + r);
            for (; nh - r >= 16; r += 16) tma_load_2d_pair(&map_b16, &aux->full[s], sB + r * 128, kb * KBE, brow + r);
            if (r < nh) tma_load_2d_pair(&map_b8, &aux->full[s], sB + r * 128, kb * KBE, brow + r);
          }
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    } else if (warp == 1 && cr == 0) {
      // ------------------------------------------------------------ MMA issuer
      const bool leader = elect_lane();
      constexpr uint32_t fmt = (FMT == FMT_I8ROW || (FMT == FMT_HALF && std::is_same<AT, __nv_bfloat16>::value)) ? 1u : 0u;
      constexpr uint32_t idesc0 =
          ((FMT == FMT_I8ROW ? 2u : 1u) << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(2 * WROWS >> 4) << 24);
      const uint64_t a0 = make_smem_desc(smem_u32(smem)), b0 = make_smem_desc(smem_u32(smem + A_BYTES));
      const uint32_t full0 = smem_u32(&aux->full[0]);
      constexpr uint32_t TO_EMPTY = (uint32_t)(offsetof(Aux, empty) - offsetof(Aux, full));
      uint32_t full = full0, ph = 0, acc_it = 0;
      uint64_t ad = a0, bd = b0;
      bool alive = true;
      Item nx = {};
      if (item0 < total) nx = fetch(item0);
      for (int item = item0; item < total && alive; item += step) {
        const Item it = nx;
        if (item + step < total) nx = fetch(item + step);
        const uint32_t idesc = idesc0 | ((uint32_t)(it.n >> 3) << 17);
        const uint32_t a = acc_it & 1, d = tmem_base + a * NTOK;
        if (!mbar_wait(&aux->tmem_empty[a], ((acc_it >> 1) & 1) ^ 1, P.status, P.wait_ns)) { alive = false; break; }
#pragma unroll 1
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait_at(full, ph, P.status, P.wait_ns)) { alive = false; break; }
          tc_fence_after();
          tc_mma_block_pair<KIND>(leader, d, ad, bd, idesc, kb > 0, full + TO_EMPTY);
          full += 8;
          ad += (uint64_t)(STAGE_BYTES >> 4);
          bd += (uint64_t)(STAGE_BYTES >> 4);
          if (full == full0 + 8 * STAGES) { full = full0; ad = a0; bd = b0; ph ^= 1; }
        }
        if (leader && alive) tc_commit_pair(&aux->tmem_full[a]);
        ++acc_it;
      }
    }
  } else {
    // -------------------------------------------------------------- consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CONSUMER_REGS));
    const int h = (warp - 4) >> 2, wq = warp & 3;
    const int et = threadIdx.x - 128;
    const uint32_t t_lane = tmem_base + ((uint32_t)(wq << 5) << 16);
    const uint32_t out_base = smem_u32(s_out);
    uint32_t acc_it = 0;
    bool alive = true;
    auto release_acc = [&](uint32_t a) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (cr == 1) mbar_arrive_remote(&aux->tmem_empty[a], 0);
        else mbar_arrive(&aux->tmem_empty[a]);
      }
    };
    Item nx = {};
    if (item0 < total) nx = fetch(item0);
    // The tile loop runs to its end even after a wait has timed out: every consumer thread reaches
    // the named barriers of every tile.
    for (int item = item0; item < total; item += step) {
      const Item it = nx;
      if (item + step < total) nx = fetch(item + step);
      const uint32_t a = acc_it & 1;
      asm volatile("bar.sync 2, %0;" ::"n"(CONS_THREADS) : "memory");  // the staging tile has been read
      if (alive) alive = warp_agrees(mbar_wait_idle(&aux->tmem_full[a], (acc_it >> 1) & 1, P.status, P.wait_ns));
      if (alive) {
        tc_fence_after();
        drain_tile<FMT, AT, GEMM1, SILU, 2, 2, 0>(P, it, cr, t_lane + a * NTOK, h, wq, lane, out_base, [&] { release_acc(a); });
        ++acc_it;
      }
      asm volatile("bar.sync 2, %0;" ::"n"(CONS_THREADS) : "memory");  // the tile is staged
      if (alive) store_rows<AT, GEMM1, 2, CONS_THREADS>(P, it, cr, s_out, et);
    }
  }

  // -------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // no CTA leaves while its partner may still signal its barriers
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
  }
}

// ------------------------------------------------------------------ host side
template <int FMT, typename AT, bool GEMM1, bool SILU, int NTOK>
static int launch(const CUtensorMap& mw, const CUtensorMap (&mb)[3], const Params& P, int grid, cudaStream_t st) {
  auto kern = wt_gemm_kernel<FMT, AT, GEMM1, SILU, NTOK>;
  constexpr size_t smem = smem_bytes<GEMM1, NTOK>();
  static const int regs = [&] {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, kern) == cudaSuccess ? fa.numRegs : 0;
  }();
  // refuse to launch rather than let setmaxnreg.inc wait for registers that do not exist
  if (128 * PRODUCER_REGS + CONS_THREADS * CONSUMER_REGS > THREADS * regs)
    return fail(MOE_E_DRIVER, "grouped GEMM: kernel was built with %d registers per thread, %d needed", regs, LAUNCH_REGS);
  const int rc = allow_smem((const void*)kern, (int)smem);
  if (rc) return rc;
  return launch_pdl(kern, dim3((unsigned)grid), THREADS, smem, 2, st, GEMM1 ? "gemm1 (pair, weights as M)" : "gemm2 (pair, weights as M)",
                    mw, mb[0], mb[1], mb[2], P);
}

}  // namespace wt

bool wt_serves(int mode, int act_dtype, int H, int I) {
  if (act_dtype != MOE_BF16 && act_dtype != MOE_F16) return false;
  if (mode == MOE_MODE_HALF) return H % 64 == 0 && I % 128 == 0;
  return (mode == MOE_MODE_FP8_ROW || mode == MOE_MODE_INT8_ROW) && H % 128 == 0 && I % 128 == 0;
}

// a: [rows_cap, K] operand rows in the order of the route plan, whose tiles have at most `tile_rows` rows
int wt_gemm(bool gemm1, int mode, int tile_rows, int act_dtype, const void* a, const float* a_scales, const void* w, const float* w_scale,
            const void* tiles, int64_t tiles_cap, const int32_t* counts, const float* row_weight, int64_t rows_cap, int E, int K,
            int Nout, void* out, int act_kind, float alpha, float beta, float limit, int32_t* status,
            cudaStream_t st) {
  using namespace wt;
  const bool half = mode == MOE_MODE_HALF;
  const int eb = half ? 2 : 1;
  const int64_t rows_w = gemm1 ? 2 * (int64_t)Nout : Nout;
  if ((int64_t)E * rows_w >= (1ll << 31) || rows_cap >= (1ll << 31)) return fail(MOE_E_TOOBIG, "grouped GEMM: extent exceeds int32 coordinates");
  const CUtensorMapDataType dt = half ? (act_dtype == MOE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16)
                                      : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  CUtensorMap mw, mb[3];
  int rc = gemm1 ? make_gate_up_map(&mw, w, dt, eb, (uint64_t)E, (uint64_t)Nout, (uint64_t)K)
                 : make_map(&mw, w, dt, eb, (uint64_t)E * rows_w, (uint64_t)K, WROWS, true);
  const uint32_t box[3] = {64, 16, 8};
  for (int i = 0; i < 3 && !rc; ++i) rc = make_map(&mb[i], a, dt, eb, (uint64_t)rows_cap, (uint64_t)K, box[i], false);
  if (rc) return rc;
  Params P;
  P.tiles = (const int4*)tiles; P.counts = counts; P.a_scales = a_scales; P.w_scale = w_scale; P.row_weight = row_weight;
  P.out = out; P.status = status; P.wait_ns = wait_limit_ns();
  P.E = E; P.K = K; P.Nout = Nout; P.R = gemm1 ? Nout / 128 : (Nout + 255) / 256;
  P.alpha = alpha; P.beta = beta; P.limit = limit;
  const int64_t items = tiles_cap * P.R;
  const int pairs = sm_count() / 2;
  const int grid = 2 * (int)(items < pairs ? items : pairs);
  // the kernel of the plan's tiles: 64 (half precision), 128 or 256 rows (layer.cu); the other activation has one
  auto go = [&](auto F, auto T) {
    constexpr int FMT = decltype(F)::value;
    using AT = decltype(T);
    if (gemm1 && act_kind != MOE_ACT_SILU) return launch<FMT, AT, true, false, 256>(mw, mb, P, grid, st);
    auto sized = [&](auto N) {
      constexpr int NTOK = decltype(N)::value;
      return gemm1 ? launch<FMT, AT, true, true, NTOK>(mw, mb, P, grid, st) : launch<FMT, AT, false, true, NTOK>(mw, mb, P, grid, st);
    };
    if constexpr (FMT == FMT_HALF) {
      if (tile_rows <= 64) return sized(std::integral_constant<int, 64>());
    }
    return tile_rows <= 128 ? sized(std::integral_constant<int, 128>()) : sized(std::integral_constant<int, 256>());
  };
  auto typed = [&](auto F) { return act_dtype == MOE_BF16 ? go(F, __nv_bfloat16()) : go(F, __half()); };
  switch (mode) {
    case MOE_MODE_HALF: return typed(std::integral_constant<int, FMT_HALF>());
    case MOE_MODE_FP8_ROW: return typed(std::integral_constant<int, FMT_FP8ROW>());
    case MOE_MODE_INT8_ROW: return typed(std::integral_constant<int, FMT_I8ROW>());
    default: return fail(MOE_E_BADARG, "grouped GEMM: mode %d", mode);
  }
}

}  // namespace moe
