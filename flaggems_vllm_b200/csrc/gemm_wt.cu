// Expert grouped GEMMs with the weights as the M operand: a CTA pair (cta_group::2) multiplies 256 weight
// rows, 128 per CTA, by one tile of n <= 256 tokens of an expert, n a multiple of 16.
//
//     D[weight row, token] = W[row, :] . X[token, :]
//
// Why this way round.  With tokens as M (gemm_tc.cu) an expert's rows are padded to 128, a fifth of all rows at
// DeepSeek-V3's prefill sizes, and every CTA fetches 48 KB of operands per 128-byte K block of a 128x256 tile.
// Here the padding is to 16 (route plan, plan.cu), and the pair shares the token tile: each CTA fetches
// its 16 KB of weights and HALF of the tokens (<= 16 KB) and the tensor cores read the other half from the peer.
// At prefill sizes the board runs at its power limit, so operands not moved and padding not multiplied are
// clock as well as cycles.
//
// Both operands arrive by TMA: token rows were put into sorted order by the scatter kernels (quant.cu).  Every load
// of both CTAs counts its bytes on the leader's barrier of the stage; the leader's MMA thread needs no other
// signal from its peer.
//
// Warp roles (384 threads):
//   warp 0      TMA producer (both CTAs; the whole warp runs the loop, one elected lane issues)
//   warp 1      MMA issuer (leader CTA; likewise)
//   warp 2      TMEM allocation: two accumulators of 256 columns, so that a tile's epilogue overlaps the next tile's
//               main loop (the whole K loop of a tile accumulates in TMEM)
//   warps 4-11  consumers: warp w owns accumulator lanes 32 (w mod 4)..., group h = (w - 4) / 4 the h-th half
//               of the tile's tokens
// The accumulators are read in the 16x256b shape (tmem_ld_frag32_async): a thread holds neighbouring tokens of lanes
// t/4 and t/4 + 8.  The GEMM1 weight tile is laid out as alternating groups of 8 gate and 8 up rows
// (make_gate_up_map), so those two lanes are gate and up of one output, and SiLU(gate) * up needs no exchange.
// Results are transposed on their way to shared memory by stmatrix.trans and leave as whole rows.
//
//
// Formats: half precision, and e4m3 / int8 with one scale per row and per output channel, which the epilogue applies
// to the finished sums.  FP8 with block scales stays with tokens as M: its sums leave the tensor core every
// 128 elements of K and are folded with one scale per token.  With tokens along the columns that is a scale per
// register (a shared-memory load each) and twice as many rounds between MMA and fold per byte of weights; it
// measured 1.3 to 1.5 times slower than gemm_tc.cu from one token to 8192.
#include "tc_common.cuh"

namespace moe {
namespace wt {
using namespace tc;

constexpr int FMT_HALF = 0, FMT_FP8ROW = 2, FMT_I8ROW = 3;
constexpr int WROWS = 128;   // weight rows per CTA
constexpr int NTOK = 256;    // most tokens of a tile
constexpr int A_BYTES = WROWS * 128;
constexpr int B_BYTES = NTOK / 2 * 128;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int THREADS = 384;
constexpr int CONS_THREADS = 256;
// setmaxnreg moves registers inside the CTA's allocation: 128 x 56 + 256 x 224 = 384 x 168
constexpr int LAUNCH_REGS = 168, PRODUCER_REGS = 56, CONSUMER_REGS = 224;
static_assert(128 * PRODUCER_REGS + CONS_THREADS * CONSUMER_REGS <= THREADS * LAUNCH_REGS, "register redistribution");

template <bool GEMM1> struct Cfg {
  static constexpr int STAGES = GEMM1 ? 5 : 4;
  static constexpr int OUT_COLS = GEMM1 ? 64 : 128;            // output columns per CTA
  static constexpr int OUT_PITCH = OUT_COLS * 2 + 16;          // bytes; the 16 spread stmatrix rows over the banks
  static constexpr int OUT_BYTES = NTOK * OUT_PITCH;
};
struct Aux {
  uint64_t full[6], empty[6];
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  uint32_t pad;
};
template <bool GEMM1> constexpr size_t smem_bytes() {
  return (size_t)Cfg<GEMM1>::STAGES * STAGE_BYTES + Cfg<GEMM1>::OUT_BYTES + sizeof(Aux) + 1024;
}
static_assert(smem_bytes<true>() <= 232448 && smem_bytes<false>() <= 232448, "shared memory of one SM");

struct Params {
  const int4* tiles;        // {first row, rows | occupied rows << 16, expert, first tile of the expert | its tile count << 16}
  const int32_t* counts;    // [0] = number of tiles
  const float* a_scales;    // row-scaled: [rows_cap]
  const float* w_scale;     // row-scaled: [E, rows_w]
  const float* row_weight;  // GEMM1 with the route weight on the input: [rows_cap], else null
  void* out;                // GEMM1: [rows_cap, I]; GEMM2: [rows_cap, H]
  int32_t* status;
  unsigned long long wait_ns;
  int E, K, Nout, R;        // R = row tiles per expert: I/128 (GEMM1), ceil(H/256) (GEMM2)
  float alpha, beta, limit;
};

// tile list entry of one work item and its row tile
struct Item {
  int row0, n, e, rt;
};

__device__ __forceinline__ void stmatrix_x2_trans(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("stmatrix.sync.aligned.m8n8.x2.trans.shared.b16 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c),
               "r"(d)
               : "memory");
}
// the other activation; its clamps let NaN through (src/flaggems_vllm/ops/fused_moe.py:733-773)
__device__ __forceinline__ float swigluoai(float g, float u, float alpha, float beta, float limit) {
  g = (g != g) ? g : fminf(g, limit);
  u = (u != u) ? u : fminf(fmaxf(u, -limit), limit);
  return g * (1.0f / (1.0f + expf(-alpha * g))) * (u + beta);
}

// SILU: the activation of GEMM1 (false: swigluoai, which reads GEMM1's result rounded to the activation type)
template <int FMT, typename AT, bool GEMM1, bool SILU>
__global__ void __launch_bounds__(THREADS, 1)
wt_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_b64,
               const __grid_constant__ CUtensorMap map_b16, const __grid_constant__ CUtensorMap map_b8, const Params P) {
  constexpr bool ROW = FMT == FMT_FP8ROW || FMT == FMT_I8ROW;
  constexpr int KIND = FMT == FMT_HALF ? MMA_F16 : (FMT == FMT_I8ROW ? MMA_I8 : MMA_F8);
  constexpr int KBE = FMT == FMT_HALF ? 64 : 128;  // elements of K per stage
  using C = Cfg<GEMM1>;
  constexpr int STAGES = C::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* s_out = smem + (size_t)STAGES * STAGE_BYTES;
  Aux* aux = reinterpret_cast<Aux*>(s_out + C::OUT_BYTES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KB = (P.K + KBE - 1) / KBE;
  const int cr = (int)cluster_ctarank();  // 0 leads
  const int item0 = blockIdx.x / 2, step = gridDim.x / 2;
  const int total = P.counts[0] * P.R;
  // Work items, expert by expert; inside an expert the token tile runs fastest, so the pairs that
  // run at the same time read the same weight tile.
  auto fetch = [&](int item) -> Item {
    Item it;
    const int t0 = item / P.R;
    int4 d = P.tiles[t0];
    const int first = d.w & 0xFFFF, q = (int)((uint32_t)d.w >> 16);
    const int within = item - first * P.R;
    it.rt = within / q;
    const int t = first + within - it.rt * q;
    if (t != t0) d = P.tiles[t];
    it.row0 = d.x; it.n = d.y & 0xFFFF; it.e = d.z;
    return it;
  };

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
      for (int item = item0; item < total && alive; item += step) {
        const Item it = nx;
        if (item + step < total) nx = fetch(item + step);
        const int nh = it.n >> 1;                 // this CTA's share of the token rows
        const int brow = it.row0 + cr * nh;
        const int wrow = GEMM1 ? it.rt * 16 + cr * 8 : it.e * P.Nout + it.rt * 256 + cr * 128;  // GEMM1: in groups of 8 outputs
        const uint32_t pair_bytes = 2 * (A_BYTES + (uint32_t)nh * 128);
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait(&aux->empty[s], ph ^ 1, P.status, P.wait_ns)) { alive = false; break; }
          if (leader) {
            if (cr == 0) mbar_expect_tx(&aux->full[s], pair_bytes);  // the peer's bytes may already have been counted
            uint8_t* sA = smem + (size_t)s * STAGE_BYTES;
            if constexpr (GEMM1) tma_load_5d_pair(&map_w, &aux->full[s], sA, kb * KBE, 0, 0, wrow, it.e);
            else tma_load_2d_pair(&map_w, &aux->full[s], sA, kb * KBE, wrow);
            uint8_t* sB = sA + A_BYTES;
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
      uint32_t s = 0, ph = 0, acc_it = 0;
      bool alive = true;
      Item nx = {};
      if (item0 < total) nx = fetch(item0);
      for (int item = item0; item < total && alive; item += step) {
        const Item it = nx;
        if (item + step < total) nx = fetch(item + step);
        const uint32_t idesc = idesc0 | ((uint32_t)(it.n >> 3) << 17);
        for (int kb = 0; kb < KB; ++kb) {
          const uint32_t a = acc_it & 1;
          if (!mbar_wait(&aux->full[s], ph, P.status, P.wait_ns)) { alive = false; break; }
          if (kb == 0) {
            if (!mbar_wait(&aux->tmem_empty[a], ((acc_it >> 1) & 1) ^ 1, P.status, P.wait_ns)) { alive = false; break; }
          }
          tc_fence_after();
          if (leader) {
            const uint64_t ad = a0 + (uint64_t)(s * (STAGE_BYTES >> 4)), bd = b0 + (uint64_t)(s * (STAGE_BYTES >> 4));
            const uint32_t d = tmem_base + a * NTOK;
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4)  // 32 bytes of K per instruction
              tc_mma_pair<KIND>(d, ad + (uint64_t)(k4 * 2), bd + (uint64_t)(k4 * 2), idesc,
                                (k4 > 0 || kb > 0) ? 1u : 0u);
            if (kb == KB - 1) tc_commit_pair(&aux->tmem_full[a]);
            tc_commit_pair(&aux->empty[s]);
          }
          if (kb == KB - 1) ++acc_it;
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    // -------------------------------------------------------------- consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CONSUMER_REGS));
    const int h = (warp - 4) >> 2, wq = warp & 3;
    const int tr = lane >> 2, tq = lane & 3;
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
    // rows of this thread: 16-lane block rh (0, 1) of the warp's 32 lanes, lanes tr and tr + 8
    // GEMM1: output 64 cr + 8 (2 wq + rh) + tr of the row tile (gate in lane tr, up in lane tr + 8)
    // GEMM2: output columns 128 cr + 32 wq + 16 rh + tr and + 8
    Item nx = {};
    if (item0 < total) nx = fetch(item0);
    // The tile loop runs to its end even after a wait has timed out: every consumer thread reaches
    // the named barriers of every tile.
    for (int item = item0; item < total; item += step) {
      const Item it = nx;
      if (item + step < total) nx = fetch(item + step);
      const int nh = it.n >> 1, tok0 = h * nh;      // this group's tokens [tok0, tok0 + nh) of the tile
      const int nst = (nh + 31) >> 5;               // steps of 32 tokens

      // (a) what is in the fragment registers r of step st, chunk c, block rh -> staged 16-bit values
      auto stage_chunk = [&](int st, int c, const float (&lo)[2][2], const float (&hi)[2][2]) {
        // lo[rh][j] / hi[rh][j]: lanes tr / tr + 8, token j of the pair (already final fp32 values)
        const int tok = tok0 + st * 32 + c * 8;
        if constexpr (GEMM1) {
          (void)hi;
          const uint32_t addr = out_base + (uint32_t)(tok + (lane & 7)) * C::OUT_PITCH + (uint32_t)((2 * wq + ((lane >> 3) & 1)) * 16);
          stmatrix_x2_trans(addr, pack2<AT>(lo[0][0], lo[0][1]), pack2<AT>(lo[1][0], lo[1][1]));
        } else {
          const uint32_t addr = out_base + (uint32_t)(tok + (lane & 7)) * C::OUT_PITCH + (uint32_t)(wq * 64 + (lane >> 3) * 16);
          stmatrix_x4_trans(addr, pack2<AT>(lo[0][0], lo[0][1]), pack2<AT>(hi[0][0], hi[0][1]), pack2<AT>(lo[1][0], lo[1][1]),
                            pack2<AT>(hi[1][0], hi[1][1]));
        }
      };
      // GEMM1: gate and up of (output, token) -> the staged activation value
      auto activate = [&](float g, float u, float rw) -> float {
        g *= rw; u *= rw;
        if constexpr (ROW || !SILU) { g = round_act<AT>(g); u = round_act<AT>(u); }
        if constexpr (SILU) return silu_mul_fast(g, u);
        else return swigluoai(g, u, P.alpha, P.beta, P.limit);
      };

      // ---------------------------------------------------------- tile epilogue
      asm volatile("bar.sync 2, %0;" ::"n"(CONS_THREADS) : "memory");  // the staging tile has been read
      {
        const uint32_t a = acc_it & 1;
        if (alive && !mbar_wait_idle(&aux->tmem_full[a], (acc_it >> 1) & 1, P.status, P.wait_ns)) alive = false;
        if (alive) {
          tc_fence_after();
          // channel scales of this thread's rows: [rh][lane tr / tr + 8]
          float cs[2][2] = {{1.0f, 1.0f}, {1.0f, 1.0f}};
          if constexpr (ROW) {
            const float* ws = P.w_scale + (int64_t)it.e * (GEMM1 ? 2 * P.Nout : P.Nout);
#pragma unroll
            for (int rh = 0; rh < 2; ++rh) {
              if constexpr (GEMM1) {
                const int o = it.rt * 128 + cr * 64 + (2 * wq + rh) * 8 + tr;
                cs[rh][0] = __ldg(ws + o);
                cs[rh][1] = __ldg(ws + P.Nout + o);
              } else {
                const int o = it.rt * 256 + cr * 128 + wq * 32 + rh * 16 + tr;
                cs[rh][0] = o < P.Nout ? __ldg(ws + o) : 0.0f;
                cs[rh][1] = o + 8 < P.Nout ? __ldg(ws + o + 8) : 0.0f;
              }
            }
          }
          const uint32_t t0 = t_lane + a * NTOK + (uint32_t)tok0;
#pragma unroll 1
          for (int st = 0; st < nst; ++st) {
            uint32_t r[32];
            tmem_ld_frag32_async(t0 + (uint32_t)st * 32, r);
            tmem_ld_frag32_async(t0 + (uint32_t)st * 32 + (16u << 16), r + 16);
            float2 as[4], rw[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const bool in = st * 32 + c * 8 < nh;
              const int64_t p = (int64_t)it.row0 + tok0 + st * 32 + c * 8 + 2 * tq;
              if constexpr (ROW) as[c] = in ? *reinterpret_cast<const float2*>(P.a_scales + p) : make_float2(0.0f, 0.0f);
              rw[c] = GEMM1 && in && P.row_weight != nullptr ? *reinterpret_cast<const float2*>(P.row_weight + p) : make_float2(1.0f, 1.0f);
            }
            tmem_wait32(r);
            if (st == nst - 1) release_acc(a);  // everything of this tile is in registers or staged
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              if (st * 32 + c * 8 < nh) {
                float lo[2][2], hi[2][2];
#pragma unroll
                for (int rh = 0; rh < 2; ++rh) {
                  float v[2][2];  // [lane tr / tr + 8][token]
#pragma unroll
                  for (int l = 0; l < 2; ++l)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                      const uint32_t raw = r[rh * 16 + 4 * c + 2 * l + j];
                      v[l][j] = FMT == FMT_I8ROW ? (float)(int)raw : __uint_as_float(raw);
                      if constexpr (ROW) v[l][j] = v[l][j] * (j == 0 ? as[c].x : as[c].y) * cs[rh][l];
                    }
                  if constexpr (GEMM1) {
                    lo[rh][0] = activate(v[0][0], v[1][0], rw[c].x);
                    lo[rh][1] = activate(v[0][1], v[1][1], rw[c].y);
                  } else {
                    lo[rh][0] = v[0][0]; lo[rh][1] = v[0][1];
                    hi[rh][0] = v[1][0]; hi[rh][1] = v[1][1];
                  }
                }
                stage_chunk(st, c, lo, hi);
              }
            }
          }
          ++acc_it;
        }
      }
      asm volatile("bar.sync 2, %0;" ::"n"(CONS_THREADS) : "memory");  // the tile is staged

      if constexpr (GEMM1) {
        const int sub = et & 7, tl = et >> 3;  // eight lanes per token: 16 bytes each
        const int64_t col = (int64_t)it.rt * 128 + cr * 64 + sub * 8;
        if (alive) {
          for (int tok = tl; tok < it.n; tok += 32)
            *reinterpret_cast<uint4*>(reinterpret_cast<AT*>(P.out) + ((int64_t)it.row0 + tok) * P.Nout + col) =
                *reinterpret_cast<const uint4*>(s_out + (size_t)tok * C::OUT_PITCH + sub * 16);
        }
      } else if (alive) {
        const int sub = et & 15;  // sixteen lanes per token
        const int col = it.rt * 256 + cr * 128 + sub * 8;
        if (col < P.Nout) {
          for (int tok = et >> 4; tok < it.n; tok += 16)
            *reinterpret_cast<uint4*>(reinterpret_cast<AT*>(P.out) + ((int64_t)it.row0 + tok) * P.Nout + col) =
                *reinterpret_cast<const uint4*>(s_out + (size_t)tok * C::OUT_PITCH + sub * 16);
        }
      }
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
template <int FMT, typename AT, bool GEMM1, bool SILU = true>
static int launch(const CUtensorMap& mw, const CUtensorMap (&mb)[3], const Params& P, int grid, cudaStream_t st) {
  auto kern = wt_gemm_kernel<FMT, AT, GEMM1, SILU>;
  constexpr size_t smem = smem_bytes<GEMM1>();
  static const int regs = [&] {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, kern) == cudaSuccess ? fa.numRegs : 0;
  }();
  // refuse to launch rather than let setmaxnreg.inc wait for registers that do not exist
  if (128 * PRODUCER_REGS + CONS_THREADS * CONSUMER_REGS > THREADS * regs)
    return fail(MOE_E_DRIVER, "grouped GEMM: kernel was built with %d registers per thread, %d needed", regs, LAUNCH_REGS);
  const int rc = allow_smem((const void*)kern, (int)smem);
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t ce = cudaLaunchKernelEx(&cfg, kern, mw, mb[0], mb[1], mb[2], P);
  if (ce != cudaSuccess) return fail((int)ce, "grouped GEMM launch: %s", cudaGetErrorString(ce));
  return check_launch(GEMM1 ? "gemm1 (pair, weights as M)" : "gemm2 (pair, weights as M)");
}

}  // namespace wt

bool wt_serves(int mode, int act_dtype, int H, int I) {
  if (act_dtype != MOE_BF16 && act_dtype != MOE_F16) return false;
  if (mode == MOE_MODE_HALF) return H % 64 == 0 && I % 128 == 0;
  return (mode == MOE_MODE_FP8_ROW || mode == MOE_MODE_INT8_ROW) && H % 128 == 0 && I % 128 == 0;
}

// a: [rows_cap, K] operand rows in the order of the route plan
int wt_gemm(bool gemm1, int mode, int act_dtype, const void* a, const float* a_scales, const void* w, const float* w_scale,
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
  if (gemm1 && act_kind != MOE_ACT_SILU) {
#define MOE_WT(F) \
  (act_dtype == MOE_BF16 ? launch<F, __nv_bfloat16, true, false>(mw, mb, P, grid, st) : launch<F, __half, true, false>(mw, mb, P, grid, st))
    switch (mode) {
      case MOE_MODE_HALF: return MOE_WT(FMT_HALF);
      case MOE_MODE_FP8_ROW: return MOE_WT(FMT_FP8ROW);
      case MOE_MODE_INT8_ROW: return MOE_WT(FMT_I8ROW);
      default: return fail(MOE_E_BADARG, "grouped GEMM: mode %d", mode);
    }
#undef MOE_WT
  }
#define MOE_WT(F)                                                                                               \
  (act_dtype == MOE_BF16 ? (gemm1 ? launch<F, __nv_bfloat16, true>(mw, mb, P, grid, st)                         \
                                  : launch<F, __nv_bfloat16, false>(mw, mb, P, grid, st))                       \
                         : (gemm1 ? launch<F, __half, true>(mw, mb, P, grid, st) : launch<F, __half, false>(mw, mb, P, grid, st)))
  switch (mode) {
    case MOE_MODE_HALF: return MOE_WT(FMT_HALF);
    case MOE_MODE_FP8_ROW: return MOE_WT(FMT_FP8ROW);
    case MOE_MODE_INT8_ROW: return MOE_WT(FMT_I8ROW);
    default: return fail(MOE_E_BADARG, "grouped GEMM: mode %d", mode);
  }
#undef MOE_WT
}

}  // namespace moe
