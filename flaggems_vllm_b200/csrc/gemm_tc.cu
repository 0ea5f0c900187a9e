// Expert grouped GEMMs on the 5th-generation tensor cores (tcgen05 / TMEM),
// fed by TMA.  One persistent CTA per SM walks a static list of
// (align block, column tile) pairs.
//
// Tile: 128 expert-sorted rows x 256 accumulator columns, K consumed 128 bytes
// per pipeline stage (128 e4m3 or 64 half elements = one 128-byte swizzle row).
//   A stage : 128 rows x 128 B.  GEMM2 reads its (already expert-sorted) input
//             with one TMA box.  GEMM1 gathers token rows: row p of the tile is
//             token sorted_ids[p] / topk, copied by 64 producer threads with
//             16-byte cp.async into the same 128-byte-swizzled layout TMA
//             would produce, so no sorted copy of the activations ever exists.
//             Two lanes share a row, so every 32-byte sector is requested once.
//   B stage : 256 rows x 128 B
// GEMM1 fetches it as two TMA boxes, 128 gate rows and the 128 up rows of the same
// 128 outputs, so one accumulator holds gate (columns 0-127) and up (128-255) of
// an output column in the same thread and SiLU(gate)*up plus the 1x128
// re-quantisation are done in registers.  GEMM2 fetches one box of 256 rows.
//
// Warp roles (384 threads):
//   warp 0      TMA producer (one lane)
//   warp 1      MMA issuer (one lane): tcgen05.mma, tcgen05.commit
//   warp 2      TMEM allocation (512 columns = two 256-column accumulators)
//   warps 2-3   GEMM1 only: cp.async gather of the A rows (2 rows per thread)
//   warps 4-11  accumulator consumers, two groups of four warps; group h owns
//               accumulator columns [128h, 128h+128) (GEMM1: gate [64h, 64h+64) and
//               up [128+64h, 128+64h+64)), warp w lanes 32*(w%4)...
// FP8 block-scaled mode: the tensor core cannot apply fp32 128x128 / 1x128
// scales, so every 128-wide K block is multiplied into a fresh TMEM
// accumulator (the two accumulators alternate) and the consumer warps fold it
// into fp32 registers with acc += part * (a_scale[row] * w_scale[block]), the
// arithmetic of the reference kernel (src/flaggems_vllm/ops/fused_moe.py:1708-1722),
// while the tensor core works on the next block.  The fold keeps two
// tcgen05.ld in flight and hands the accumulator
// back to the tensor core before its last FMAs.  The scales of the K blocks
// in flight sit in a small shared-memory ring filled by the producer side, so
// the consumers issue no global loads inside the K loop.
// Bound (FP8, 2048 rows per expert, cycles per K block, tile boundaries included): GEMM1 the fold's chain, 701 (620 without
// the fold, whatever the number of MMAs or commits: the operand stream); GEMM2, 16 K blocks per tile, the chain and the tile
// boundary, 836.  The chain is a consumer warp's instructions and their latencies, not the MMAs (the same with one of
// the four) nor the loads (the same with none); before barriers, slots and descriptors were carried in registers it was
// 811 and 900.  The clock those cycles run at is what power leaves: 1.4 GHz with 32 experts, 0.9 to 1.2 with 256, whose
// weights come out of HBM; there time follows energy and 14 % fewer cycles are 3 to 8 % of the time.
// Half mode: the whole K loop accumulates in TMEM; the two accumulators let
// the epilogue of one tile overlap the main loop of the next.
//
// Every barrier wait is bounded (wall-clock limit); on expiry the kernel sets
// MOE_ST_WAIT_TIMEOUT, leaves its loops, frees TMEM and returns.
#include <algorithm>

#include "tc_common.cuh"

namespace moe {
namespace tc {

constexpr int BM = 128;
constexpr int BN = 256;
// operand formats: half precision; e4m3 with 1x128 / 128x128 block scales (folded per K block);
// e4m3 or int8 with one scale per row and per output channel (applied to the finished sums)
constexpr int FMT_HALF = 0, FMT_FP8 = 1, FMT_FP8ROW = 2, FMT_I8ROW = 3;
constexpr int A_STAGE_BYTES = BM * 128;
constexpr int B_STAGE_BYTES = BN * 128;       // whole B tile (single-CTA kernel)
constexpr int B_HALF_BYTES = B_STAGE_BYTES / 2;  // what each CTA of a pair holds
constexpr int MAX_STAGES = 6;
// single CTA: 4 stages of A + B; CTA pair (cta_group::2): 6 stages of A + half of B;
// wide tile (RB = 2, half precision only): 3 stages of two A blocks + B, i.e. a 256x256
// output tile whose two accumulators fill TMEM, each B tile fetched once per 256 rows;
// wide pair: 4 stages of two A blocks + half of B, a 512x256 tile per pair, each B tile
// fetched once per 512 rows and each CTA loading only half of it
template <bool PAIR, int RB> struct Cfg {
  static constexpr int STAGES = PAIR ? (RB == 2 ? 4 : 6) : (RB == 2 ? 3 : 4);
  static constexpr int A_LOCAL = RB * A_STAGE_BYTES;
  static constexpr int STAGE_BYTES = A_LOCAL + (PAIR ? B_HALF_BYTES : B_STAGE_BYTES);
};
constexpr int THREADS = 384;
constexpr int EPI_THREADS = 256;
constexpr int GATHER_THREADS = 64;  // warps 2-3 (GEMM1)
constexpr int SCALE_THREADS = 32;   // warp 3 (FP8 GEMM2): scale staging
constexpr int SCALE_SLOTS = 8;
// setmaxnreg only moves registers inside the allocation the CTA got at launch
// (THREADS x the per-thread count ptxas reports under __launch_bounds__, 168).
// The consumers' increase must be covered by what the producer group gives
// up, otherwise setmaxnreg.inc waits forever.
constexpr int LAUNCH_REGS = 168;
constexpr int PRODUCER_REGS = 56;
constexpr int CONSUMER_REGS = 224;
static_assert((THREADS - EPI_THREADS) * PRODUCER_REGS + EPI_THREADS * CONSUMER_REGS <= THREADS * LAUNCH_REGS,
              "register redistribution exceeds the CTA's allocation");
static_assert(THREADS * LAUNCH_REGS <= 65536, "CTA does not fit the register file");

struct SmemAux {
  uint64_t full[MAX_STAGES];       // this CTA's operands (and scales) of the stage have landed
  uint64_t empty[MAX_STAGES];      // the tensor core has finished reading the stage
  uint64_t peer_full[MAX_STAGES];  // pair leader only: the partner CTA's stage has landed
  alignas(16) uint64_t tmem_full[2];  // the FP8 loops toggle between the two by address bit 3, and find tmem_empty 16 bytes on
  uint64_t tmem_empty[2];
  uint64_t xch_bar;
  uint32_t tmem_base;
  uint32_t pad;
  float xch[2][2][BM];  // [tile parity][consumer group][row] amax exchange
  // FP8: scales of the K blocks in flight, written by the producer-side threads
  // with cp.async and read by the consumers.  The ring is deeper than
  // STAGES + the two accumulators, so a slot is never rewritten before the
  // consumers have read it.
  struct Slot {
    float a[BM];  // activation scale of each tile row
    float w[4];   // weight scales of the two column halves
  } sc[SCALE_SLOTS];
};
static_assert(offsetof(SmemAux, tmem_full) % 16 == 0 && offsetof(SmemAux, tmem_empty) == offsetof(SmemAux, tmem_full) + 16, "barrier addresses");
constexpr int OUT_STAGE_BYTES = BM * BN * 2;  // staged output tile of the TMAOUT variant
template <bool PAIR, int RB, bool TMAOUT = false> constexpr size_t smem_bytes() {
  return TMAOUT ? (size_t)3 * Cfg<PAIR, RB>::STAGE_BYTES + sizeof(SmemAux) + 1024 + OUT_STAGE_BYTES + 1024
                : (size_t)Cfg<PAIR, RB>::STAGES * Cfg<PAIR, RB>::STAGE_BYTES + sizeof(SmemAux) + 1024;
}

struct Params {
  const uint8_t* a_rows;    // GEMM1: activations [tokens, K] in token order (gathered by cp.async)
  const float* a_scales_t;  // [K/128, a_scale_ld]        (FP8)
  const float* w_scale;     // FP8: [E, rows_w/128, K/128]; half mode: optional per-row scale [E, rows_w]
  const int4* tiles;        // route plan (plan.cu): one entry {row0, rows | occupied rows << 16, expert, -} per 128-row block;
                            // null: the blocks are described by expert_ids and sorted_ids
  const int32_t* expert_ids;
  const int32_t* sorted_ids;
  const int32_t* num_post_pad;
  const float* route_weight;
  void* out;
  float* out_scales_t;      // [I/128, rows_cap]          (FP8 GEMM1)
  int32_t* inv;             // TMAOUT: [numel] sorted row of every route
  int32_t* status;
  unsigned long long wait_ns;  // limit of every bounded barrier wait
  int64_t numel;
  int64_t rows_cap;
  int64_t a_scale_ld;       // tokens (GEMM1) or rows_cap (GEMM2)
  int topk;
  int mul_weight;
  int E;
  int K;        // contraction length in elements
  int Nout;     // output columns (I for GEMM1, H for GEMM2)
  int rows_w;   // weight rows per expert (2I or H)
  int n_tiles;  // column tiles per align block
  int group_m;  // align blocks per group of the tile order; BY_EXPERT: most blocks of an expert in a group
  int w_row0;   // GEMM2 over a window of the output columns: first weight row (output column) of the window
  bool wide_store;  // the output is 32-byte aligned: rows are written with 32-byte stores
};

// Instruction descriptor: fp32 accumulator (bits 4-5 = 1), A/B element format
// (bits 7-9 / 10-12: e4m3 = 0 for kind::f8f6f4; f16 = 0, bf16 = 1 for
// kind::f16), both operands K-major, N >> 3 at bit 17, M >> 4 at bit 24.
// Int8 operands (kind::i8): int32 accumulator (2), signed 8-bit elements (1).
template <int FMT, typename AT, bool PAIR>
struct IDesc {
  static constexpr uint32_t fmt = (FMT == FMT_I8ROW || (FMT == FMT_HALF && std::is_same<AT, __nv_bfloat16>::value)) ? 1u : 0u;
  static constexpr uint32_t m = PAIR ? 2 * BM : BM;  // a pair multiplies 256 rows per instruction
  static constexpr uint32_t value =
      ((FMT == FMT_I8ROW ? 2u : 1u) << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
};

// B tile = 256 accumulator columns = 256 weight rows, fetched with as few TMA instructions
// as the weight layout allows (every instruction costs the single producer thread issue
// time, whatever the box size).  GEMM1: columns [0,128) are gate rows nt*128.., columns
// [128,256) the up rows of the same outputs: two boxes of 128 rows (a CTA pair: one each).
// GEMM2: 256 consecutive rows, one box (a pair: 128 rows each).
template <bool GEMM1, bool PAIR> struct BBox {
  static constexpr int COUNT = (GEMM1 && !PAIR) ? 2 : 1;  // boxes per CTA and stage
  static constexpr int ROWS = (GEMM1 || PAIR) ? 128 : 256;
};
// weight row (inside the expert) of the first row of this CTA's box `c` of column tile `nt`
template <bool GEMM1, bool PAIR>
__device__ __forceinline__ int box_row(int nt, int c, int cr, int Nout) {
  if constexpr (GEMM1) return nt * 128 + (PAIR ? cr : c) * Nout;
  else return nt * BN + (PAIR ? cr * 128 : 0);
}

// PAIR = true: two CTAs of a cluster work as one cta_group::2 unit on a 256-row
// align block.  Each CTA holds its own 128 rows of A and ONE HALF of the B tile;
// the leader CTA (cluster rank 0) issues a single M=256 instruction per K step
// that reads both CTAs' shared memory and writes each CTA's own TMEM.  Every
// weight tile therefore crosses L2 -> shared memory once per 256 rows instead
// of once per 128.  Nothing is multicast: every TMA load and cp.async lands in
// the issuing CTA and signals a local barrier; the partner CTA forwards "stage
// landed" to the leader with a remote mbarrier arrive, and the leader's
// tcgen05.commit signals the stage-free / accumulator-ready barriers of both
// CTAs.
//
// RB = 2 (half precision, single CTA): the tile is 256 rows x 256 columns; both TMEM
// accumulators belong to it (rows 0-127 and 128-255), so every B stage is used by two
// instruction groups and each weight tile crosses L2 -> shared memory once per 256 rows
// without any cross-CTA traffic.  FP8 cannot use it: its fp32 fold accumulators live in
// registers and two blocks would need the whole register file.
//
// SORTED (GEMM1, half precision): the token rows were copied into sorted order beforehand
// (moe_gather_rows), so A arrives as one TMA box per 128 rows like in GEMM2 and warps 2-3 idle.
// With many rows per expert the in-kernel cp.async gather is the limiter of GEMM1 (its
// per-lane requests keep the load/store unit busier than the tensor core: 1.07 against
// 1.37 PFLOP/s for the TMA-fed GEMM2 on the Mixtral shape), and the copy costs far less.
//
// TMAOUT (GEMM2, single CTA): the output tile is staged in shared memory (bf16 / f16, the layout
// a 128-byte-swizzled tensor map expects) and written by TMA bulk stores to y in SORTED row
// order; the kernel also records where every route's row went (P.inv[route] = sorted row) for
// the combine.  A thread owns one tile row, so direct stores hand the memory system 32
// separate 32-byte sectors per warp instruction, and the consumers -- the same warps that fold
// the next tile -- sat in those stores for ~5000 cycles per tile; staged, they are done after
// sixteen conflict-free shared-memory stores.  Costs one pipeline stage of shared memory.
//
// PLAN: 0 the blocks of moe_align_block_size; over a route plan made with 128-row tiles (FP8) 1 the occupied rows, 2 whole blocks.
// BY_EXPERT (2): the blocks of an expert, which the plan knows, share its column tiles in the tile order.
// Fixed groups of blocks start somewhere inside an expert and read its weights once per group: DSV3 FP8, 8192 tokens, the
// layer 4799 -> 4719 us.  With few rows per expert the order is the same and the plan entries cost up to 1 %.  At most `group_m`
// blocks make a pass over the column tiles together: their rows are read again for every column tile and have to stay in L2.
//
// Row-scaled formats (FMT_FP8ROW, FMT_I8ROW): one-byte operands like the block-scaled mode, but
// nothing has to happen between K blocks, so the whole K loop accumulates in TMEM like half
// precision (int8: exact int32 sums) and the epilogue multiplies by the row's and the channel's
// scale.  Qwen3 shape, 500 tokens, e4m3: 5605 us for the two GEMMs on CUDA cores before.
template <int FMT, typename AT, bool GEMM1, bool PAIR, int RB, bool SORTED = false, bool TMAOUT = false, int PLAN = 0>
__global__ void __launch_bounds__(THREADS, 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_out, const __grid_constant__ CUtensorMap map_a16,
               const __grid_constant__ CUtensorMap map_a8, const Params P) {
  constexpr bool FP8 = FMT == FMT_FP8, ROW = FMT == FMT_FP8ROW || FMT == FMT_I8ROW;
  constexpr bool BYTE = FMT != FMT_HALF;  // one-byte operands
  constexpr int KIND = FMT == FMT_HALF ? MMA_F16 : (FMT == FMT_I8ROW ? MMA_I8 : MMA_F8);
  static_assert(!ROW || (!PAIR && RB == 1 && !SORTED), "row-scaled formats: the single-CTA kernel");
  static_assert(!TMAOUT || (!GEMM1 && !PAIR && RB == 1), "staged output: single-CTA GEMM2 only");
  static_assert(!SORTED || GEMM1, "pre-sorted A rows: GEMM1 only");
  constexpr bool BY_EXPERT = PLAN == 2;
  static_assert(PLAN == 0 || (FP8 && !PAIR && RB == 1 && (!GEMM1 || SORTED)), "route plan: the single-CTA FP8 kernels over sorted rows");
  static_assert(!BY_EXPERT || GEMM1 || TMAOUT, "whole blocks go with staged stores");
  constexpr bool GATHER = GEMM1 && !SORTED;  // A rows gathered inside the kernel
  static_assert(RB == 1 || (RB == 2 && !BYTE), "wide tiles: half precision only");
  constexpr int STAGES = TMAOUT ? 3 : Cfg<PAIR, RB>::STAGES;
  constexpr int A_LOCAL_BYTES = Cfg<PAIR, RB>::A_LOCAL;
  constexpr int B_LOCAL_BYTES = PAIR ? B_HALF_BYTES : B_STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_1024(smem_raw);
  uint8_t* sA = smem;
  uint8_t* sB = smem + (size_t)STAGES * A_LOCAL_BYTES;
  SmemAux* aux = reinterpret_cast<SmemAux*>(smem + (size_t)STAGES * Cfg<PAIR, RB>::STAGE_BYTES);
  // staged output tile: four sub-tiles of 128 rows x 64 columns (128 bytes per row), 1024-byte aligned
  [[maybe_unused]] uint8_t* s_out = smem + (((size_t)STAGES * Cfg<PAIR, RB>::STAGE_BYTES + sizeof(SmemAux) + 1023) & ~(size_t)1023);

  const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // the compiler sees that `warp` is uniform
  constexpr int KBE = BYTE ? 128 : 64;  // elements of K per stage
  const int KB = (P.K + KBE - 1) / KBE;
  const int npp = min((int64_t)__ldcg(P.num_post_pad), P.rows_cap);
  // work unit: one CTA and a 128-row align block; a CTA pair and a 256-row block; or one
  // CTA and a 256-row block (RB = 2).  UNIT = 128-row blocks per align block.
  constexpr int UNIT = PAIR ? 2 * RB : RB;
  constexpr int CTAS = PAIR ? 2 : 1;
  const int cr = PAIR ? (int)cluster_ctarank() : 0;  // rank inside the pair; 0 leads
  const int tile0 = blockIdx.x / CTAS, tile_step = gridDim.x / CTAS;
  const int nblk = (npp + UNIT * BM - 1) / (UNIT * BM);
  const int total_tiles = nblk * P.n_tiles;
  // Tile order: groups of `group_m` consecutive align blocks; inside a group the block index runs
  // fastest, then the column tile.  The CTAs that run at the same time then work on the blocks of
  // one expert for the SAME few column tiles, so a weight tile is fetched from DRAM once and
  // served to the other row blocks from L2.  (Column tile fastest sends every row block of an
  // expert over the expert's whole weight matrix at a different time; a matrix larger than L2
  // is then read once per row block.)
  auto tile_blk_nt = [&](int tile, int& blk, int& nt) {
    const int per_group = P.group_m * P.n_tiles;
    const int grp = tile / per_group;
    const int first = grp * P.group_m;
    const int gsz = min(nblk - first, P.group_m);
    const int within = tile - grp * per_group;
    nt = within / gsz;
    blk = first + within - nt * gsz;
  };
  auto expert_of = [&](int blk) -> int { return PLAN != 0 ? __ldcg(&P.tiles[blk].z) : P.expert_ids[blk]; };
  // BY_EXPERT: plan entry of one of the blocks of the expert that the NEXT tile belongs to, loaded a whole tile before it is used
  [[maybe_unused]] int2 ahead = make_int2(-1, 1 << 16);  // {expert, first block | blocks << 16}
  [[maybe_unused]] auto look_ahead = [&](int tile) {
    if (tile < total_tiles) ahead = __ldcg(reinterpret_cast<const int2*>(P.tiles + tile / P.n_tiles) + 1);
  };
  // tile of the expert whose plan entry is `ahead`: its blocks in as few groups of up to group_m as hold them, of one size
  [[maybe_unused]] auto expert_tile = [&](int tile, int& blk, int& nt) {
    int first = ahead.y & 0xFFFF, blocks = (int)((uint32_t)ahead.y >> 16), within = tile - first * P.n_tiles;
    if (blocks > P.group_m) {
      const int parts = (blocks + P.group_m - 1) / P.group_m, size = (blocks + parts - 1) / parts;
      const int part = within / (size * P.n_tiles);
      first += part * size;
      within -= part * size * P.n_tiles;
      blocks = min(blocks - part * size, size);
    }
    nt = within / blocks;
    blk = first + within - nt * blocks;
  };
  // tile -> expert_ids index (blk), this CTA's 128-row block (mb), column tile (nt).  The expert of
  // the NEXT tile is fetched while the current one is worked on: a tile starts without waiting
  // for a global load (every role walks the same tile list with its own copy of e_next).
  int e_next = -1;
  if constexpr (BY_EXPERT) {
    look_ahead(tile0);
  } else if (tile0 < total_tiles) {
    int blk0, nt0;
    tile_blk_nt(tile0, blk0, nt0);
    e_next = expert_of(blk0);
  }
  auto coords = [&](int tile, int& blk, int& nt) -> int {
    if constexpr (BY_EXPERT) {
      const int e = ahead.x;
      expert_tile(tile, blk, nt);
      look_ahead(tile + tile_step);
      return e;
    } else {
      tile_blk_nt(tile, blk, nt);
      const int e = e_next;
      e_next = -1;
      if (tile + tile_step < total_tiles) {
        int blk2, nt2;
        tile_blk_nt(tile + tile_step, blk2, nt2);
        e_next = expert_of(blk2);
      }
      return e;
    }
  };
#define MOE_TILE_COORDS(tile)                             \
  int blk, nt;                                            \
  const int e = coords((tile), blk, nt);                  \
  [[maybe_unused]] const int mb = UNIT * blk + RB * cr;

  if constexpr (PLAN == 1) {
    // Occupied rows only: the other rows of a stage are multiplied all the same.  They start as zeros and stay zeros
    // until a larger tile comes by.  Without this: DSV3 FP8, 61 tokens 1005 -> 1103 us per layer, one of 8 ranks with 2000
    // tokens 319 -> 323.
    for (int i = threadIdx.x; i < STAGES * A_LOCAL_BYTES / 16; i += THREADS) reinterpret_cast<uint4*>(sA)[i] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&aux->full[s], GATHER ? 1 + GATHER_THREADS : (FP8 ? 1 + SCALE_THREADS : 1));
      mbar_init(&aux->empty[s], 1);
      mbar_init(&aux->peer_full[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&aux->tmem_full[a], 1);
      mbar_init(&aux->tmem_empty[a], CTAS * (EPI_THREADS / 32));  // a pair's leader also collects the partner's warps
    }
    mbar_init(&aux->xch_bar, EPI_THREADS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&aux->tmem_base)),
                   "r"(512));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&aux->tmem_base)),
                   "r"(512));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
  }
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();  // both CTAs' barriers exist before anyone signals across
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = aux->tmem_base;
  // launched with a programmatic dependency over a route plan only (tc_gemm_plan)
  if (warp != 0) {
    pdl_wait();
    pdl_trigger();
  }

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGS));
    if (warp == 0) {
      // ------------------------------------------------------------ TMA producer
      const bool leader = elect_lane();
      if constexpr (!GATHER) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
      uint32_t s = 0, ph = 1;  // stage, and the parity its "empty" barrier is waited for with
      bool alive = true;
      auto occupied_rows = [&]([[maybe_unused]] int blk) -> int {  // rows of A to fetch
        if constexpr (PLAN == 1) return ((__ldcg(&P.tiles[blk].y) >> 16) + 7) & ~7;
        else return RB * BM;
      };
      // the stage's byte count and its weight tile
      auto load_weights = [&](int kb, int s, int a_rows, int wrow0, int nt) {
        mbar_expect_tx(&aux->full[s], (GATHER ? 0u : (uint32_t)a_rows * 128) + B_LOCAL_BYTES);  // GATHER: A rows arrive by cp.async (warps 2-3)
#pragma unroll
        for (int c = 0; c < BBox<GEMM1, PAIR>::COUNT; ++c)
          tma_load_2d(&map_b, &aux->full[s], sB + (size_t)s * B_LOCAL_BYTES + c * (BBox<GEMM1, PAIR>::ROWS * 128),
                      kb * KBE, wrow0 + box_row<GEMM1, PAIR>(nt, c, cr, P.Nout));
      };
      // route plan: the weights of the first stages do not wait for the kernel in front
      int early = 0;
      if constexpr (PLAN != 0) {
        if (tile0 < total_tiles) {
          int blk, nt, e0;
          if constexpr (BY_EXPERT) {  // as coords(), which moves on
            expert_tile(tile0, blk, nt);
            e0 = ahead.x;
          } else {
            tile_blk_nt(tile0, blk, nt);
            e0 = e_next;
          }
          const int a_rows = occupied_rows(blk), wrow0 = e0 * P.rows_w + P.w_row0;
          for (; early < STAGES && early < KB; ++early)
            if (leader) load_weights(early, early, a_rows, wrow0, nt);
        }
      }
      pdl_wait();
      for (int tile = tile0; tile < total_tiles && alive; tile += tile_step) {
        MOE_TILE_COORDS(tile)
        if (e < 0 || e >= P.E) continue;
        [[maybe_unused]] const int row0 = mb * BM;
        const int wrow0 = e * P.rows_w + P.w_row0;
        [[maybe_unused]] const int a_rows = occupied_rows(blk);
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait_at(smem_u32(&aux->empty[s]), ph, P.status, P.wait_ns)) { alive = false; break; }
          if (leader) {
            if (early > 0) --early;
            else load_weights(kb, (int)s, a_rows, wrow0, nt);
            if constexpr (!GATHER) {
              uint8_t* dst = sA + (size_t)s * A_LOCAL_BYTES;
              if (a_rows < RB * BM) {  // route plan, few rows: the rest of the stage keeps stale bytes, its results are never stored
                int r = 0;
                for (; a_rows - r >= 16; r += 16) tma_load_2d(&map_a16, &aux->full[s], dst + r * 128, kb * KBE, row0 + r);
                if (r < a_rows) tma_load_2d(&map_a8, &aux->full[s], dst + r * 128, kb * KBE, row0 + r);
              } else {
#pragma unroll
                for (int j = 0; j < RB; ++j) tma_load_2d(&map_a, &aux->full[s], dst + j * A_STAGE_BYTES, kb * KBE, row0 + j * BM);
              }
            }
          }
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    } else if (FP8 && !PAIR && warp == 1) {
      // ------------------------------------------------------------ MMA issuer, FP8: a fresh accumulator per K block
      // Every barrier and descriptor is carried in a register: what stands between "accumulator released" and the MMAs is a
      // fence.  (A loop that computed them took 118 cycles from one K block's commits to its next wait.)
      constexpr uint32_t idesc = IDesc<FMT, AT, PAIR>::value;
      const bool leader = elect_lane();
      const uint64_t adesc0 = make_smem_desc(smem_u32(sA)), bdesc0 = make_smem_desc(smem_u32(sB));
      const uint32_t full0 = smem_u32(&aux->full[0]);
      constexpr uint32_t TO_EMPTY = (uint32_t)(offsetof(SmemAux, empty) - offsetof(SmemAux, full));
      uint32_t full = full0, sph = 0, acc_empty = smem_u32(&aux->tmem_empty[0]), aph = 1, d = tmem_base;
      uint64_t adesc = adesc0, bdesc = bdesc0;
      bool alive = true;
      for (int tile = tile0; tile < total_tiles && alive; tile += tile_step) {
        MOE_TILE_COORDS(tile)
        if (e < 0 || e >= P.E) continue;
#pragma unroll 1
        for (int left = KB; left > 0; --left) {
          if (!mbar_wait_at(full, sph, P.status, P.wait_ns) || !mbar_wait_at(acc_empty, aph, P.status, P.wait_ns)) { alive = false; break; }
          if constexpr (GATHER) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // cp.async writes -> tensor core reads
          tc_fence_after();
          tc_mma_block_f8(leader, d, adesc, bdesc, idesc, acc_empty - 16, full + TO_EMPTY);
          d ^= BN;
          acc_empty ^= 8;
          aph ^= ((acc_empty >> 3) & 1) ^ 1;
          full += 8;
          adesc += (uint64_t)(A_LOCAL_BYTES >> 4);
          bdesc += (uint64_t)(B_LOCAL_BYTES >> 4);
          if (full == full0 + 8 * STAGES) { full = full0; adesc = adesc0; bdesc = bdesc0; sph ^= 1; }
        }
      }
    } else if (warp == 1 && cr == 0) {
      // ------------------------------------------------------------ MMA issuer (pair: leader only)
      constexpr uint32_t idesc = IDesc<FMT, AT, PAIR>::value;
      [[maybe_unused]] uint32_t it = 0;
      uint32_t acc_it = 0;
      bool alive = true;
      if constexpr (!PAIR) {
        const bool leader = elect_lane();
        const uint64_t adesc0 = make_smem_desc(smem_u32(sA));
        const uint64_t bdesc0 = make_smem_desc(smem_u32(sB));
        uint32_t s = 0, sph = 0;
        for (int tile = tile0; tile < total_tiles && alive; tile += tile_step) {
          MOE_TILE_COORDS(tile)
          if (e < 0 || e >= P.E) continue;
          for (int kb = 0; kb < KB; ++kb) {
            const uint32_t a = RB == 2 ? 0u : (acc_it & 1);
            const uint32_t aph = RB == 2 ? (acc_it & 1) : ((acc_it >> 1) & 1);
            const uint64_t bdesc = bdesc0 + (uint64_t)(s * (uint32_t)(B_LOCAL_BYTES >> 4));
            const uint64_t adesc = adesc0 + (uint64_t)(s * (uint32_t)(A_LOCAL_BYTES >> 4));
            const uint32_t d0 = tmem_base + a * BN;
            if (!mbar_wait(&aux->full[s], sph, P.status, P.wait_ns)) { alive = false; break; }
            if constexpr (GATHER) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // cp.async writes -> tensor core reads
            if (kb == 0) {
              if (!mbar_wait(&aux->tmem_empty[a], aph ^ 1, P.status, P.wait_ns)) { alive = false; break; }
            }
            tc_fence_after();
            if (leader) {
#pragma unroll
            for (int j = 0; j < RB; ++j) {
              const uint64_t aj = adesc + (uint64_t)(j * (A_STAGE_BYTES >> 4));
              const uint32_t d = RB == 2 ? tmem_base + (uint32_t)j * BN : d0;
              tc_mma<KIND>(d, aj, bdesc, idesc, kb > 0);
#pragma unroll
              for (int k4 = 1; k4 < 4; ++k4)  // 32 bytes of K per instruction: start address advances by 32 B >> 4
                tc_mma_const<KIND, true>(d, aj + (uint64_t)(k4 * 2), bdesc + (uint64_t)(k4 * 2), idesc);
            }
            if (kb == KB - 1) tc_commit(&aux->tmem_full[a]);
            tc_commit(&aux->empty[s]);
            }
            if (kb == KB - 1) ++acc_it;
            if (++s == STAGES) { s = 0; sph ^= 1; }
          }
        }
      } else {
      const bool leader = elect_lane();
      for (int tile = tile0; tile < total_tiles && alive; tile += tile_step) {
        MOE_TILE_COORDS(tile)
        if (e < 0 || e >= P.E) continue;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          // accumulator barrier and phase: the two accumulators alternate (per K block in FP8
          // mode, per tile in half mode); a wide tile owns both and uses barrier 0
          const uint32_t a = RB == 2 ? 0u : (acc_it & 1);
          const uint32_t aph = RB == 2 ? (acc_it & 1) : ((acc_it >> 1) & 1);
          if (FP8 || kb == 0) {
            if (!mbar_wait<PAIR>(&aux->tmem_empty[a], aph ^ 1, P.status, P.wait_ns)) { alive = false; break; }
            tc_fence_after();
          }
          const int s = it % STAGES;
          if (!mbar_wait(&aux->full[s], (it / STAGES) & 1, P.status, P.wait_ns)) { alive = false; break; }
          if (!mbar_wait<true>(&aux->peer_full[s], (it / STAGES) & 1, P.status, P.wait_ns)) { alive = false; break; }
          if constexpr (GATHER) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // cp.async writes -> tensor core reads
          tc_fence_after();
          const uint64_t bdesc = make_smem_desc(smem_u32(sB + (size_t)s * B_LOCAL_BYTES));
          if (leader) {
#pragma unroll
          for (int j = 0; j < RB; ++j) {
            const uint64_t adesc = make_smem_desc(smem_u32(sA + (size_t)s * A_LOCAL_BYTES + j * A_STAGE_BYTES));
            const uint32_t d = tmem_base + (RB == 2 ? (uint32_t)j : a) * BN;
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4) {
              // 32 bytes of K per instruction: start address advances by 32 B >> 4
              const uint32_t accum = FP8 ? (k4 > 0) : (kb > 0 || k4 > 0);
              tc_mma_pair<KIND>(d, adesc + (uint64_t)(k4 * 2), bdesc + (uint64_t)(k4 * 2), idesc, accum);
            }
          }
          tc_commit_pair(&aux->empty[s]);
          if (FP8 || kb == KB - 1) tc_commit_pair(&aux->tmem_full[a]);
          }
          if (FP8 || kb == KB - 1) ++acc_it;
        }
      }
      }
    } else if (PAIR && warp == 1 && lane == 0 && cr == 1) {
      // ------------------------------------------------------------ partner CTA: tell the leader a stage has landed
      uint32_t it = 0;
      bool alive = true;
      for (int tile = tile0; tile < total_tiles && alive; tile += tile_step) {
        MOE_TILE_COORDS(tile)
        if (e < 0 || e >= P.E) continue;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(&aux->full[s], (it / STAGES) & 1, P.status, P.wait_ns)) { alive = false; break; }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          mbar_arrive_remote(&aux->peer_full[s], 0);
        }
      }
    } else if (GATHER && warp >= 2) {
      // ------------------------------------------------------------ A-row gather (cp.async)
      // Two lanes share a row: lane pair q copies the 32-byte sector {2c, 2c+1} of rows
      // q + 32 j in step c, so every warp instruction fetches 16 whole sectors (one lane per row
      // would touch 32 sectors per instruction and fetch every sector twice).
      const int g = threadIdx.x - 64;  // 0..63
      const int q = g >> 1, half = g & 1;
      const int64_t pitch = (int64_t)P.K * (BYTE ? 1 : 2);
      uint32_t it = 0;
      bool alive = true;
      for (int tile = tile0; tile < total_tiles && alive; tile += tile_step) {
        MOE_TILE_COORDS(tile)
        if (e < 0 || e >= P.E) continue;
        constexpr int RPT = 4 * RB;  // rows per lane pair
        const uint8_t* src[RPT];
        bool ok[RPT];
        // FP8: thread g also stages the activation scales of rows g and g + 64 and (g < 2) the
        // weight scale of the gate (g = 0: rows nt*128..) or up (g = 1: rows I + nt*128..) block
        [[maybe_unused]] const float* ws_src = nullptr;
        [[maybe_unused]] const float* as_src[2] = {nullptr, nullptr};
        auto row_token = [&](int r, bool& valid) -> int64_t {
          const int64_t p = (int64_t)mb * BM + r;
          const int64_t sid = p < P.rows_cap ? (int64_t)P.sorted_ids[p] : P.numel;
          valid = sid >= 0 && sid < P.numel;  // padding slot: the row keeps stale bytes, its results are never stored
          return valid ? sid / P.topk : 0;
        };
        if constexpr (FP8) {
          const int sblk_per_e = (P.rows_w + 127) / 128;
          ws_src = P.w_scale + ((int64_t)e * sblk_per_e + (g == 1 ? (P.Nout >> 7) + nt : nt)) * KB;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            bool valid;
            const int64_t tok = row_token(g + 64 * j, valid);
            if (valid) as_src[j] = P.a_scales_t + tok;
          }
        }
#pragma unroll
        for (int j = 0; j < RPT; ++j) {
          const int64_t tok = row_token(q + 32 * j, ok[j]);
          src[j] = P.a_rows + tok * pitch + half * 16;
        }
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(&aux->empty[s], ((it / STAGES) & 1) ^ 1, P.status, P.wait_ns)) { alive = false; break; }
          const uint32_t base = smem_u32(sA + (size_t)s * A_LOCAL_BYTES);
#pragma unroll
          for (int j = 0; j < RPT; ++j) {
            if (ok[j]) {
              const int r = q + 32 * j;  // row inside the (RB x 128)-row tile
              const uint8_t* sp = src[j] + (int64_t)kb * 128;
#pragma unroll
              for (int c = 0; c < 4; ++c)  // 128-byte swizzle: 16-byte chunk index XOR (row mod 8)
                cp_async16(base + (uint32_t)r * 128u + (uint32_t)(((2 * c + half) ^ (r & 7)) << 4), sp + c * 32);
            }
          }
          if constexpr (FP8) {
            const int slot = it % SCALE_SLOTS;
#pragma unroll
            for (int j = 0; j < 2; ++j)
              if (as_src[j] != nullptr) cp_async4(smem_u32(&aux->sc[slot].a[g + 64 * j]), as_src[j] + (int64_t)kb * P.a_scale_ld);
            if (g < 2) cp_async4(smem_u32(&aux->sc[slot].w[g]), ws_src + kb);
          }
          cp_async_arrive_noinc(&aux->full[s]);
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (FP8 && !GATHER && warp == 3) {
      // ------------------------------------------------------------ scale staging (FP8, A rows read by TMA)
      uint32_t it = 0;
      bool alive = true;
      const int sblk_per_e = (P.rows_w + 127) / 128;
      for (int tile = tile0; tile < total_tiles && alive; tile += tile_step) {
        MOE_TILE_COORDS(tile)
        if (e < 0 || e >= P.E) continue;
        const float* as_row = P.a_scales_t + (int64_t)mb * BM + 4 * lane;
        // GEMM2: the two 128-column weight blocks of the tile; GEMM1: the gate block and the up block
        const int wblk = GEMM1 ? (lane == 1 ? (P.Nout >> 7) + nt : nt)
                               : min((P.w_row0 >> 7) + 2 * nt + lane, sblk_per_e - 1);
        const float* ws_src = P.w_scale + ((int64_t)e * sblk_per_e + wblk) * KB;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(&aux->empty[s], ((it / STAGES) & 1) ^ 1, P.status, P.wait_ns)) { alive = false; break; }
          const int slot = it % SCALE_SLOTS;
          cp_async16(smem_u32(&aux->sc[slot].a[4 * lane]), as_row + (int64_t)kb * P.a_scale_ld);
          if (lane < 2) cp_async4(smem_u32(&aux->sc[slot].w[lane]), ws_src + kb);
          cp_async_arrive_noinc(&aux->full[s]);
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else {
    // -------------------------------------------------------------- consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CONSUMER_REGS));
    const int h = (warp - 4) >> 2;                  // column half owned by this group
    const int row = ((warp & 3) << 5) + lane;       // accumulator lane = tile row
    const uint32_t t_lane = tmem_base + ((uint32_t)((warp & 3) << 5) << 16) + (uint32_t)(h * (GEMM1 ? 64 : 128));
    constexpr uint32_t SECOND = GEMM1 ? 128 : 64;  // column distance of the group's second 64-column chunk
    [[maybe_unused]] uint32_t acc_it = 0, tile_it = 0;
    bool alive = true;
    // FP8: the accumulator, its barrier and phase, and the scale slot of the next K block
    [[maybe_unused]] uint32_t t_acc = t_lane, acc_full = smem_u32(&aux->tmem_full[0]), acc_ph = 0, slot_at = 0;
    [[maybe_unused]] const uint32_t row_at = smem_u32(aux) + 4 * (uint32_t)row, w_at = smem_u32(aux) + (GEMM1 ? 0u : 4u * (uint32_t)h);
    // releasing an accumulator: the pair's leader collects the arrivals of both CTAs
    auto release_acc = [&](uint32_t a) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR && cr == 1) mbar_arrive_remote(&aux->tmem_empty[a], 0);
        else mbar_arrive(&aux->tmem_empty[a]);
      }
    };
    // The consumers' own walk over the tile list.  Coordinates, expert and this thread's sorted id
    // of the NEXT tile are fetched inside the K loop of the current one (FP8: while the warp would
    // wait for the tensor core anyway), so a tile starts folding without integer divisions or a
    // dependent global load in front of it.
    int nx_blk = 0, nx_nt = 0, nx_e = -1;
    [[maybe_unused]] int nx_occupied = 0;
    [[maybe_unused]] int64_t nx_sid = P.numel;
    auto prefetch_tile = [&](int t) {
      nx_e = -1;
      nx_sid = P.numel;
      if (t < total_tiles) {
        tile_blk_nt(t, nx_blk, nx_nt);
        if constexpr (PLAN != 0) {  // rows leave in sorted order, weighted by the combine
          const int4 d = __ldcg(P.tiles + nx_blk);
          nx_occupied = d.y >> 16;
          nx_e = d.z;
        } else {
          const int64_t pn = (int64_t)(UNIT * nx_blk + RB * cr) * BM + row;
          nx_e = P.expert_ids[nx_blk];
          if (pn < P.rows_cap) nx_sid = (int64_t)P.sorted_ids[pn];
        }
      }
    };
    // Staged output: the warps meet twice per tile around the staging buffer, also a warp whose wait has timed out.
    [[maybe_unused]] auto meet = [&] { asm volatile("bar.sync 2, %0;" ::"n"(EPI_THREADS) : "memory"); };
    if constexpr (!BY_EXPERT) prefetch_tile(tile0);
    for (int tile = tile0; tile < total_tiles && (alive || TMAOUT); tile += tile_step) {
      int blk = nx_blk, nt = nx_nt, e = nx_e;
      [[maybe_unused]] int occupied = nx_occupied;
      if constexpr (BY_EXPERT) {
        e = coords(tile, blk, nt);
        occupied = __ldcg(&P.tiles[blk].y) >> 16;  // first looked at behind the K loop
      }
      [[maybe_unused]] const int64_t sid_first = nx_sid;
      [[maybe_unused]] const int mb = UNIT * blk + RB * cr;
      if constexpr (!BY_EXPERT) {
        if (!FP8 || e < 0 || e >= P.E) prefetch_tile(tile + tile_step);  // half precision has no K loop here
      }
      if (e < 0 || e >= P.E) continue;
      if constexpr (TMAOUT) {
        if (!alive) {
          if constexpr (FP8 && !BY_EXPERT) prefetch_tile(tile + tile_step);
          meet();
          meet();
          continue;
        }
      }
      for (int sub = 0; sub < RB && alive; ++sub) {  // the 128-row blocks of this tile (two for wide tiles)
      const int64_t p = (int64_t)(mb + sub) * BM + row;
      int64_t sid = P.numel;
      if (PLAN != 0) sid = p;
      else if (sub == 0) sid = sid_first;
      else if (p < P.rows_cap) sid = (int64_t)P.sorted_ids[p];
      const bool row_ok = PLAN != 0 ? row < occupied : sid >= 0 && sid < P.numel;
      if (PLAN == 0 && (sid < 0 || sid > P.numel)) set_status(P.status, MOE_ST_BAD_ROW);  // the pad value is numel; anything else outside is corrupt
      float acc[128];
      [[maybe_unused]] float as = 0.0f;  // row-scaled formats: activation scale of this row
      float rw = 1.0f;  // route weight of this row, fetched early: the epilogue must not wait for it
      if constexpr (FP8) {
#pragma unroll
        for (int i = 0; i < 128; ++i) acc[i] = 0.0f;
        // Each K block: wait for its accumulator, fold it into acc, release it.  The accumulator is held from the first load
        // to the release, and the tensor core's next K block into it waits for that.  The second half is therefore reloaded into
        // each 32-register staging set as soon as its FMAs have consumed it, under the FMAs of the other set, and the FMAs of
        // the second half run after the release; the probe for the next accumulator is in flight under them.  Packed pair
        // FMAs: the fold's issue slots are what the MMA-issuing thread on the same scheduler competes with.
        // Two warps per scheduler do not hide each other's latencies (both wait for the same barrier), so what is not an
        // FMA counts: barrier, scale slot and accumulator are addresses carried in registers and toggled, the release is
        // predicated and not branched around, nothing is asked per K block that can be asked per tile.  811 -> 701 cycles per K
        // block of GEMM1 (2048 rows per expert), of which the FMAs are 256.
        uint32_t ra[32], rb[32];
        unsigned long long* acc2 = reinterpret_cast<unsigned long long*>(acc);
        constexpr int SC = (int)offsetof(SmemAux, sc), SLOT = (int)sizeof(SmemAux::Slot);
        float sa, w_lo, w_hi;
        // scales from the shared-memory ring filled by the producer side: GEMM1 halves are (gate, up) -> w[0], w[1]; GEMM2 group
        // h owns one weight block
        auto next_scales = [&] {
          sa = lds_f32<SC>(row_at + slot_at);
          w_lo = lds_f32<SC + BM * 4>(w_at + slot_at);
          w_hi = GEMM1 ? lds_f32<SC + BM * 4 + 4>(w_at + slot_at) : w_lo;
          slot_at += SLOT;
          if (slot_at == SCALE_SLOTS * SLOT) slot_at = 0;
        };
        if constexpr (!BY_EXPERT) prefetch_tile(tile + tile_step);
        if (P.mul_weight && row_ok) rw = P.route_weight[sid];
        if (!warp_agrees(mbar_wait_at(acc_full, acc_ph, P.status, P.wait_ns))) {
          alive = false;
          if constexpr (TMAOUT) { meet(); meet(); }
          break;
        }
        __syncwarp();  // without it the compiler spills registers
        tc_fence_after();
        next_scales();
#pragma unroll 1
        for (int left = KB; left > 0; --left) {
          const unsigned long long lo2 = splat2(sa * w_lo), hi2 = GEMM1 ? splat2(sa * w_hi) : lo2;
          tmem_ld64_sync(t_acc, ra, rb);
#pragma unroll
          for (int i = 0; i < 16; ++i) fma2(acc2[i], ra[2 * i], ra[2 * i + 1], lo2);
          tmem_ld32_async(t_acc + SECOND, ra);
#pragma unroll
          for (int i = 0; i < 16; ++i) fma2(acc2[16 + i], rb[2 * i], rb[2 * i + 1], lo2);
          tmem_ld32_async(t_acc + SECOND + 32, rb);
          tmem_wait64(ra, rb);
          if constexpr (PAIR) {
            release_acc((acc_full >> 3) & 1);
          } else {
            tc_fence_before();
            __syncwarp();
            mbar_arrive_at<16>(acc_full, lane == 0);
          }
          t_acc ^= BN;
          acc_full ^= 8;
          acc_ph ^= ((acc_full >> 3) & 1) ^ 1;
          bool ready = true;
          if (left > 1) ready = mbar_try_at(acc_full, acc_ph);
#pragma unroll
          for (int i = 0; i < 16; ++i) fma2(acc2[32 + i], ra[2 * i], ra[2 * i + 1], hi2);
          if (left > 1) {
            if (!warp_agrees(ready)) {
              ready = mbar_wait_at(acc_full, acc_ph, P.status, P.wait_ns);
              if (!warp_agrees(ready)) { alive = false; break; }
            }
            tc_fence_after();
            next_scales();
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) fma2(acc2[48 + i], rb[2 * i], rb[2 * i + 1], hi2);
        }
        if (!alive) {
          if constexpr (TMAOUT) { meet(); meet(); }
          break;
        }
      } else {
        const uint32_t a = RB == 2 ? 0u : (acc_it & 1);
        const uint32_t aph = RB == 2 ? (acc_it & 1) : ((acc_it >> 1) & 1);
        if (P.mul_weight && row_ok) rw = P.route_weight[sid];
        if constexpr (ROW) {
          if (row_ok) as = GEMM1 ? P.a_scales_t[sid / P.topk] : P.a_scales_t[p];
        }
        if (sub == 0) {
          if (!warp_agrees(mbar_wait(&aux->tmem_full[a], aph, P.status, P.wait_ns))) {
            alive = false;
            if constexpr (TMAOUT) { meet(); meet(); }
            break;
          }
          tc_fence_after();
        }
        const uint32_t t0 = t_lane + (RB == 2 ? (uint32_t)sub : a) * BN;
        uint32_t* r = reinterpret_cast<uint32_t*>(acc);
        tmem_ld64_sync(t0, r, r + 32);
        tmem_ld64_sync(t0 + SECOND, r + 64, r + 96);
        if (sub == RB - 1) {  // everything of this tile is in registers (or already stored)
          release_acc(a);
          ++acc_it;
        }
      }

      // ---------------------------------------------------------- tile epilogue
      if constexpr (ROW) {
#pragma unroll
        for (int i = 0; i < 128; ++i) {
          if constexpr (FMT == FMT_I8ROW) acc[i] = (float)__float_as_int(acc[i]);
          acc[i] *= as;
        }
      }
      if constexpr (!FP8) {
        if (P.w_scale != nullptr) {
          // row-scaled formats, and weight-only int8: weights were widened exactly to the activation dtype, the
          // per-output-channel scale is applied here in fp32
          const float* cs = P.w_scale + (int64_t)e * P.rows_w;
          if constexpr (GEMM1) {
            const int n0 = nt * 128 + 64 * h;
#pragma unroll
            for (int j4 = 0; j4 < 16; ++j4) {
              const float4 sg = *reinterpret_cast<const float4*>(cs + n0 + 4 * j4);
              const float4 su = *reinterpret_cast<const float4*>(cs + P.Nout + n0 + 4 * j4);
              acc[4 * j4 + 0] *= sg.x; acc[4 * j4 + 1] *= sg.y; acc[4 * j4 + 2] *= sg.z; acc[4 * j4 + 3] *= sg.w;
              acc[64 + 4 * j4 + 0] *= su.x; acc[64 + 4 * j4 + 1] *= su.y;
              acc[64 + 4 * j4 + 2] *= su.z; acc[64 + 4 * j4 + 3] *= su.w;
            }
          } else {
            const int n0 = nt * BN + 128 * h;
#pragma unroll
            for (int j4 = 0; j4 < 32; ++j4) {
              if (n0 + 4 * j4 < P.Nout) {
                const float4 sc = *reinterpret_cast<const float4*>(cs + n0 + 4 * j4);
                acc[4 * j4 + 0] *= sc.x; acc[4 * j4 + 1] *= sc.y; acc[4 * j4 + 2] *= sc.z; acc[4 * j4 + 3] *= sc.w;
              }
            }
          }
        }
      }
      if constexpr (GEMM1) {
        // acc[0..63] gate, acc[64..127] up of output columns nt*128 + 64h + j
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          // row-scaled formats: GEMM 1's output is rounded to the activation dtype before the activation reads it
          if constexpr (ROW) acc[j] = round_act<AT>(silu_mul_fast(round_act<AT>(acc[j] * rw), round_act<AT>(acc[64 + j] * rw)));
          else acc[j] = round_act<AT>(silu_mul_fast(acc[j] * rw, acc[64 + j] * rw));
          amax = fmaxf(amax, fabsf(acc[j]));
        }
        const int64_t col0 = (int64_t)nt * 128 + 64 * h;
        if constexpr (FP8) {
          float* x = &aux->xch[tile_it & 1][0][0];
          x[h * BM + row] = amax;
          mbar_arrive(&aux->xch_bar);
          if (!warp_agrees(mbar_wait(&aux->xch_bar, tile_it & 1, P.status, P.wait_ns))) { alive = false; break; }
          amax = fmaxf(amax, x[(1 - h) * BM + row]);
          const float s = fmaxf(amax, kQuantEps) * (1.0f / kFp8Max);
          const float inv_s = 1.0f / s;  // one reciprocal per row instead of 64 divisions
          if (row_ok || BY_EXPERT) {  // zero rows stay zero for GEMM2
            uint4 pieces[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint32_t w[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                uint32_t pk = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                  const float qv = fminf(fmaxf(acc[v * 16 + q * 4 + b] * inv_s, -kFp8Max), kFp8Max);
                  pk |= (uint32_t)f32_to_fp8e4m3(qv) << (8 * b);
                }
                w[q] = pk;
              }
              pieces[v] = make_uint4(w[0], w[1], w[2], w[3]);
            }
            store_row_pieces(reinterpret_cast<uint8_t*>(P.out) + p * P.Nout + col0, pieces, P.wide_store);
            if (h == 0) P.out_scales_t[(int64_t)nt * P.rows_cap + p] = s;
          }
        } else if (row_ok) {
          uint4 pieces[8];
#pragma unroll
          for (int v = 0; v < 8; ++v)
            pieces[v] = make_uint4(pack2<AT>(acc[v * 8 + 0], acc[v * 8 + 1]), pack2<AT>(acc[v * 8 + 2], acc[v * 8 + 3]),
                                   pack2<AT>(acc[v * 8 + 4], acc[v * 8 + 5]), pack2<AT>(acc[v * 8 + 6], acc[v * 8 + 7]));
          store_row_pieces(reinterpret_cast<AT*>(P.out) + p * P.Nout + col0, pieces, P.wide_store);
        }
      } else if constexpr (TMAOUT) {
        // the previous tile's bulk stores have finished reading the staging buffer
        if (threadIdx.x == 128) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        meet();
#pragma unroll
        for (int c = 0; c < 16; ++c) {  // 16-byte chunk c of this thread's 128 columns -> sub-tile 2h + c/8, chunk c%8
          const uint4 piece = make_uint4(pack2<AT>(acc[c * 8 + 0] * rw, acc[c * 8 + 1] * rw),
                                         pack2<AT>(acc[c * 8 + 2] * rw, acc[c * 8 + 3] * rw),
                                         pack2<AT>(acc[c * 8 + 4] * rw, acc[c * 8 + 5] * rw),
                                         pack2<AT>(acc[c * 8 + 6] * rw, acc[c * 8 + 7] * rw));
          uint8_t* dst = s_out + (size_t)(2 * h + (c >> 3)) * (BM * 128) + row * 128 + (((c & 7) ^ (row & 7)) << 4);
          *reinterpret_cast<uint4*>(dst) = piece;
        }
        if (PLAN == 0 && row_ok && h == 0 && P.inv != nullptr) P.inv[sid] = (int32_t)p;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> TMA reads
        meet();
        if (threadIdx.x == 128) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            const int c0 = nt * BN + q4 * 64;
            if (c0 < P.Nout)
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
                           ::"l"(&map_out), "r"(c0), "r"((int)(mb * BM)), "r"(smem_u32(s_out + (size_t)q4 * (BM * 128)))
                           : "memory");
          }
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      } else if (row_ok) {
        const int col0 = nt * BN + 128 * h;
        AT* o = reinterpret_cast<AT*>(P.out) + sid * P.Nout + col0;
#pragma unroll
        for (int v = 0; v < 16; v += 2) {
          if (col0 + v * 8 < P.Nout) {  // Nout is a multiple of 64: the two pieces are in or out together
            uint4 pieces[2];
#pragma unroll
            for (int u = 0; u < 2; ++u)
              pieces[u] = make_uint4(pack2<AT>(acc[(v + u) * 8 + 0] * rw, acc[(v + u) * 8 + 1] * rw),
                                     pack2<AT>(acc[(v + u) * 8 + 2] * rw, acc[(v + u) * 8 + 3] * rw),
                                     pack2<AT>(acc[(v + u) * 8 + 4] * rw, acc[(v + u) * 8 + 5] * rw),
                                     pack2<AT>(acc[(v + u) * 8 + 6] * rw, acc[(v + u) * 8 + 7] * rw));
            store_row_pieces(o + v * 8, pieces, P.wide_store);
          }
        }
      }
      }  // sub
      ++tile_it;
    }
  }

  // -------------------------------------------------------------------- teardown
  if constexpr (TMAOUT) {
    if (threadIdx.x == 128) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // the last tile's stores are complete
  }
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();  // no CTA leaves while its partner may still signal its barriers
  else __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    if constexpr (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
  }
#undef MOE_TILE_COORDS
}

// ------------------------------------------------------------------ host side
template <int FMT, typename AT, bool GEMM1, bool PAIR, int RB, bool SORTED = false, bool TMAOUT = false, int PLAN = 0>
static int launch(const CUtensorMap& ma, const CUtensorMap& mb, const Params& P, int grid, cudaStream_t st,
                  const CUtensorMap* mo = nullptr, const CUtensorMap* ms = nullptr) {
  auto kern = tc_gemm_kernel<FMT, AT, GEMM1, PAIR, RB, SORTED, TMAOUT, PLAN>;
  constexpr size_t smem = smem_bytes<PAIR, RB, TMAOUT>();
  static const int regs = [&] {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, kern) == cudaSuccess ? fa.numRegs : 0;
  }();
  // see LAUNCH_REGS: refuse to launch rather than let setmaxnreg.inc wait for registers that do not exist
  if ((THREADS - EPI_THREADS) * PRODUCER_REGS + EPI_THREADS * CONSUMER_REGS > THREADS * regs)
    return fail(MOE_E_DRIVER, "tensor-core GEMM: kernel was built with %d registers per thread, %d needed", regs, LAUNCH_REGS);
  const int rc = allow_smem((const void*)kern, (int)smem);
  if (rc) return rc;
  const CUtensorMap &m_out = mo != nullptr ? *mo : ma, &m16 = ms != nullptr ? ms[0] : ma, &m8 = ms != nullptr ? ms[1] : ma;
  const char* what = GEMM1 ? "gemm1 (tcgen05)" : "gemm2 (tcgen05)";
  if (PLAN != 0) return launch_pdl(kern, dim3((unsigned)grid), THREADS, smem, 1, st, what, ma, mb, m_out, m16, m8, P);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = PAIR ? 2 : 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t ce = cudaLaunchKernelEx(&cfg, kern, ma, mb, m_out, m16, m8, P);
  if (ce != cudaSuccess) return fail((int)ce, "tensor-core GEMM launch: %s", cudaGetErrorString(ce));
  return check_launch(what);
}

}  // namespace tc

// gemm1: `a` holds [a_tokens, K] activations in token order (row p of a tile is token
// sorted_ids[p] / topk); gemm2: `a` holds [rows_cap, K] rows in sorted order.
int tc_gemm(bool gemm1, int mode, int act_dtype, const void* a, const float* a_scales_t, const void* w,
            const float* w_scale, const int32_t* expert_ids, const int32_t* sorted_ids, const int32_t* npp,
            const float* route_weight, int mul_weight, int64_t numel, int64_t rows_cap, int64_t a_tokens, int topk,
            int block_m, int E, int K, int Nout, void* out, float* out_scales_t, int32_t* status, cudaStream_t st,
            int variant, int a_sorted, int32_t* inv, int w_row0, int w_rows, int grid_limit) {
  // w_row0, w_rows (gemm2 with inv only; 0, 0 = the whole matrix): the call produces the Nout output
  //   columns that start at column w_row0 of a weight matrix with w_rows rows per expert, into an
  //   `out` that is Nout wide; grid_limit > 0 caps the number of CTAs (SMs left to other work)
  // inv (gemm2, variant 1): `out` is y in SORTED row order [rows_cap, Nout], written by TMA from a staged
  //   tile, and inv[route] receives the sorted row of every route
  // a_sorted (gemm1): `a` holds [rows_cap, K] rows already in sorted order (moe_gather_rows)
  // variant: 1 = one CTA per 128-row block, 2 = cta_group::2 CTA pair per 256-row block,
  //          3 = one CTA per 256-row block with a 256x256 tile (half precision only),
  //          4 = CTA pair per 512-row block, 256x256 per CTA (half precision only)
  using namespace tc;
  const bool pair = variant == 2 || variant == 4, wide = variant == 3 || variant == 4;
  if (variant < 1 || variant > 4) return fail(MOE_E_BADARG, "tensor-core GEMM: unknown kernel variant %d", variant);
  if (wide && mode != MOE_MODE_HALF) return fail(MOE_E_SHAPE, "tensor-core GEMM: the 256-row-per-CTA tiles serve half precision only");
  const bool fp8 = mode == MOE_MODE_FP8_BLOCK;
  const bool row = mode == MOE_MODE_FP8_ROW || mode == MOE_MODE_INT8_ROW, byte = fp8 || row;
  if (row && (variant != 1 || a_sorted || w_rows > 0))
    return fail(MOE_E_SHAPE, "tensor-core GEMM: the row-scaled modes run on kernel 1, whole matrices, unsorted rows");
  const bool sorted = gemm1 && a_sorted != 0;
  if (sorted && ((pair && !fp8) || (fp8 && wide)))
    return fail(MOE_E_SHAPE, "tensor-core GEMM1: pre-sorted rows are served by the single-CTA kernels and the FP8 CTA pair");
  if (!byte && mode != MOE_MODE_HALF)
    return fail(MOE_E_SHAPE, "tensor-core GEMM: mode %d is served by the generic kernel", mode);
  if (act_dtype != MOE_BF16 && act_dtype != MOE_F16)
    return fail(MOE_E_DTYPE, "tensor-core GEMM: activations must be f16 or bf16");
  const int unit_rows = BM * (pair ? 2 : 1) * (wide ? 2 : 1);
  if (block_m != unit_rows) return fail(MOE_E_SHAPE, "tensor-core GEMM: align block must be %d", unit_rows);
  if (rows_cap % unit_rows != 0 || rows_cap <= 0)
    return fail(MOE_E_SHAPE, "tensor-core GEMM: row capacity must be a positive multiple of %d", unit_rows);
  const int kbe = byte ? 128 : 64;
  if (K % kbe != 0) return fail(MOE_E_SHAPE, "tensor-core GEMM: K must be a multiple of %d", kbe);
  if (gemm1 && Nout % 128 != 0) return fail(MOE_E_SHAPE, "tensor-core GEMM1: intermediate size must be a multiple of 128");
  if (!gemm1 && Nout % 64 != 0) return fail(MOE_E_SHAPE, "tensor-core GEMM2: hidden size must be a multiple of 64");
  if (fp8 && !gemm1 && Nout % 128 != 0) return fail(MOE_E_SHAPE, "tensor-core GEMM2 (fp8): hidden size must be a multiple of 128");
  const bool window = w_rows > 0;
  if (window && mode == MOE_MODE_HALF && w_scale != nullptr)
    return fail(MOE_E_SHAPE, "tensor-core GEMM2: column windows do not serve per-channel scales");
  if (window && (gemm1 || inv == nullptr || w_row0 < 0 || w_row0 % 256 != 0 || Nout % 256 != 0 || w_row0 + Nout > w_rows))
    return fail(MOE_E_SHAPE, "tensor-core GEMM2: a column window starts and ends on multiples of 256 columns of the staged-output kernel");
  const int rows_w = gemm1 ? 2 * Nout : (window ? w_rows : Nout);
  if ((int64_t)E * rows_w >= (1ll << 31) || rows_cap >= (1ll << 31)) return fail(MOE_E_TOOBIG, "tensor-core GEMM: extent exceeds int32 coordinates");

  const int eb = byte ? 1 : 2;
  const CUtensorMapDataType dt = byte ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                     : (act_dtype == MOE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
  CUtensorMap ma, mb;
  int rc = 0;
  if (gemm1 && !sorted) {
    memset(&ma, 0, sizeof(ma));  // A rows are gathered with cp.async, no tensor map
    if (((uintptr_t)a & 15) != 0) return fail(MOE_E_BADARG, "tensor-core GEMM1: activations not 16-byte aligned");
    if (topk <= 0 || a_tokens * topk != numel) return fail(MOE_E_BADARG, "tensor-core GEMM1: tokens * topk != numel");
  } else {
    rc = make_map(&ma, a, dt, eb, (uint64_t)rows_cap, (uint64_t)K, BM, false);
    if (rc) return rc;
  }
  rc = make_map(&mb, w, dt, eb, (uint64_t)E * rows_w, (uint64_t)K, (gemm1 || pair) ? 128 : 256, true);
  if (rc) return rc;

  Params P;
  if (sorted && (topk <= 0 || a_tokens * topk != numel)) return fail(MOE_E_BADARG, "tensor-core GEMM1: tokens * topk != numel");
  P.tiles = nullptr;
  P.a_rows = (const uint8_t*)a; P.a_scale_ld = (gemm1 && !sorted) ? a_tokens : rows_cap; P.topk = gemm1 ? topk : 1;
  P.a_scales_t = a_scales_t; P.w_scale = w_scale; P.expert_ids = expert_ids; P.sorted_ids = sorted_ids;
  P.num_post_pad = npp; P.route_weight = route_weight; P.out = out; P.out_scales_t = out_scales_t; P.inv = nullptr;
  P.status = status; P.wait_ns = wait_limit_ns(); P.numel = numel; P.rows_cap = rows_cap; P.mul_weight = mul_weight; P.E = E; P.K = K;
  P.Nout = Nout; P.rows_w = rows_w; P.w_row0 = window ? w_row0 : 0;
  P.n_tiles = gemm1 ? Nout / 128 : (Nout + BN - 1) / BN;
  {
    // about as many blocks per group as one expert owns (rows per expert / rows per block, one of them partial)
    const int64_t per_expert = numel / (E > 0 ? E : 1);
    int64_t gm = per_expert / unit_rows + 1;
    P.group_m = (int)(gm < 1 ? 1 : (gm > 16 ? 16 : gm));
  }
  P.wide_store = ((uintptr_t)out & 31) == 0;

  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t cap_tiles = (rows_cap / unit_rows) * (int64_t)P.n_tiles;
  if (grid_limit > 0 && grid_limit < sms) sms = grid_limit;
  const int units = pair ? sms / 2 : sms;  // work units resident at once: CTAs, or CTA pairs
  const int grid = (int)(cap_tiles < units ? cap_tiles : units) * (pair ? 2 : 1);

#define MOE_TC_LAUNCH2(F, T, G) \
  (pair ? launch<F, T, G, true, 1>(ma, mb, P, grid, st) : launch<F, T, G, false, 1>(ma, mb, P, grid, st))
#define MOE_TC_LAUNCH(F, T) (gemm1 ? MOE_TC_LAUNCH2(F, T, true) : MOE_TC_LAUNCH2(F, T, false))
  if (inv != nullptr) {
    if (gemm1 || variant != 1) return fail(MOE_E_SHAPE, "tensor-core GEMM: sorted output is written by GEMM2 of kernel 1 only");
    CUtensorMap mo;
    rc = make_map(&mo, out, act_dtype == MOE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                  (uint64_t)rows_cap, (uint64_t)Nout, BM, false);
    if (rc) return rc;
    P.inv = inv;
    if (mode == MOE_MODE_FP8_ROW)
      return act_dtype == MOE_BF16 ? launch<FMT_FP8ROW, __nv_bfloat16, false, false, 1, false, true>(ma, mb, P, grid, st, &mo)
                                   : launch<FMT_FP8ROW, __half, false, false, 1, false, true>(ma, mb, P, grid, st, &mo);
    if (mode == MOE_MODE_INT8_ROW)
      return act_dtype == MOE_BF16 ? launch<FMT_I8ROW, __nv_bfloat16, false, false, 1, false, true>(ma, mb, P, grid, st, &mo)
                                   : launch<FMT_I8ROW, __half, false, false, 1, false, true>(ma, mb, P, grid, st, &mo);
    if (fp8)
      return act_dtype == MOE_BF16 ? launch<FMT_FP8, __nv_bfloat16, false, false, 1, false, true>(ma, mb, P, grid, st, &mo)
                                   : launch<FMT_FP8, __half, false, false, 1, false, true>(ma, mb, P, grid, st, &mo);
    return act_dtype == MOE_BF16 ? launch<FMT_HALF, __nv_bfloat16, false, false, 1, false, true>(ma, mb, P, grid, st, &mo)
                                 : launch<FMT_HALF, __half, false, false, 1, false, true>(ma, mb, P, grid, st, &mo);
  }
#define MOE_TC_ROW(F, T) (gemm1 ? launch<F, T, true, false, 1>(ma, mb, P, grid, st) : launch<F, T, false, false, 1>(ma, mb, P, grid, st))
  if (mode == MOE_MODE_FP8_ROW)
    return act_dtype == MOE_BF16 ? MOE_TC_ROW(FMT_FP8ROW, __nv_bfloat16) : MOE_TC_ROW(FMT_FP8ROW, __half);
  if (mode == MOE_MODE_INT8_ROW)
    return act_dtype == MOE_BF16 ? MOE_TC_ROW(FMT_I8ROW, __nv_bfloat16) : MOE_TC_ROW(FMT_I8ROW, __half);
#undef MOE_TC_ROW
  if (fp8 && sorted && pair)
    return act_dtype == MOE_BF16 ? launch<FMT_FP8, __nv_bfloat16, true, true, 1, true>(ma, mb, P, grid, st)
                                 : launch<FMT_FP8, __half, true, true, 1, true>(ma, mb, P, grid, st);
  if (fp8 && sorted)
    return act_dtype == MOE_BF16 ? launch<FMT_FP8, __nv_bfloat16, true, false, 1, true>(ma, mb, P, grid, st)
                                 : launch<FMT_FP8, __half, true, false, 1, true>(ma, mb, P, grid, st);
  if (fp8) return act_dtype == MOE_BF16 ? MOE_TC_LAUNCH(FMT_FP8, __nv_bfloat16) : MOE_TC_LAUNCH(FMT_FP8, __half);
  if (sorted) {
    if (act_dtype == MOE_BF16)
      return wide ? launch<FMT_HALF, __nv_bfloat16, true, false, 2, true>(ma, mb, P, grid, st)
                  : launch<FMT_HALF, __nv_bfloat16, true, false, 1, true>(ma, mb, P, grid, st);
    return wide ? launch<FMT_HALF, __half, true, false, 2, true>(ma, mb, P, grid, st)
                : launch<FMT_HALF, __half, true, false, 1, true>(ma, mb, P, grid, st);
  }
#define MOE_TC_WIDE(T, G) \
  (pair ? launch<FMT_HALF, T, G, true, 2>(ma, mb, P, grid, st) : launch<FMT_HALF, T, G, false, 2>(ma, mb, P, grid, st))
  if (wide) {
    if (act_dtype == MOE_BF16) return gemm1 ? MOE_TC_WIDE(__nv_bfloat16, true) : MOE_TC_WIDE(__nv_bfloat16, false);
    return gemm1 ? MOE_TC_WIDE(__half, true) : MOE_TC_WIDE(__half, false);
  }
#undef MOE_TC_WIDE
  return act_dtype == MOE_BF16 ? MOE_TC_LAUNCH(FMT_HALF, __nv_bfloat16) : MOE_TC_LAUNCH(FMT_HALF, __half);
#undef MOE_TC_LAUNCH
#undef MOE_TC_LAUNCH2
}

// The FP8 GEMMs over the blocks of a route plan made with 128-row tiles (plan.cu): A rows (GEMM1: scattered token
// rows, GEMM2: the intermediate) in sorted order, results in sorted order.  all_rows: the padding rows of A are zero,
// fetch whole blocks.
int tc_gemm_plan(bool gemm1, int act_dtype, const void* a, const float* a_scales_t, const void* w, const float* w_scale,
                 const void* tiles, const int32_t* rows, int64_t numel, int64_t rows_cap, int E, int K, int Nout, void* out,
                 float* out_scales_t, const float* row_weight, bool all_rows, bool staged, int32_t* status, cudaStream_t st) {
  using namespace tc;
  constexpr int eb = 1;
  const int rows_w = gemm1 ? 2 * Nout : Nout;
  if ((int64_t)E * rows_w >= (1ll << 31) || rows_cap >= (1ll << 31)) return fail(MOE_E_TOOBIG, "tensor-core GEMM: extent exceeds int32 coordinates");
  const CUtensorMapDataType half_t = act_dtype == MOE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_UINT8;
  CUtensorMap ma, mb, mo, ms[2];
  int rc = make_map(&ma, a, dt, eb, (uint64_t)rows_cap, (uint64_t)K, BM, false);
  if (!rc) rc = make_map(&ms[0], a, dt, eb, (uint64_t)rows_cap, (uint64_t)K, 16, false);
  if (!rc) rc = make_map(&ms[1], a, dt, eb, (uint64_t)rows_cap, (uint64_t)K, 8, false);
  if (!rc) rc = make_map(&mb, w, dt, eb, (uint64_t)E * rows_w, (uint64_t)K, gemm1 ? 128 : 256, true);
  if (!rc && staged) rc = make_map(&mo, out, half_t, 2, (uint64_t)rows_cap, (uint64_t)Nout, BM, false);
  if (rc) return rc;
  Params P = {};
  P.a_rows = (const uint8_t*)a; P.a_scale_ld = rows_cap; P.topk = 1;
  P.a_scales_t = a_scales_t; P.w_scale = w_scale; P.tiles = (const int4*)tiles;
  P.route_weight = row_weight; P.mul_weight = row_weight != nullptr;  // sorted order: row p's weight
  P.num_post_pad = rows; P.out = out; P.out_scales_t = out_scales_t; P.status = status; P.wait_ns = wait_limit_ns();
  P.numel = rows_cap; P.rows_cap = rows_cap; P.E = E; P.K = K; P.Nout = Nout; P.rows_w = rows_w;
  P.n_tiles = gemm1 ? Nout / 128 : (Nout + BN - 1) / BN;
  // Blocks that share a pass over the column tiles.  Whole blocks: 16 MB of rows (18 blocks at K = 7168, 64 at 2048).  K 7168,
  // I 2048, us per layer, groups of 16 across experts / 16 MB / 32 / 64 / an expert's blocks all together: 128 blocks per expert (4
  // experts) 3545 / 3297 / 3425 / 3537 / 3878, 96 blocks 2619 / 2475 / 2462 / 2560 / 2843, 64 blocks 1813 / 1660 / 1691 / 1699 / 1741;
  // 32 experts, half of the routes on four of them (128 blocks each) 6864 / 6388 / 6585 / 6639 / 6951.
  const int64_t gm = numel / E / BM + 1;
  P.group_m = all_rows ? std::max(16, (16 << 20) / (BM * K)) : (int)(gm > 16 ? 16 : gm);
  P.wide_store = ((uintptr_t)out & 31) == 0;
  const int64_t cap_tiles = (rows_cap / BM) * (int64_t)P.n_tiles;
  const int sms = sm_count();
  const int grid = (int)(cap_tiles < sms ? cap_tiles : sms);
  // whole blocks: from 128 rows per expert on (layer.cu), where an expert has several
  if (all_rows && !staged) return fail(MOE_E_SHAPE, "tensor-core GEMM over a route plan: whole blocks go with staged stores");
#define MOE_TCP(T)                                                                                                                \
  (gemm1 ? (all_rows ? launch<FMT_FP8, T, true, false, 1, true, false, 2>(ma, mb, P, grid, st, nullptr, ms)                        \
                     : launch<FMT_FP8, T, true, false, 1, true, false, 1>(ma, mb, P, grid, st, nullptr, ms))                       \
         : (all_rows ? launch<FMT_FP8, T, false, false, 1, false, true, 2>(ma, mb, P, grid, st, &mo, ms)                           \
            : staged ? launch<FMT_FP8, T, false, false, 1, false, true, 1>(ma, mb, P, grid, st, &mo, ms)                           \
                     : launch<FMT_FP8, T, false, false, 1, false, false, 1>(ma, mb, P, grid, st, nullptr, ms)))
  return act_dtype == MOE_BF16 ? MOE_TCP(__nv_bfloat16) : MOE_TCP(__half);
#undef MOE_TCP
}

}  // namespace moe
