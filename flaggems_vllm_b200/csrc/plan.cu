// Route plan of one layer call: where every route's row sits in expert-sorted order, and the list of token
// tiles that the grouped GEMMs walk.
//
// A stable counting sort of the expert ids like moe_align_block_size, with three differences that the
// layer wants: each expert's run is padded to `gran` rows (16, or 32) only, so that hardly any padding is multiplied
// (a tile of n rows costs n, see gemm_wt.cu); the result is the inverse map row_index[route] = sorted row
// (-1: id out of range or expert not local) that the scatter in front of GEMM 1 and the sum behind
// GEMM 2 read; and each run is cut into tiles of at most `tile_rows` rows, as even as multiples of gran allow.
// expert_map is applied here, so routes of other ranks' experts get no rows at all.
//
// The sort itself is sort_ids.cuh.
#include <climits>

#include "sort_ids.cuh"

namespace moe {
namespace {

template <typename IdT, int CTAS, int ROUNDS, int LANES>
__device__ __forceinline__ void plan_body(const IdT* __restrict__ ids, int numel, int E, const int32_t* __restrict__ emap,
                                          int E_local, int gran_shift, int tile_rows, int32_t* __restrict__ row_index, int rows_cap,
                                          int4* __restrict__ tiles, int tiles_cap, int32_t* __restrict__ counts,
                                          int32_t* __restrict__ status) {
  using namespace sorting;
  extern __shared__ __align__(16) int32_t sort_smem[];
  const Shared sh = carve<CTAS>(sort_smem, E_local);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int rank = 0;
  if constexpr (CTAS > 1) rank = (int)cg::this_cluster().block_rank();
  bool bad = false;
  int packed[ROUNDS], first, end;
  rank_ids<CTAS, ROUNDS, LANES>(numel, E_local, sh, [&](int i) -> int {
    const long long e = (long long)ids[i];
    if (e < 0 || e >= E) {
      if (e >= E) bad = true;  // negative ids mean "no route" (padding rows, other ranks' slots)
      return -1;
    }
    if (emap == nullptr) return (int)e;
    const int m = emap[(int)e];
    return m >= 0 && m < E_local ? m : -1;
  }, packed, first, end);
  if (bad) set_status(status, MOE_ST_BAD_EXPERT_ID);
  // rows of an expert in units of the granule, and the tiles they are cut into; both fit 16 bits (launch_plan)
  auto units_of = [&](int n) { return (n + (1 << gran_shift) - 1) >> gran_shift; };
  auto tiles_of = [&](int units) { return ((units << gran_shift) + tile_rows - 1) / tile_rows; };
  int before = 0, all = 0;
  unsigned mine = 0, sum;
  if (tid < E_local) {
    all = count_all<CTAS>(sh, tid, E_local, rank, before);
    const int units = units_of(all);
    mine = (unsigned)units | (unsigned)tiles_of(units) << 16;
  }
  const unsigned base = scan_cta(mine, sum);
  if (tid < E_local) {
    sh.base[tid] = (int)base;
    sh.count[tid] = all;
    sh.place[tid] = (int)((base & 0xFFFFu) << gran_shift) + before;
  }
  if (rank == 0 && tid == 0) {
    counts[0] = min((int)(sum >> 16), tiles_cap);
    counts[1] = min((int)((sum & 0xFFFFu) << gran_shift), rows_cap);
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int i = first + 32 * r + lane;
    if (packed[r] != kNone) {
      const int e = packed[r] & 0x7FF;
      row_index[i] = sh.place[e] + sh.hist[(size_t)warp * E_local + e] + (packed[r] >> 11);
    } else if (i < end) {
      row_index[i] = -1;
    }
  }
  // The tiles, an even split in multiples of the granule.  A warp per expert, which may have many; in one CTA (2048 ids at
  // most) the experts do not have enough tiles for that, and a warp would come to eight of them in turn: a thread each.
  constexpr bool BY_WARP = CTAS > 1;
  for (int e = BY_WARP ? rank * kWarps + warp : tid; e < E_local; e += BY_WARP ? CTAS * kWarps : kThreads) {
    const int n_all = sh.count[e];
    if (n_all == 0) continue;
    const unsigned at0 = (unsigned)sh.base[e];
    const int row0 = (int)((at0 & 0xFFFFu) << gran_shift), at = (int)(at0 >> 16), units = units_of(n_all), q = tiles_of(units);
    const int padded = units << gran_shift, size = ((units + q - 1) / q) << gran_shift;
    for (int t = BY_WARP ? lane : 0; t < q; t += BY_WARP ? 32 : 1) {
      const int r = min(padded, t * size), n = min(size, padded - r), occupied = max(0, min(n, n_all - r));
      if (at + t < tiles_cap) tiles[at + t] = make_int4(row0 + r, max(n, 0) | (occupied << 16), e, at | (q << 16));
    }
  }
}

template <typename IdT, int CTAS, int ROUNDS, int LANES>
__global__ void __launch_bounds__(sorting::kThreads) plan_kernel(const IdT* ids, int numel, int E, const int32_t* emap, int E_local,
                                                                 int gran_shift, int tile_rows, int32_t* row_index, int rows_cap,
                                                                 int4* tiles, int tiles_cap, int32_t* counts, int32_t* status) {
  plan_body<IdT, CTAS, ROUNDS, LANES>(ids, numel, E, emap, E_local, gran_shift, tile_rows, row_index, rows_cap, tiles, tiles_cap, counts, status);
}

// Up to 32 ids: one warp, everything in registers and votes, no shared memory and no barrier (one token of 8 routes:
// 4.1 us of the layer with the kernel above, 1.4 us here).  No expert has more than one tile.
constexpr int kWarpIds = 32;
template <typename IdT>
__global__ void __launch_bounds__(32) plan_warp_kernel(const IdT* __restrict__ ids, int numel, int E, const int32_t* __restrict__ emap,
                                                       int E_local, int gran, int32_t* __restrict__ row_index, int rows_cap,
                                                       int4* __restrict__ tiles, int tiles_cap, int32_t* __restrict__ counts,
                                                       int32_t* __restrict__ status) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x;
  int e = INT_MAX;
  if (lane < numel) {
    const long long id = (long long)ids[lane];
    if (id >= 0 && id < E) {
      const int m = emap == nullptr ? (int)id : emap[(int)id];
      if (m >= 0 && m < E_local) e = m;
    } else if (id >= E) {
      set_status(status, MOE_ST_BAD_EXPERT_ID);
    }
  }
  const unsigned same = __match_any_sync(0xFFFFFFFFu, e), earlier = (1u << lane) - 1u;
  const int mine = __popc(same);
  const bool first = e != INT_MAX && (same & earlier) == 0;
  const unsigned firsts = __ballot_sync(0xFFFFFFFFu, first);
  int row0 = 0, at = 0, rows = 0;
  for (unsigned left = firsts; left != 0; left &= left - 1) {
    const int j = __ffs(left) - 1;
    const int ej = __shfl_sync(0xFFFFFFFFu, e, j), nj = (__shfl_sync(0xFFFFFFFFu, mine, j) + gran - 1) / gran * gran;
    rows += nj;
    if (ej < e) { row0 += nj; ++at; }
  }
  if (first && at < tiles_cap) tiles[at] = make_int4(row0, ((mine + gran - 1) / gran * gran) | (mine << 16), e, at | (1 << 16));
  if (lane < numel) row_index[lane] = e == INT_MAX ? -1 : row0 + __popc(same & earlier);
  if (lane == 0) {
    counts[0] = min(__popc(firsts), tiles_cap);
    counts[1] = min(rows, rows_cap);
  }
}

template <typename IdT>
int launch_plan(const void* ids, int numel, int E, const int32_t* emap, int E_local, int gran, int tile_rows, int32_t* row_index,
                int rows_cap, int4* tiles, int tiles_cap, int32_t* counts, int32_t* status, cudaStream_t st) {
  using namespace sorting;
  if (numel <= kWarpIds && (kWarpIds + gran - 1) / gran * gran <= tile_rows)
    return launch_pdl(plan_warp_kernel<IdT>, dim3(1), 32, 0, 1, st, "route plan (warp)", (const IdT*)ids, numel, E, emap, E_local, gran,
                      row_index, rows_cap, tiles, tiles_cap, counts, status);
  // the kernel counts rows in granules and tiles in 16 bits each
  if (gran < 16 || (gran & (gran - 1)) != 0 || rows_cap / gran > 65535 || tiles_cap > 65535)
    return fail(MOE_E_SHAPE, "route plan: granules of %d rows, at most 65535 of them and of tiles", gran);
  const int gran_shift = __builtin_ctz((unsigned)gran);
#define MOE_PLAN_B(C, R, B)                                                                                                    \
  launch_cluster(plan_kernel<IdT, C, R, B>, C, E_local, st, "route plan", (const IdT*)ids, numel, E, emap, E_local, gran_shift, \
                 tile_rows, row_index, rows_cap, tiles, tiles_cap, counts, status)
#define MOE_PLAN(C, R)                                                                                       \
  (lanes_by(E_local) == ONE_FIRST   ? MOE_PLAN_B(C, R, ONE_FIRST)                                            \
   : lanes_by(E_local) == LANE_BITS ? MOE_PLAN_B(C, R, LANE_BITS) : MOE_PLAN_B(C, R, VOTES))
  // one CTA while a warp sees at most two rounds of ids: no cluster barriers
  if (numel <= capacity(1, 2)) return MOE_PLAN(1, 2);
  if (numel <= capacity(kSmall, 2)) return MOE_PLAN(kSmall, 2);
  if (numel <= capacity(kLarge, 4)) return MOE_PLAN(kLarge, 4);
  return MOE_PLAN(kLarge, 16);
#undef MOE_PLAN
#undef MOE_PLAN_B
}
}  // namespace

// Capacities that hold for any routing of `numel` ids over E_local experts.
void plan_caps(int64_t numel, int E_local, int gran, int tile_rows, int64_t* rows_cap, int64_t* tiles_cap) {
  const int64_t used = numel < E_local ? numel : E_local;
  *rows_cap = ((numel + used * (gran - 1)) + gran - 1) / gran * gran;
  *tiles_cap = *rows_cap / tile_rows + used + 1;
}

// Not served where the device (or the partition of it) holds no cluster of the size that `numel` ids take: the layer then
// goes through moe_align_block_size, which has kernels without clusters.
bool plan_serves(int64_t numel, int E, int E_local) {
  using namespace sorting;
  if (E <= 0 || E_local <= 0 || E_local > kMaxExperts || numel <= 0 || numel > capacity(kLarge, 16)) return false;
  if (numel <= capacity(1, 2)) return true;
  if (numel <= capacity(kSmall, 2)) return cluster_fits(plan_kernel<int32_t, kSmall, 2, VOTES>, kSmall, E_local);
  if (numel <= capacity(kLarge, 4)) return cluster_fits(plan_kernel<int32_t, kLarge, 4, VOTES>, kLarge, E_local);
  return cluster_fits(plan_kernel<int32_t, kLarge, 16, VOTES>, kLarge, E_local);
}

int plan_routes(const void* ids, int ids64, int64_t numel, int E, const int32_t* emap, int E_local, int gran, int tile_rows,
                int32_t* row_index, int64_t rows_cap, void* tiles, int64_t tiles_cap, int32_t* counts, int32_t* status,
                cudaStream_t st) {
  return ids64 ? launch_plan<int64_t>(ids, (int)numel, E, emap, E_local, gran, tile_rows, row_index, (int)rows_cap, (int4*)tiles,
                                      (int)tiles_cap, counts, status, st)
               : launch_plan<int32_t>(ids, (int)numel, E, emap, E_local, gran, tile_rows, row_index, (int)rows_cap, (int4*)tiles,
                                      (int)tiles_cap, counts, status, st);
}

}  // namespace moe
