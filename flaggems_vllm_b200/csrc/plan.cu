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
// One CTA, or (from 4096 ids on) a cluster of 8 that exchange their per-expert counts through distributed
// shared memory.  Each warp owns a contiguous slice of the ids.  One pass ranks the ids inside the slice
// (__match_any_sync, the slice's running counts in shared memory) and parks the rank in row_index; after the
// scan over slices and experts a second pass adds the base.  Bound: the latency of that chain.
#include <cooperative_groups.h>

#include "moe_common.cuh"

namespace cg = cooperative_groups;

namespace moe {
namespace {

constexpr int kPlanThreads = 1024;
constexpr int kPlanCluster = 8;

template <typename IdT, int CL>
__device__ __forceinline__ void plan_body(const IdT* __restrict__ ids, int numel, int E, const int32_t* __restrict__ emap,
                                          int E_local, int W, int gran, int tile_rows, int32_t* __restrict__ row_index, int rows_cap,
                                          int4* __restrict__ tiles, int tiles_cap, int32_t* __restrict__ counts,
                                          int32_t* __restrict__ status) {
  extern __shared__ int32_t smem[];
  // hist[W][E_local] | cta_tot[E_local] | scan words
  int32_t* hist = smem;
  int32_t* cta_tot = hist + (size_t)W * E_local;
  __shared__ unsigned long long warp_sums[32];
  __shared__ unsigned long long carry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
  int rank = 0;
  if constexpr (CL > 1) rank = (int)cg::this_cluster().block_rank();

  for (int i = tid; i < W * E_local; i += T) hist[i] = 0;
  if (tid == 0) carry = 0;
  __syncthreads();

  const int per_cta = ((numel + CL - 1) / CL + 31) & ~31;
  const int cbegin = rank * per_cta, cend = min(numel, cbegin + per_cta);
  const int per_warp = (((per_cta + W - 1) / W) + 31) & ~31;
  const int begin = cbegin + warp * per_warp, end = min(cend, begin + per_warp);
  auto local_expert = [&](int i, bool& bad) -> int {
    const long long e = (long long)ids[i];
    if (e < 0 || e >= E) {
      if (e >= E) bad = true;  // negative ids mean "no route" (padding rows, other ranks' slots)
      return -1;
    }
    if (emap == nullptr) return (int)e;
    const int m = emap[(int)e];
    return m >= 0 && m < E_local ? m : -1;
  };
  bool bad = false;
  if (warp < W) {
    int32_t* h = hist + (size_t)warp * E_local;
    for (int i0 = begin; i0 < end; i0 += 32) {
      const int i = i0 + lane;
      const int e = i < end ? local_expert(i, bad) : -1;
      const unsigned same = __match_any_sync(0xFFFFFFFFu, e);
      const int leader = __ffs(same) - 1;
      int old = 0;
      if (e >= 0 && lane == leader) {
        old = h[e];
        h[e] = old + __popc(same);
      }
      old = __shfl_sync(0xFFFFFFFFu, old, leader);
      if (i < end) row_index[i] = e >= 0 ? old + __popc(same & ((1u << lane) - 1u)) : -1;
      __syncwarp();
    }
  }
  if (bad) set_status(status, MOE_ST_BAD_EXPERT_ID);
  __syncthreads();
  for (int e = tid; e < E_local; e += T) {
    int run = 0;
#pragma unroll 8
    for (int w = 0; w < W; ++w) {
      const int c = hist[(size_t)w * E_local + e];
      hist[(size_t)w * E_local + e] = run;  // rows of expert e in earlier slices
      run += c;
    }
    cta_tot[e] = run;
  }
  if constexpr (CL > 1) cg::this_cluster().sync();
  else __syncthreads();

  // experts in chunks of T: exclusive scan of (tiles << 32 | padded rows)
  for (int e0 = 0; e0 < E_local; e0 += T) {
    const int e = e0 + tid;
    int before = 0, total = 0, padded = 0, q = 0;
    if (e < E_local) {
      if constexpr (CL > 1) {
        cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
        for (int r = 0; r < CL; ++r) {
          const int c = cluster.map_shared_rank(cta_tot, r)[e];
          if (r < rank) before += c;
          total += c;
        }
      } else {
        total = cta_tot[e];
      }
      padded = (total + gran - 1) / gran * gran;
      q = (padded + tile_rows - 1) / tile_rows;
    }
    const unsigned long long mine = ((unsigned long long)q << 32) | (unsigned)padded;
    unsigned long long incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long o = __shfl_up_sync(0xFFFFFFFFu, incl, off);
      if (lane >= off) incl += o;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const unsigned long long v = lane < (T >> 5) ? warp_sums[lane] : 0ull;
      unsigned long long s = v;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long o = __shfl_up_sync(0xFFFFFFFFu, s, off);
        if (lane >= off) s += o;
      }
      warp_sums[lane] = s - v;
    }
    __syncthreads();
    const unsigned long long base = carry + warp_sums[warp] + incl - mine;
    if (e < E_local) {
      const int row0 = (int)(base & 0xFFFFFFFFull), first = (int)(base >> 32);
#pragma unroll 8
      for (int w = 0; w < W; ++w) hist[(size_t)w * E_local + e] += row0 + before;
      if (q > 0 && (CL == 1 || e % CL == rank)) {
        const int size = ((padded / gran + q - 1) / q) * gran;  // even split, in multiples of gran rows
        for (int t = 0; t < q; ++t) {
          const int r = min(padded, t * size), n = min(size, padded - r);
          const int occupied = max(0, min(n, total - r));
          if (first + t < tiles_cap) tiles[first + t] = make_int4(row0 + r, max(n, 0) | (occupied << 16), e, first | (q << 16));
        }
      }
    }
    __syncthreads();
    if (tid == T - 1) carry = base + mine;
    __syncthreads();
  }
  if (rank == 0 && tid == 0) {
    counts[0] = min((int)(carry >> 32), tiles_cap);
    counts[1] = min((int)(carry & 0xFFFFFFFFull), rows_cap);
  }
  // second pass: every lane meets the ids it ranked itself
  if (warp < W) {
    const int32_t* h = hist + (size_t)warp * E_local;
    for (int i = begin + lane; i < end; i += 32) {
      const int r = row_index[i];
      if (r >= 0) row_index[i] = h[local_expert(i, bad)] + r;
    }
  }
  if constexpr (CL > 1) cg::this_cluster().sync();  // no CTA leaves while its counts may still be read
}

template <typename IdT>
__global__ void __launch_bounds__(kPlanThreads) plan_kernel(const IdT* ids, int numel, int E, const int32_t* emap, int E_local,
                                                            int W, int gran, int tile_rows, int32_t* row_index, int rows_cap,
                                                            int4* tiles, int tiles_cap, int32_t* counts, int32_t* status) {
  plan_body<IdT, 1>(ids, numel, E, emap, E_local, W, gran, tile_rows, row_index, rows_cap, tiles, tiles_cap, counts, status);
}
template <typename IdT>
__global__ void __cluster_dims__(kPlanCluster, 1, 1) __launch_bounds__(kPlanThreads)
plan_cluster_kernel(const IdT* ids, int numel, int E, const int32_t* emap, int E_local, int W, int gran, int tile_rows,
                    int32_t* row_index, int rows_cap, int4* tiles, int tiles_cap, int32_t* counts, int32_t* status) {
  plan_body<IdT, kPlanCluster>(ids, numel, E, emap, E_local, W, gran, tile_rows, row_index, rows_cap, tiles, tiles_cap, counts, status);
}

template <typename IdT>
int launch_plan(const void* ids, int numel, int E, const int32_t* emap, int E_local, int gran, int tile_rows, int32_t* row_index,
                int rows_cap, int4* tiles, int tiles_cap, int32_t* counts, int32_t* status, cudaStream_t st) {
  const bool cluster = numel >= 4096;
  // one slice per 64 ids: a decode-sized call clears and scans one or two histograms
  int W = kPlanThreads / 32;
  const int slices = ((cluster ? numel / kPlanCluster : numel) + 63) / 64;
  if (slices < W) W = slices < 1 ? 1 : slices;
  while (W > 1 && ((size_t)(W + 1) * E_local) * 4 > 160 * 1024) W >>= 1;
  const size_t smem = (size_t)(W + 1) * E_local * 4;
  auto kern = cluster ? plan_cluster_kernel<IdT> : plan_kernel<IdT>;
  const int rc = allow_smem((const void*)kern, 168 * 1024);
  if (rc) return rc;
  const int threads = cluster ? kPlanThreads : (W * 32 > E_local ? W * 32 : (E_local < kPlanThreads ? (E_local + 31) / 32 * 32 : kPlanThreads));
  kern<<<cluster ? kPlanCluster : 1, threads, smem, st>>>((const IdT*)ids, numel, E, emap, E_local, W, gran, tile_rows, row_index,
                                                          rows_cap, tiles, tiles_cap, counts, status);
  return check_launch("route plan");
}
}  // namespace

// Capacities that hold for any routing of `numel` ids over E_local experts.
void plan_caps(int64_t numel, int E_local, int gran, int tile_rows, int64_t* rows_cap, int64_t* tiles_cap) {
  const int64_t used = numel < E_local ? numel : E_local;
  *rows_cap = ((numel + used * (gran - 1)) + gran - 1) / gran * gran;
  *tiles_cap = *rows_cap / tile_rows + used + 1;
}

bool plan_serves(int64_t numel, int E, int E_local) {
  return E <= 1024 && E_local <= 1024 && E_local > 0 && numel > 0 && numel <= (1 << 20);
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
