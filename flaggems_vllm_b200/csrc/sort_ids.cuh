// Stable counting sort of expert ids, the part that moe_align_block_size (align.cu) and the route plan (plan.cu)
// share.  One CTA of 1024 threads, or a cluster of 8 or 16 that exchange their per-expert counts through distributed shared
// memory.  Every warp owns a contiguous slice of the ids, at most ROUNDS x 32 of them: all loads are issued first,
// then the slice's ids are ranked round by round (lane bits or votes, running counts of the slice in shared memory) and
// (expert, rank) stay in registers.  The position of an id is then
//     expert base + ids of that expert in earlier CTAs + in earlier warps + rank,
// its place in a stable sort.  Bound: the latency of this chain; ids are read once.  What it was before lane masks for votes,
// pushed totals for fetched ones and a scan of the warp sums by every warp, and is now, us back to back (256 experts): route
// plan of 488 ids 5.4 -> 3.4, 4000 6.5 -> 4.8, 16000 8.3 -> 5.8, 65536 12.3 -> 7.2.
#pragma once

#include <cooperative_groups.h>

#include "moe_common.cuh"

namespace moe {
namespace sorting {
namespace cg = cooperative_groups;

constexpr int kThreads = 1024, kWarps = 32;
constexpr int kMaxExperts = 1024;
constexpr int kNone = 0x7FF;  // expert field of an id that gets no place

// Clusters: 8 CTAs up to 16384 ids (two rounds per warp), 16 beyond; what a CTA does with its ids, not the exchange,
// is what grows.
constexpr int kSmall = 8, kLarge = 16;
// ids a launch with this many CTAs and rounds sorts
constexpr int64_t capacity(int ctas, int rounds) { return (int64_t)ctas * kWarps * rounds * 32; }
// Lanes of a warp with the same expert.  LANE_BITS: from a word of lane bits per expert and warp; its lanes queue for it, which
// costs most in a warp that has one expert alone.  Few experts make such warps likely, so below 16 that is asked first (ONE_FIRST):
// 262144 ids of 8 experts, in order: lane bits 16.5 us, asked first 9.7; drawn: 11.8, 12.3 (votes of four bits: 12.3, 13.8).
// VOTES: from 512 experts on, where the words would not fit.
constexpr int ONE_FIRST = 0, LANE_BITS = 1, VOTES = 2;
constexpr int lanes_by(int E) { return E < 16 ? ONE_FIRST : (E < 512 ? LANE_BITS : VOTES); }
constexpr bool by_masks(int E) { return lanes_by(E) != VOTES; }
inline size_t smem_bytes(int E, int ctas) {
  return ((size_t)kWarps * E * (by_masks(E) ? 2 : 1) + ((size_t)ctas + 3) * E + 1) * 4;
}

struct Shared {
  int32_t* hist;   // [kWarps][E]: ids of the expert in earlier warps of this CTA
  int32_t* total;  // [CTAS][E]: ids of the expert in every CTA of the cluster
  int32_t* base;   // [E + 1], [E], [E]: the caller's
  int32_t* count;
  int32_t* place;
  uint32_t* mask;  // by_masks: [kWarps][E], zero between rounds
};
template <int CTAS>
__device__ __forceinline__ Shared carve(int32_t* smem, int E) {
  Shared s;
  s.hist = smem;
  s.total = smem + (size_t)kWarps * E;
  s.base = s.total + (size_t)CTAS * E;
  s.count = s.base + E + 1;
  s.place = s.count + E;
  s.mask = reinterpret_cast<uint32_t*>(s.place + E);
  return s;
}

// Lanes with the same value as this one; values < 2^BITS.  One vote per bit: match.any walks the distinct values of
// the warp, up to 32 of them, and 32 warps of a CTA queue for it.  Votes are slow, too: 1300 cycles per round of 32 warps and
// nine bits, where setting and reading lane bits in shared memory takes 600.
constexpr int kBits = 11;
template <int BITS>
__device__ __forceinline__ unsigned peers(int v) {
  unsigned same = 0xFFFFFFFFu;
#pragma unroll
  for (int b = 0; b < BITS; ++b) {
    const unsigned vote = __ballot_sync(0xFFFFFFFFu, (v & (1 << b)) != 0);
    same &= ~(vote ^ (unsigned)((v << (31 - b)) >> 31));
  }
  return same;
}

// `expert(i)`: expert of id i in [0, E), or -1.  Returns with packed[r] = rank << 11 | expert (or kNone) of id
// first + 32 r + lane < end, hist filled and every CTA's totals in everybody's `total` (each CTA writes its own into all of
// them: a remote store waits for nothing, the barrier behind them for all of them).
template <int CTAS, int ROUNDS, int LANES, typename Expert>
__device__ __forceinline__ void rank_ids(int numel, int E, Shared sh, Expert expert, int (&packed)[ROUNDS], int& first, int& end) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  pdl_trigger();
  int rank = 0;
  if constexpr (CTAS > 1) {
    rank = (int)cg::this_cluster().block_rank();
    cg::this_cluster().barrier_arrive();  // this CTA runs: it may be written to
  }
  const int per_cta = ((numel + CTAS - 1) / CTAS + 31) & ~31;
  const int per_warp = ((per_cta + kWarps - 1) / kWarps + 31) & ~31;
  first = rank * per_cta + warp * per_warp;
  end = min(min(numel, (rank + 1) * per_cta), first + per_warp);
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int i = first + 32 * r + lane;
    packed[r] = i < end ? expert(i) : -1;
  }
  const int slices = min(kWarps, (per_cta + per_warp - 1) / per_warp);  // warps that own ids
  for (int i = tid; i < slices * E; i += kThreads) {
    sh.hist[i] = 0;
    if constexpr (LANES != VOTES) sh.mask[i] = 0;
  }
  __syncthreads();
  int32_t* h = sh.hist + (size_t)warp * E;
  [[maybe_unused]] uint32_t* mask = sh.mask + (size_t)warp * E;
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    if (first + 32 * r >= end) {  // warp-uniform
      packed[r] = kNone;
      continue;
    }
    const int e = packed[r];
    unsigned same = 0;
    if constexpr (LANES == VOTES) {
      same = peers<kBits>(e >= 0 ? e : E);  // E itself stands for "none"
    } else if (LANES == ONE_FIRST && __all_sync(0xFFFFFFFFu, e == __shfl_sync(0xFFFFFFFFu, e, 0))) {
      same = e >= 0 ? 0xFFFFFFFFu : 0u;
    } else {
      if (e >= 0) atomicOr(&mask[e], 1u << lane);
      __syncwarp();
      if (e >= 0) same = mask[e];
      __syncwarp();
    }
    const int leader = __ffs(same) - 1;
    int old = 0;
    if (e >= 0 && lane == leader) {
      old = h[e];
      h[e] = old + __popc(same);
      if constexpr (LANES != VOTES) mask[e] = 0;
    }
    old = __shfl_sync(0xFFFFFFFFu, old, leader & 31);
    packed[r] = e >= 0 ? ((old + __popc(same & ((1u << lane) - 1u))) << 11) | e : kNone;
    __syncwarp();
  }
  __syncthreads();
  if constexpr (CTAS > 1) cg::this_cluster().barrier_wait();
  if (tid < E) {
    int run = 0;
#pragma unroll 8
    for (int w = 0; w < slices; ++w) {
      const int c = sh.hist[(size_t)w * E + tid];
      sh.hist[(size_t)w * E + tid] = run;
      run += c;
    }
    if constexpr (CTAS > 1) {
#pragma unroll
      for (int r = 0; r < CTAS; ++r) cg::this_cluster().map_shared_rank(sh.total, r)[(size_t)rank * E + tid] = run;
    } else {
      sh.total[tid] = run;
    }
  }
  if constexpr (CTAS > 1) cg::this_cluster().sync();
  else __syncthreads();
}

// ids of expert e in all CTAs, and in the CTAs before this one
template <int CTAS>
__device__ __forceinline__ int count_all(const Shared& sh, int e, int E, int rank, int& before) {
  before = 0;
  int all = 0;
#pragma unroll
  for (int r = 0; r < CTAS; ++r) {
    const int c = sh.total[(size_t)r * E + e];
    if (r < rank) before += c;
    all += c;
  }
  return all;
}

// Inclusive prefix over the lanes of a warp.
__device__ __forceinline__ unsigned scan_warp(unsigned v, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned o = __shfl_up_sync(0xFFFFFFFFu, v, off);
    if (lane >= off) v += o;
  }
  return v;
}
// Exclusive prefix of one value per thread over the CTA, and the sum.  Every warp scans the warp sums for itself: 400 cycles
// with the barrier, where adding them up one by one in 64 bits took 2700.
__device__ __forceinline__ unsigned scan_cta(unsigned v, unsigned& sum) {
  __shared__ unsigned warp_sums[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned incl = scan_warp(v, lane);
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  const unsigned sums = scan_warp(warp_sums[lane], lane);
  sum = __shfl_sync(0xFFFFFFFFu, sums, 31);
  const unsigned before = __shfl_sync(0xFFFFFFFFu, sums, (warp + 31) & 31);
  return (warp > 0 ? before : 0u) + incl - v;
}

// Whether a cluster of this size can run at all; the callers have another way where it cannot.
template <typename Kernel>
bool cluster_fits(Kernel kern, int ctas, int E) {
  if (ctas == 1 || allow_smem((const void*)kern, (int)smem_bytes(kMaxExperts, ctas), ctas > 8) != 0) return true;
  return max_clusters((const void*)kern, ctas, kThreads, smem_bytes(E, ctas)) != 0;
}

template <typename Kernel, typename... Args>
int launch_cluster(Kernel kern, int ctas, int E, cudaStream_t st, const char* what, Args... args) {
  int rc = allow_smem((const void*)kern, (int)smem_bytes(kMaxExperts, ctas), ctas > 8);
  if (rc) return rc;
  return launch_pdl(kern, dim3((unsigned)ctas), kThreads, smem_bytes(E, ctas), ctas, st, what, args...);
}

}  // namespace sorting
}  // namespace moe
