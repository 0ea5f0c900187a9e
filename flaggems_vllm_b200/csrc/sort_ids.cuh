// Stable counting sort of expert ids, the part that moe_align_block_size (align.cu) and the route plan (plan.cu)
// share.  One CTA of 1024 threads, or a cluster of 8 or 16 that exchange their per-expert counts through distributed shared
// memory.  Every warp owns a contiguous slice of the ids, at most ROUNDS x 32 of them: all loads are issued first,
// then the slice's ids are ranked round by round (votes, running counts of the slice in shared memory) and
// (expert, rank) stay in registers.  The position of an id is then
//     expert base + ids of that expert in earlier CTAs + in earlier warps + rank,
// its place in a stable sort.  Bound: the latency of this chain; ids are read once.
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
inline size_t smem_bytes(int E) { return ((size_t)kWarps * E + 4 * (size_t)E + 1) * 4; }

struct Shared {
  int32_t* hist;   // [kWarps][E]: ids of the expert in earlier warps of this CTA
  int32_t* total;  // [E]: ids of the expert in this CTA
  int32_t* base;   // [E + 1], [E], [E]: the caller's
  int32_t* count;
  int32_t* place;
};
__device__ __forceinline__ Shared carve(int32_t* smem, int E) {
  Shared s;
  s.hist = smem;
  s.total = smem + (size_t)kWarps * E;
  s.base = s.total + E;
  s.count = s.base + E + 1;
  s.place = s.count + E;
  return s;
}

// Lanes with the same value as this one; values < 2^bits.  One vote per bit: match.any walks the distinct values of
// the warp, up to 32 of them, and 32 warps of a CTA queue for it.
__device__ __forceinline__ unsigned peers(int v, int bits) {
  unsigned same = 0xFFFFFFFFu;
  for (int b = 0; b < bits; ++b) {
    const bool set = (v >> b) & 1;
    const unsigned vote = __ballot_sync(0xFFFFFFFFu, set);
    same &= set ? vote : ~vote;
  }
  return same;
}

// `expert(i)`: expert of id i in [0, E), or -1.  Returns with packed[r] = rank << 11 | expert (or kNone) of id
// first + 32 r + lane < end, hist / total filled and (cluster) every CTA's totals visible to all.
template <int CTAS, int ROUNDS, typename Expert>
__device__ __forceinline__ void rank_ids(int numel, int E, Shared sh, Expert expert, int (&packed)[ROUNDS], int& first, int& end) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  pdl_trigger();
  int rank = 0;
  if constexpr (CTAS > 1) rank = (int)cg::this_cluster().block_rank();
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
  for (int i = tid; i < slices * E; i += kThreads) sh.hist[i] = 0;
  __syncthreads();
  int32_t* h = sh.hist + (size_t)warp * E;
  const int bits = 32 - __clz(E);  // E itself stands for "none"
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    if (first + 32 * r >= end) {  // warp-uniform
      packed[r] = kNone;
      continue;
    }
    const int e = packed[r];
    const unsigned same = peers(e >= 0 ? e : E, bits);
    const int leader = __ffs(same) - 1;
    int old = 0;
    if (e >= 0 && lane == leader) {
      old = h[e];
      h[e] = old + __popc(same);
    }
    old = __shfl_sync(0xFFFFFFFFu, old, leader);
    packed[r] = e >= 0 ? ((old + __popc(same & ((1u << lane) - 1u))) << 11) | e : kNone;
    __syncwarp();
  }
  __syncthreads();
  for (int e = tid; e < E; e += kThreads) {
    int run = 0;
#pragma unroll 4
    for (int w = 0; w < slices; ++w) {
      const int c = sh.hist[(size_t)w * E + e];
      sh.hist[(size_t)w * E + e] = run;
      run += c;
    }
    sh.total[e] = run;
  }
  if constexpr (CTAS > 1) cg::this_cluster().sync();
  else __syncthreads();
}

// ids of expert e in all CTAs, and in the CTAs before this one
template <int CTAS>
__device__ __forceinline__ int count_all(const Shared& sh, int e, int& before) {
  before = 0;
  if constexpr (CTAS == 1) return sh.total[e];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  int all = 0;
#pragma unroll
  for (int r = 0; r < CTAS; ++r) {
    const int c = cluster.map_shared_rank(sh.total, r)[e];
    if (r < rank) before += c;
    all += c;
  }
  return all;
}

// Exclusive prefix of one 64-bit value per thread over the CTA (E <= threads: one chunk), and the sum.
__device__ __forceinline__ unsigned long long scan_cta(unsigned long long v, unsigned long long& sum) {
  __shared__ unsigned long long warp_sums[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned long long o = __shfl_up_sync(0xFFFFFFFFu, incl, off);
    if (lane >= off) incl += o;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  unsigned long long before = 0;
  sum = 0;
#pragma unroll 4
  for (int w = 0; w < kWarps; ++w) {
    const unsigned long long t = warp_sums[w];
    if (w < warp) before += t;
    sum += t;
  }
  return before + incl - v;
}

// Whether a cluster of this size can run at all; the callers have another way where it cannot.
template <typename Kernel>
bool cluster_fits(Kernel kern, int ctas, int E) {
  if (ctas == 1 || allow_smem((const void*)kern, (int)smem_bytes(kMaxExperts), ctas > 8) != 0) return true;
  return max_clusters((const void*)kern, ctas, kThreads, smem_bytes(E)) != 0;
}

template <typename Kernel, typename... Args>
int launch_cluster(Kernel kern, int ctas, int E, cudaStream_t st, const char* what, Args... args) {
  int rc = allow_smem((const void*)kern, (int)smem_bytes(kMaxExperts), ctas > 8);
  if (rc) return rc;
  return launch_pdl(kern, dim3((unsigned)ctas), kThreads, smem_bytes(E), ctas, st, what, args...);
}

}  // namespace sorting
}  // namespace moe
