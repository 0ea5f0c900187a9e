// What the grouped GEMMs with the weights as the M operand share (gemm_wt.cu: both operands from shared memory;
// gemm_w8t.cu: weight-only int8, the weights through tensor memory): the work list, and the way of a finished
// accumulator tile [weight row, token] through registers and shared memory to rows in HBM.
#pragma once

#include "tc_common.cuh"

namespace moe {
namespace wt {
using namespace tc;

constexpr int FMT_HALF = 0, FMT_FP8ROW = 2, FMT_I8ROW = 3, FMT_W8 = 4;

struct Params {
  const int4* tiles;        // {first row, rows | occupied rows << 16, expert, first tile of the expert | its tile count << 16}
  const int32_t* counts;    // [0] = number of tiles
  const float* a_scales;    // row-scaled: [rows_cap]
  const float* w_scale;     // row-scaled, weight-only int8: [E, rows_w]
  const float* row_weight;  // GEMM1 with the route weight on the input: [rows_cap], else null
  void* out;                // GEMM1: [rows_cap, I]; GEMM2: [rows_cap, H]
  int32_t* status;
  unsigned long long wait_ns;
  int E, K, Nout, R;        // R = row tiles per expert: 64 (GEMM1) or 128 (GEMM2) output columns for each CTA of a tile
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

// Work items, expert by expert; inside an expert the token tile runs fastest, so the CTAs that run at the same time
// read the same weight tile.
__device__ __forceinline__ Item fetch_item(const Params& P, int item) {
  Item it;
  const int t0 = item / P.R;
  int4 d = __ldcg(P.tiles + t0);  // past L1: this may run before pdl_wait()
  const int first = d.w & 0xFFFF, q = (int)((uint32_t)d.w >> 16);
  const int within = item - first * P.R;
  it.rt = within / q;
  const int t = first + within - it.rt * q;
  if (t != t0) d = __ldcg(P.tiles + t);
  it.row0 = d.x; it.n = d.y & 0xFFFF; it.e = d.z;
  return it;
}

// output columns of a warp's 32 weight rows
template <bool GEMM1> __host__ __device__ constexpr int warp_cols() { return GEMM1 ? 16 : 32; }

// Accumulator tile -> staged 16-bit rows [token][64 or 128 columns].  Warp quarter wq owns lanes 32 wq.., group h of
// GROUPS the h-th part of the tile's tokens; CTAS CTAs hold 128 weight rows each.  t_acc: TMEM address of the tile in
// the warp's lanes.  `release` runs when the whole accumulator is in registers or staged.  Rows are padded by
// 16 bytes, which spreads the rows of a stmatrix over the banks.
// WARP_TOKENS > 0 (one CTA, one group): the staging buffer at out_base is the warp's own and holds that many tokens of its 16
// (GEMM1) or 32 columns; it goes to HBM whenever it is full, in whole sectors, without a barrier between the warps.
// Rows of a thread: in 16-lane block rh (0, 1) of the warp's 32 lanes, lanes tr and tr + 8:
//   GEMM1: output 64 cr + 8 (2 wq + rh) + tr of the row tile (gate in lane tr, up in lane tr + 8)
//   GEMM2: output columns 128 cr + 32 wq + 16 rh + tr and + 8
template <int FMT, typename AT, bool GEMM1, bool SILU, int CTAS, int GROUPS, int WARP_TOKENS, typename Release>
__device__ __forceinline__ void drain_tile(const Params& P, const Item& it, int cr, uint32_t t_acc, int h, int wq, int lane,
                                           uint32_t out_base, Release release) {
  constexpr bool ROW = FMT == FMT_FP8ROW || FMT == FMT_I8ROW, CHANNEL = ROW || FMT == FMT_W8;
  constexpr bool WARP_STORE = WARP_TOKENS > 0;
  static_assert(!WARP_STORE || (CTAS == 1 && GROUPS == 1 && (WARP_TOKENS == 16 || WARP_TOKENS == 32)), "a warp's own staging buffer");
  constexpr int PITCH = (WARP_STORE ? warp_cols<GEMM1>() : (GEMM1 ? 64 : 128)) * 2 + 16;
  const int tr = lane >> 2, tq = lane & 3;
  const int nh = it.n / GROUPS, tok0 = h * nh;  // this group's tokens [tok0, tok0 + nh) of the tile
  const int nst = (nh + 31) >> 5;               // steps of 32 tokens
  // GEMM1: gate and up of (output, token) -> activation value
  auto activate = [&](float g, float u, float rw) -> float {
    g *= rw; u *= rw;
    if constexpr (ROW || !SILU) { g = round_act<AT>(g); u = round_act<AT>(u); }
    if constexpr (SILU) return silu_mul_fast(g, u);
    else return swigluoai(g, u, P.alpha, P.beta, P.limit);
  };
  float cs[2][2] = {{1.0f, 1.0f}, {1.0f, 1.0f}};  // channel scales of this thread's rows: [rh][lane tr / tr + 8]
  if constexpr (CHANNEL) {
    const float* ws = P.w_scale + (int64_t)it.e * (GEMM1 ? 2 * P.Nout : P.Nout);
#pragma unroll
    for (int rh = 0; rh < 2; ++rh) {
      if constexpr (GEMM1) {
        const int o = it.rt * (64 * CTAS) + cr * 64 + (2 * wq + rh) * 8 + tr;
        cs[rh][0] = __ldg(ws + o);
        cs[rh][1] = __ldg(ws + P.Nout + o);
      } else {
        const int o = it.rt * (128 * CTAS) + cr * 128 + wq * 32 + rh * 16 + tr;
        cs[rh][0] = o < P.Nout ? __ldg(ws + o) : 0.0f;
        cs[rh][1] = o + 8 < P.Nout ? __ldg(ws + o + 8) : 0.0f;
      }
    }
  }
#pragma unroll 1
  for (int st = 0; st < nst; ++st) {
    uint32_t r[32];
    tmem_ld_frag32_async(t_acc + (uint32_t)(tok0 + st * 32), r);
    tmem_ld_frag32_async(t_acc + (uint32_t)(tok0 + st * 32) + (16u << 16), r + 16);
    float2 as[4], rw[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const bool in = st * 32 + c * 8 < nh;
      const int64_t p = (int64_t)it.row0 + tok0 + st * 32 + c * 8 + 2 * tq;
      if constexpr (ROW) as[c] = in ? *reinterpret_cast<const float2*>(P.a_scales + p) : make_float2(0.0f, 0.0f);
      rw[c] = GEMM1 && in && P.row_weight != nullptr ? *reinterpret_cast<const float2*>(P.row_weight + p) : make_float2(1.0f, 1.0f);
    }
    tmem_wait32(r);
    if (st == nst - 1) release();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (st * 32 + c * 8 < nh) {
        float lo[2][2], hi[2][2];  // lanes tr / tr + 8 of block rh, token j of the pair
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
              else if constexpr (CHANNEL) v[l][j] *= cs[rh][l];
            }
          if constexpr (GEMM1) {
            lo[rh][0] = activate(v[0][0], v[1][0], rw[c].x);
            lo[rh][1] = activate(v[0][1], v[1][1], rw[c].y);
          } else {
            lo[rh][0] = v[0][0]; lo[rh][1] = v[0][1];
            hi[rh][0] = v[1][0]; hi[rh][1] = v[1][1];
          }
        }
        const uint32_t row = out_base + (uint32_t)((WARP_STORE ? c * 8 % (WARP_STORE ? WARP_TOKENS : 1) : tok0 + st * 32 + c * 8) + (lane & 7)) * PITCH;
        const int wqs = WARP_STORE ? 0 : wq;
        if constexpr (GEMM1)
          stmatrix_x2_trans(row + (uint32_t)((2 * wqs + ((lane >> 3) & 1)) * 16), pack2<AT>(lo[0][0], lo[0][1]), pack2<AT>(lo[1][0], lo[1][1]));
        else
          stmatrix_x4_trans(row + (uint32_t)(wqs * 64 + (lane >> 3) * 16), pack2<AT>(lo[0][0], lo[0][1]), pack2<AT>(hi[0][0], hi[0][1]),
                            pack2<AT>(lo[1][0], lo[1][1]), pack2<AT>(hi[1][0], hi[1][1]));
      }
      if constexpr (WARP_STORE) {
        if ((c + 1) * 8 % WARP_TOKENS == 0) {
          constexpr int LANES = warp_cols<GEMM1>() / 8;  // lanes of a row, 16 bytes each
          const int col = it.rt * (GEMM1 ? 64 : 128) + wq * warp_cols<GEMM1>() + (lane % LANES) * 8;
          const int first = st * 32 + (c + 1) * 8 - WARP_TOKENS, left = nh - first;
          __syncwarp();
          if (col < P.Nout) {
#pragma unroll
            for (int t0 = 0; t0 < WARP_TOKENS; t0 += 32 / LANES) {
              const int tok = t0 + lane / LANES;
              if (tok < left) {
                uint4 v;
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                             : "r"(out_base + (uint32_t)(tok * PITCH + (lane % LANES) * 16)) : "memory");
                *reinterpret_cast<uint4*>(reinterpret_cast<AT*>(P.out) + ((int64_t)it.row0 + first + tok) * P.Nout + col) = v;
              }
            }
          }
          __syncwarp();
        }
      }
    }
  }
}

// Staged rows -> HBM, 8 (GEMM1) or 16 lanes per row with 16 bytes each.
template <typename AT, bool GEMM1, int CTAS, int NTHREADS>
__device__ __forceinline__ void store_rows(const Params& P, const Item& it, int cr, const uint8_t* s_out, int et) {
  constexpr int LANES = GEMM1 ? 8 : 16, COLS = GEMM1 ? 64 : 128, PITCH = COLS * 2 + 16;
  const int sub = et % LANES;
  const int col = it.rt * (COLS * CTAS) + cr * COLS + sub * 8;
  if (col >= P.Nout) return;
  for (int tok = et / LANES; tok < it.n; tok += NTHREADS / LANES)
    *reinterpret_cast<uint4*>(reinterpret_cast<AT*>(P.out) + ((int64_t)it.row0 + tok) * P.Nout + col) =
        *reinterpret_cast<const uint4*>(s_out + (size_t)tok * PITCH + sub * 16);
}

}  // namespace wt
}  // namespace moe
