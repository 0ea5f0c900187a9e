// The whole expert layer behind one call: route plan -> scatter -> GEMM1 -> GEMM2 -> combine.
//
// The launches of a decode step take a few microseconds each; made one by one from Python (a dozen allocations, a
// ctypes call per launch) they cost the host more than the device.  Here the caller passes the workspaces and the
// launches follow each other in native code.  No state is kept between calls.
#include <cstring>

#include "moe_common.cuh"

namespace moe {
void plan_caps(int64_t numel, int E_local, int gran, int tile_rows, int64_t* rows_cap, int64_t* tiles_cap);
bool plan_serves(int64_t numel, int E, int E_local);
int plan_routes(const void* ids, int ids64, int64_t numel, int E, const int32_t* emap, int E_local, int gran, int tile_rows,
                int32_t* row_index, int64_t rows_cap, void* tiles, int64_t tiles_cap, int32_t* counts, int32_t* status,
                cudaStream_t st);
int scatter_quant_group(const void* x, int dtype, int64_t M, int H, int k, const int32_t* row_index, int64_t rows_cap, void* q,
                        float* scales_t, bool early, cudaStream_t st);
int scatter_rows(const void* x, int64_t M, int64_t row_bytes, int k, const int32_t* row_index, void* out, bool early,
                 cudaStream_t st);
int zero_padding(const void* tiles, int64_t tiles_cap, const int32_t* counts, int64_t row_bytes, void* rows, int groups,
                 int64_t rows_cap, float* scales_t, cudaStream_t st);
int tc_gemm_plan(bool gemm1, int act_dtype, const void* a, const float* a_scales_t, const void* w, const float* w_scale,
                 const void* tiles, const int32_t* rows, int64_t numel, int64_t rows_cap, int E, int K, int Nout, void* out,
                 float* out_scales_t, const float* row_weight, bool all_rows, bool staged, int32_t* status, cudaStream_t st);
int small_align(const void* ids, int ids64, int numel, int E, int32_t* sorted_ids, int rows_cap, int32_t* expert_ids, int32_t* npp,
                int32_t* counters, int ncounters, int32_t* status, cudaStream_t st);
int small_slices(int mode, bool gemm1, int K, int N, int blocks);
int small_gemm(bool pdl, int gemm1, int mode, int act_dtype, const void* a, int64_t num_tokens, int topk, const void* w,
               const float* w_scale, const int32_t* expert_ids, const int32_t* sorted_ids, const int32_t* num_post_pad,
               const int32_t* expert_map, int num_experts_global, const float* route_weight, int mul_weight, const void* topk_ids,
               int ids_int64, int64_t rows_cap, int E, int K, int Nout, void* out, void* final_out, int k_slices, float* partial,
               int32_t* unit_counters, int32_t* token_counters, int32_t* status, cudaStream_t st);
int scatter_floats(const float* src, int64_t numel, int div, const int32_t* row_index, float* dst, cudaStream_t st);
int combine_rows(const void* y, int dtype, const float* weight, const int32_t* row_index, int64_t M, int k, int64_t H, void* out,
                 bool early, cudaStream_t st);
int rowwise_quant(const void* x, int x_dtype, int64_t rows, int64_t cols, int kind, const float* scale_in,
                  const int32_t* row_ids, int64_t valid_below, const int32_t* indirect, void* q, float* scale_out, cudaStream_t st);
bool rowwise_scatter_serves(int kind, int64_t cols);
int rowwise_scatter(const void* x, int x_dtype, int64_t rows, int64_t cols, int kind, int k, const int32_t* row_index, void* q,
                    float* scales, bool early, cudaStream_t st);
bool wt_serves(int mode, int act_dtype, int H, int I);
int wt_gemm(bool gemm1, int mode, int tile_rows, int act_dtype, const void* a, const float* a_scales, const void* w, const float* w_scale,
            const void* tiles, int64_t tiles_cap, const int32_t* counts, const float* row_weight, int64_t rows_cap, int E, int K,
            int Nout, void* out, int act_kind, float alpha, float beta, float limit, int32_t* status,
            cudaStream_t st);
bool w8t_serves(int act_dtype, int H, int I);
int w8t_tile(bool wide);
int w8t_gemm(bool gemm1, bool wide, int act_dtype, const void* a, const void* w, const float* w_scale, const void* tiles,
             int64_t tiles_cap, const int32_t* counts, const float* row_weight, int64_t rows_cap, int E, int K, int Nout, void* out,
             int32_t* status, cudaStream_t st);

namespace {
// Which grouped GEMM serves the call and how the plan cuts the rows for it.
struct Choice {
  bool small;       // gemm_small.cu: blocks of 8 routes, K split over the chip; no scatter, the sum inside GEMM2
  bool pair;        // gemm_wt.cu: weights as the M operand of a CTA pair; else gemm_tc.cu (FP8 block scales): 128 tokens as M
  bool wide;        // weight-only int8 (gemm_w8t.cu): tiles of up to 160 tokens instead of 64
  int gran, tile;   // row granule and most rows of a tile
  bool zero_pad;    // gemm_tc.cu: zero the padding rows and fetch whole blocks
  bool staged;      // gemm_tc.cu: GEMM2 leaves through staged TMA stores of whole tiles
};

bool sizes_served(int mode, int act_dtype, int H, int I, int act_kind) {
  if (mode == MOE_MODE_FP8_BLOCK)
    return act_kind == MOE_ACT_SILU && (act_dtype == MOE_BF16 || act_dtype == MOE_F16) && H % 128 == 0 && I % 128 == 0;
  if (mode == MOE_MODE_W8A16) return act_kind == MOE_ACT_SILU && w8t_serves(act_dtype, H, I);
  return wt_serves(mode, act_dtype, H, I);
}

// The split-K weight streaming of gemm_small.cu: three launches instead of five, every SM busy however few tiles there
// are, but one CTA needs more instructions per byte than the pair.  It serves up to 8 routes that read up to 1 GB of weights if
// no two share an expert, which the host cannot see.  us per layer, bf16, split K against the pair in tiles of 64:
//   Mixtral shape    1 token  0.7 GB  137 : 127   2 tokens 1.4 GB  256 : 253 (against tokens as M; one pair of experts 143 : 168)
//   E8 H1024 I2048   1 token   25 MB   17 : 20    2 tokens          21 : 23    3 tokens 29 : 26    4 tokens 27 : 30
//   E8 H2048 I4096   1 token  101 MB   30 : 35    2 tokens 201 MB   43 : 44    4 tokens 403 MB     79 : 62
//   E128 H2048 I768  1 token   75 MB   29 : 29    E64 H2048 I1408   1 token 104 MB 34 : 32
// The times cross between 100 MB and 0.7 GB, but the line is not drawn there: the results are not the same.  Here the K slices' sums
// are added in fp32 and the activation is expf and a true division; the pair accumulates all of K in tensor memory and takes
// the fast exponential (Mixtral shape, one token: outputs up to 3.4e-3 apart).  Up to 1 GB a call keeps the former; beyond,
// distinct experts, the usual case, lose more than that is worth.
constexpr int kSmallRoutes = 8;
constexpr int64_t kSmallBytes = 1000000000;

bool row_mode(int mode) { return mode == MOE_MODE_FP8_ROW || mode == MOE_MODE_INT8_ROW; }

// Most rows of a pair's tile.  Small tiles leave shared memory to the ring and stream an even load's weights fastest; an expert
// with more rows than a tile reads its weights once more per tile, while HBM idles.  The host sees the mean load only (and that
// no expert has more rows than there are tokens), so the lines lie where skewed routing is no slower than under the
// schedule that was there before either tile: half precision tokens as M below 96 rows per expert and 256 from there on, else 256.
// us per layer (graph replay); even: uniform routing, zipf: popularity 1 / rank, hot: every token takes expert 0:
//   bf16 E8 k2 H4096 I14336      before    64    128    256          bf16 E64 k6 H2048 I1408   before    64    128    256
//     112 tokens (28 rows) even     455   428    437    475            200 tokens (18)  zipf      189   190    183    192
//                          hot      462   434    440    476            400 (37)         zipf      201   201    193    199
//     150 (37)             even     457   430    442    478            600 (56)         zipf      209   219    201    207
//                          hot      469   474    448    482            900 (84)         zipf      238   248    217    220
//     232 (58)             even     464   471    447    486            1200 (112)       even      227   246    213    220
//                          hot      477   522    455    499                             zipf      240   284    245    234
//     350 (87)             even     483   527    457    493
//                          zipf     640   590    520    504          e4m3, E128 k8 H2048 I768
//     400 (100)            even     519   539    465    509            1000 (62)        even      153          146    148
//                          hot      548   634    558    514                             zipf      158          153    152
//     440 (110)            even     522   548    472    509            1500 (93)        even      171          165    165
//                          hot      538   592    571    541                             zipf      178          179    172
//     480 (120)            zipf     528   622    542    527            1900 (118)       hot4      200          197    192
// The other activation has GEMM1 in tiles of 256 only, so half of the gain: bf16 232 tokens even 497 / 522 / 461 / 481 and hot 510 / 528 /
// 471 / 494, 300 tokens hot 517 / 572 / 547 / 506; int8 rows 256 is ahead from 31 rows per expert on (142 / - / 140 / 138).
int pair_tile(int mode, int act_kind, int64_t M, int64_t per_expert) {
  const bool half = mode == MOE_MODE_HALF;
  if (act_kind != MOE_ACT_SILU) return half && per_expert <= 64 ? 128 : 256;
  if (half) return M <= 128 && per_expert <= 32 ? 64 : (per_expert <= 100 ? 128 : 256);
  return per_expert <= 64 ? 128 : 256;
}

Choice choose(int mode, int act_kind, int64_t M, int topk, int E, int H, int I) {
  const int64_t numel = M * topk;
  const int64_t per_expert = numel / (E > 0 ? E : 1);
  Choice c = {};
  if (mode == MOE_MODE_W8A16) {
    // Qwen3 shape, GEMM1 + GEMM2 in us, narrow (more stages) against wide: 40 rows per expert 128 : 139, 50 rows 133 : 140,
    // 62 rows 170 : 153 (every second expert has more than 64 rows: two tiles).  Half of the routes on four experts, 51 rows: the
    // layer 173 us, 190 when it was wide from 40 rows on.
    c.wide = per_expert > 52;
    c.gran = 16;
    c.tile = w8t_tile(c.wide);
    return c;
  }
  if (mode == MOE_MODE_HALF && act_kind == MOE_ACT_SILU && numel <= kSmallRoutes && numel * 6 * H * I <= kSmallBytes &&
      H % 128 == 0 && I % 64 == 0) {
    c.small = true;
    return c;
  }
  // FP8 block scales: tokens as M (gemm_wt.cu says why).  All else: the pair, in tiles of pair_tile() rows.
  c.pair = mode != MOE_MODE_FP8_BLOCK;
  if (c.pair) {
    c.gran = mode == MOE_MODE_INT8_ROW ? 32 : 16;  // kind::i8 on a pair takes multiples of 32
    c.tile = pair_tile(mode, act_kind, M, per_expert);
  } else {
    c.gran = c.tile = 128;
    c.zero_pad = per_expert >= 128;
    c.staged = per_expert >= 64;
  }
  return c;
}

// Pieces of the four workspaces (plan; rows of GEMM1; intermediate; rows behind GEMM2): 256-byte aligned, with at
// least kGap bytes that nobody writes behind each, so that a write past the end of a piece can be seen.
constexpr int64_t kGap = 256;
struct Piece { int64_t ws, at, bytes; };
struct Pieces {
  Piece row_index, tiles, counts, row_weight, tmp_scales, x_rows, x_scales, tmp_q, act, act_q, act_scales, y, small_counters;
};
static_assert(sizeof(Pieces) == MOE_LAYER_PIECES * 3 * sizeof(int64_t), "moe_layer_layout hands the table out as it is");
struct Layout : Pieces {
  int64_t rows_cap, tiles_cap;
  int64_t bytes[4];
  int slices[2];         // gemm_small.cu: K slices of GEMM1, GEMM2
  int64_t ncounters[3];  // and its counters: units of GEMM1, of GEMM2, tokens of GEMM2
};

Layout layout(int mode, const Choice& c, int64_t M, int k, int E, int E_local, int H, int I) {
  Layout L = {};
  const int64_t numel = M * k;
  auto take = [&](int ws, int64_t bytes) {
    const Piece p = {ws, L.bytes[ws], bytes};
    if (bytes > 0) L.bytes[ws] += (bytes + 255) / 256 * 256 + kGap;
    return p;
  };
  const bool byte = mode != MOE_MODE_HALF && mode != MOE_MODE_W8A16, row = row_mode(mode), block = mode == MOE_MODE_FP8_BLOCK;
  if (c.small) {
    const int64_t used = numel < E ? numel : E;
    L.rows_cap = (numel + used * 7 + 7) / 8 * 8;
    int64_t part[2] = {0, 0}, units[2] = {0, 0}, toks = 0;
    for (int g = 0; g < 2; ++g) {
      L.slices[g] = small_slices(mode, g == 0, g == 0 ? H : I, g == 0 ? I : H, (int)used);
      moe_small_m_plan(g == 0, mode, g == 0 ? H : I, g == 0 ? I : H, L.rows_cap, M, L.slices[g], &part[g], &units[g], &toks);
    }
    L.ncounters[0] = units[0]; L.ncounters[1] = units[1]; L.ncounters[2] = toks;
    L.row_index = take(0, L.rows_cap * 4);   // sorted_ids
    L.tiles = take(0, L.rows_cap / 8 * 4);   // expert_ids
    L.counts = take(0, 8);                   // num_post_pad
    L.small_counters = take(0, (units[0] + units[1] + toks) * 4);
    L.x_rows = take(1, (part[0] > part[1] ? part[0] : part[1]) * 4 + 16);  // partial sums
    L.act = take(2, L.rows_cap * I * 2);
    L.y = take(3, numel * H * 2);
    return L;
  }
  plan_caps(numel, E_local, c.gran, c.tile, &L.rows_cap, &L.tiles_cap);
  L.row_index = take(0, numel * 4);
  L.tiles = take(0, L.tiles_cap * 16);
  L.counts = take(0, 8);
  L.row_weight = take(0, L.rows_cap * 4);
  L.tmp_scales = take(0, row ? M * 4 : 0);
  L.x_rows = take(1, L.rows_cap * H * (byte ? 1 : 2));
  L.x_scales = take(1, block ? L.rows_cap * (H / 128) * 4 : (row ? L.rows_cap * 4 : 0));
  L.tmp_q = take(1, row ? M * H : 0);
  L.act = take(2, L.rows_cap * I * (block ? 1 : 2));
  L.act_q = take(2, row ? L.rows_cap * I : 0);
  L.act_scales = take(2, block ? L.rows_cap * (I / 128) * 4 : (row ? L.rows_cap * 4 : 0));
  L.y = take(3, L.rows_cap * H * 2);
  return L;
}
}  // namespace
}  // namespace moe

extern "C" int moe_layer_workspace(int mode, int act_dtype, int64_t num_tokens, int topk, int num_experts, int E_local, int H,
                                   int I, int activation, int64_t* bytes) {
  return moe_layer_layout(mode, act_dtype, num_tokens, topk, num_experts, E_local, H, I, activation, bytes, nullptr);
}

extern "C" int moe_layer_layout(int mode, int act_dtype, int64_t num_tokens, int topk, int num_experts, int E_local, int H, int I,
                                int activation, int64_t* bytes, int64_t* pieces) {
  using namespace moe;
  if (num_tokens <= 0 || num_tokens > 65535 || topk <= 0 || topk > 32 || E_local <= 0 || H <= 0 || I <= 0 || !bytes ||
      !plan_serves(num_tokens * topk, num_experts, E_local) || !sizes_served(mode, act_dtype, H, I, activation))
    return fail(MOE_E_SHAPE, "layer: mode, type or sizes are not served by this call");
  const Layout L = layout(mode, choose(mode, activation, num_tokens, topk, num_experts, H, I), num_tokens, topk, num_experts, E_local, H, I);
  for (int i = 0; i < 4; ++i) bytes[i] = L.bytes[i];
  if (pieces) std::memcpy(pieces, static_cast<const Pieces*>(&L), sizeof(Pieces));
  return 0;
}

extern "C" int moe_layer(int mode, int act_dtype, const void* x, int64_t num_tokens, int topk, const void* topk_ids, int ids_int64,
                         const float* topk_weights, const void* w1, const float* w1_scale, const void* w2, const float* w2_scale,
                         void* out, int num_experts, const int32_t* expert_map, int E_local, int H, int I, int weight_on_input,
                         int activation, float alpha, float beta, float limit, int quant_kind1, const float* quant_scale1,
                         int quant_kind2, const float* quant_scale2, void* ws_plan, void* ws_x, void* ws_act, void* ws_y, int stages,
                         int32_t* status, void* stream) {
  using namespace moe;
  const int64_t M = num_tokens, numel = M * topk;
  int64_t bytes[4];
  int rc = moe_layer_workspace(mode, act_dtype, M, topk, num_experts, E_local, H, I, activation, bytes);
  if (rc) return rc;
  if (!x || !topk_ids || !topk_weights || !w1 || !w2 || !out || !ws_plan || !ws_x || !ws_act || !ws_y)
    return fail(MOE_E_BADARG, "layer: null pointer");
  if (((uintptr_t)x | (uintptr_t)out | (uintptr_t)ws_plan | (uintptr_t)ws_x | (uintptr_t)ws_act | (uintptr_t)ws_y) & 15)
    return fail(MOE_E_BADARG, "layer: rows and workspaces must be 16-byte aligned");
  const bool row = row_mode(mode), block = mode == MOE_MODE_FP8_BLOCK;
  if (mode != MOE_MODE_HALF && (!w1_scale || !w2_scale)) return fail(MOE_E_BADARG, "layer: weight scales missing");
  cudaStream_t st = (cudaStream_t)stream;
  const Choice c = choose(mode, activation, M, topk, num_experts, H, I);
  const Layout L = layout(mode, c, M, topk, num_experts, E_local, H, I);
  void* const base[4] = {ws_plan, ws_x, ws_act, ws_y};
  auto at = [&](const Piece& p) -> void* { return (uint8_t*)base[p.ws] + p.at; };
  int32_t* row_index = (int32_t*)at(L.row_index);
  int32_t* counts = (int32_t*)at(L.counts);
  void* tiles = at(L.tiles);
  float* x_scales = (float*)at(L.x_scales);
  float* act_scales = (float*)at(L.act_scales);
  float* row_weight = weight_on_input ? (float*)at(L.row_weight) : nullptr;
  if (c.small) {
    int32_t* cnt = (int32_t*)at(L.small_counters);
    int32_t* experts = (int32_t*)tiles;
    const int64_t* n = L.ncounters;
    if (stages & 1)
      rc = small_align(topk_ids, ids_int64, (int)numel, num_experts, row_index, (int)L.rows_cap, experts, counts, cnt,
                       (int)(n[0] + n[1] + n[2]), status, st);
    if (!rc && (stages & 4))
      rc = small_gemm(true, 1, mode, act_dtype, x, M, topk, w1, w1_scale, experts, row_index, counts, expert_map, num_experts,
                      topk_weights, weight_on_input, topk_ids, ids_int64, L.rows_cap, E_local, H, I, at(L.act), nullptr, L.slices[0],
                      (float*)at(L.x_rows), cnt, nullptr, status, st);
    if (!rc && (stages & 16))
      rc = small_gemm(true, 0, mode, act_dtype, at(L.act), M, topk, w2, w2_scale, experts, row_index, counts, expert_map, num_experts,
                      topk_weights, !weight_on_input, topk_ids, ids_int64, L.rows_cap, E_local, I, H, at(L.y), out, L.slices[1],
                      (float*)at(L.x_rows), cnt + n[0], cnt + n[0] + n[1], status, st);
    return rc;
  }
  if (stages & 1) {
    rc = plan_routes(topk_ids, ids_int64, numel, num_experts, expert_map, E_local, c.gran, c.tile,
                     row_index, L.rows_cap, tiles, L.tiles_cap, counts, status, st);
    if (rc) return rc;
  }
  if (stages & 2) {
    const bool early = (stages & 1) != 0 && M < 4 * sm_count();  // the kernel in front is this call's route plan, x is older
    if (block) {
      rc = scatter_quant_group(x, act_dtype, M, H, topk, row_index, L.rows_cap, at(L.x_rows), x_scales, early, st);
    } else if (row) {
      const bool per_row = quant_kind1 == 0 || quant_kind1 == 1;
      if (rowwise_scatter_serves(quant_kind1, H)) {
        rc = rowwise_scatter(x, act_dtype, M, H, quant_kind1, topk, row_index, at(L.x_rows), x_scales, early, st);
      } else {
        float* sc = (float*)at(L.tmp_scales);
        rc = rowwise_quant(x, act_dtype, M, H, quant_kind1, quant_scale1, nullptr, 0, nullptr, at(L.tmp_q), sc, st);
        if (!rc) rc = scatter_rows(at(L.tmp_q), M, H, topk, row_index, at(L.x_rows), false, st);  // behind the quantiser of its rows
        if (!rc) rc = scatter_floats(sc, numel, per_row ? topk : (int)numel, row_index, x_scales, st);
      }
    } else {
      rc = scatter_rows(x, M, (int64_t)H * 2, topk, row_index, at(L.x_rows), early, st);
    }
    if (!rc && c.zero_pad)
      rc = zero_padding(tiles, L.tiles_cap, counts, (int64_t)H * (block ? 1 : 2), at(L.x_rows), block ? H / 128 : 0, L.rows_cap,
                        block ? x_scales : nullptr, st);
    if (!rc && row_weight != nullptr) rc = scatter_floats(topk_weights, numel, 1, row_index, row_weight, st);
    if (rc) return rc;
  }
  if (stages & 4) {
    rc = mode == MOE_MODE_W8A16 ? w8t_gemm(true, c.wide, act_dtype, at(L.x_rows), w1, w1_scale, tiles, L.tiles_cap, counts, row_weight,
                                           L.rows_cap, E_local, H, I, at(L.act), status, st)
         : c.pair ? wt_gemm(true, mode, c.tile, act_dtype, at(L.x_rows), x_scales, w1, w1_scale, tiles, L.tiles_cap, counts, row_weight,
                          L.rows_cap, E_local, H, I, at(L.act), activation, alpha, beta, limit, status, st)
                : tc_gemm_plan(true, act_dtype, at(L.x_rows), x_scales, w1, w1_scale, tiles, counts + 1, numel, L.rows_cap,
                               E_local, H, I, at(L.act), act_scales, row_weight, c.zero_pad, c.staged, status, st);
    if (rc) return rc;
  }
  const void* act = at(L.act);
  if (row) {
    act = at(L.act_q);
    if (stages & 8) {
      const bool per_row = quant_kind2 == 0 || quant_kind2 == 1;
      float* sc = (float*)at(L.tmp_scales);
      rc = rowwise_quant(at(L.act), act_dtype, numel, I, quant_kind2, quant_scale2, nullptr, 0, row_index, at(L.act_q),
                         per_row ? act_scales : sc, st);
      if (!rc && !per_row) rc = scatter_floats(sc, numel, (int)numel, row_index, act_scales, st);
      if (rc) return rc;
    }
  }
  if (stages & 16) {
    rc = mode == MOE_MODE_W8A16 ? w8t_gemm(false, c.wide, act_dtype, act, w2, w2_scale, tiles, L.tiles_cap, counts, nullptr, L.rows_cap,
                                           E_local, I, H, at(L.y), status, st)
         : c.pair ? wt_gemm(false, mode, c.tile, act_dtype, act, act_scales, w2, w2_scale, tiles, L.tiles_cap, counts, nullptr, L.rows_cap,
                          E_local, I, H, at(L.y), MOE_ACT_SILU, 0.0f, 0.0f, 0.0f, status, st)
                : tc_gemm_plan(false, act_dtype, act, act_scales, w2, w2_scale, tiles, counts + 1, numel, L.rows_cap, E_local,
                               I, H, at(L.y), nullptr, nullptr, c.zero_pad, c.staged, status, st);
    if (rc) return rc;
  }
  if (stages & 32)
    rc = combine_rows(at(L.y), act_dtype, weight_on_input ? nullptr : topk_weights, row_index, M, topk, H, out, (stages & 16) != 0, st);
  return rc;
}
