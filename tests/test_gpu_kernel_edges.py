"""The newer kernels at the sizes where they can go wrong: edges of tiles, remainders, the smallest and the
largest of the range that their dispatch rule sends them."""

import ctypes

import pytest
import torch

import flaggems_vllm_b200 as fg
from flaggems_vllm_b200 import _lib, testing as T
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _route(M, E, k, seed=5):
    logits, _ = T.make_router_inputs(M, E, DEV, seed=seed)
    w, ids = torch.topk(torch.softmax(logits, -1), k, dim=-1)
    return (w / w.sum(-1, keepdim=True)).contiguous(), ids.to(torch.int32).contiguous()


def _parity(out, ref, what):
    assert _lib.read_status() == 0
    assert O.rel_l2(out.float(), ref) < 1e-2 and O.cosine(out.float(), ref) > 0.9999, what


@pytest.mark.parametrize("fmt", ["fp8", "int8"])
@pytest.mark.parametrize("M,E,k,H,I", [(1, 8, 2, 256, 128), (129, 4, 2, 1152, 384), (700, 4, 2, 256, 640),
                                         (208, 16, 4, 1408, 1920), (212, 16, 4, 1408, 1920)])  # last of the 64-row tiles, first of the others
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_row_scaled_tensor_core_layer(fmt, M, E, k, H, I, dtype):
    x = T.make_activations(M, H, DEV, dtype=dtype)
    w1f = torch.randn(E, 2 * I, H, device=DEV) * H**-0.5
    w2f = torch.randn(E, H, I, device=DEV) * I**-0.5
    tw, ti = _route(M, E, k)
    top = 448.0 if fmt == "fp8" else 127.0
    s1, s2 = w1f.abs().amax(-1) / top, w2f.abs().amax(-1) / top
    cast = (lambda w: w.to(torch.float8_e4m3fn)) if fmt == "fp8" else (lambda w: w.round().to(torch.int8))
    w1, w2 = cast(w1f / s1[..., None]), cast(w2f / s2[..., None])
    kw = {"use_fp8_w8a8": True} if fmt == "fp8" else {"use_int8_w8a8": True}
    out = fg.fused_experts_impl(x, w1, w2, tw, ti, per_channel_quant=True, w1_scale=s1, w2_scale=s2, **kw)
    _parity(out, O.fused_moe_row_scaled_oracle(x, w1, w2, s1, s2, tw, ti, fmt=fmt, per_token=True), (fmt, M))


@pytest.mark.parametrize("cols", [8, 768, 2048, 2056, 7168, 8192, 8200])
def test_rowwise_quant_widths(cols):
    """A warp per row up to 2048 columns, a CTA per row up to 8192, the scalar kernel beyond; padding rows skipped."""
    x = (torch.randn(11, cols, device=DEV) * 3).to(torch.bfloat16)
    x[4] = 0
    ids = torch.arange(11, dtype=torch.int32, device=DEV)
    ids[7] = 11
    for kind, oracle in ((0, O.int8_per_token_quant_oracle), (1, O.fp8_per_token_quant_oracle)):
        q = torch.full(x.shape, 77, dtype=torch.uint8, device=DEV)
        sc = torch.full((11,), -1.0, device=DEV)
        _lib.check(_lib.lib().moe_rowwise_quant(x.data_ptr(), _lib.dtype_code(x.dtype), 11, cols, kind, None,
                                                ids.data_ptr(), 11, q.data_ptr(), sc.data_ptr(), _lib.stream_of(x)))
        oq, os_ = oracle(x.cpu())
        rows = [r for r in range(11) if r != 7]
        assert torch.equal(q.cpu()[rows], oq.view(torch.uint8)[rows]) and torch.equal(sc.cpu()[rows], os_.reshape(-1)[rows])
        assert bool((q[7] == 77).all()) and float(sc[7]) == -1.0


@pytest.mark.parametrize("M,N,K", [(5, 256, 7168), (65, 256, 7168), (128, 8, 64), (129, 33, 72), (200, 256, 7168), (257, 40, 520),
                                   (4097, 128, 2048), (640, 1024, 512)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_router_gemm_tensor_core_tiles(M, N, K, dtype):
    """Row, column and K remainders of the tcgen05 tiles, every split of K over a cluster that the rule picks."""
    x = T.make_activations(M, K, DEV, seed=M, dtype=dtype)
    w = torch.randn((N, K), generator=torch.Generator(device=DEV).manual_seed(N), device=DEV).to(dtype)
    out = fg.router_gemm(x, w)
    ref = x.double() @ w.double().t()
    assert float((out.double() - ref).norm() / ref.norm()) < 4e-6 and _lib.read_status() == 0
    assert torch.equal(out, fg.router_gemm(x, w))


@pytest.mark.parametrize("M", [1, 2, 3, 4])
def test_router_gemm_row_tiles_share_one_order(M):
    """The decode kernel's tiles differ in shape only: row m of a batch equals the one-row call, bit for bit."""
    x = T.make_activations(M, 2048, DEV, seed=M)
    w = torch.randn((130, 2048), device=DEV).to(torch.bfloat16)
    out = fg.router_gemm(x, w)
    for m in range(M):
        assert torch.equal(out[m:m + 1], fg.router_gemm(x[m:m + 1], w))
    x32 = T.make_activations(37, 2048, DEV, seed=M, dtype=torch.float32)  # 8-row tiles, 1 and 4 columns wide
    out = fg.router_gemm(x32, w)
    assert torch.equal(out[:9], fg.router_gemm(x32[:9], w)) and torch.equal(out[36:], fg.router_gemm(x32[36:], w))


def _half_layer(M, E, k, H, I, dtype, **kw):
    x = T.make_activations(M, H, DEV, seed=M, dtype=dtype)
    w1 = T.make_half_weights(E, 2 * I, H, DEV, seed=1, dtype=dtype, std=H**-0.5)
    w2 = T.make_half_weights(E, H, I, DEV, seed=2, dtype=dtype, std=I**-0.5)
    tw, ti = _route(M, E, k)
    return x, w1, w2, tw, ti


@pytest.mark.parametrize("M,E,k,H,I", [
    (16, 4, 1, 192, 128), (50, 8, 2, 320, 256),      # tokens as M: a few rows per block, K of an odd number of stages
    (290, 3, 1, 256, 128), (1000, 4, 2, 448, 384),   # CTA pair: tiles of 96 / 112 .. rows, last 256-column tile half empty
    (2100, 4, 2, 128, 128), (513, 1, 1, 576, 256)])  # several tiles per expert, one expert
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_half_layer_tiles(M, E, k, H, I, dtype):
    x, w1, w2, tw, ti = _half_layer(M, E, k, H, I, dtype)
    _parity(fg.fused_experts_impl(x, w1, w2, tw, ti), O.fused_moe_half_oracle(x, w1, w2, tw, ti), (M, E))


@pytest.mark.parametrize("M,E,k", [(2, 8, 2), (40, 8, 2), (520, 4, 2), (1100, 4, 2)])
def test_fp8_block_layer_tiles(M, E, k):
    """Occupied rows only, whole blocks, row stores and staged stores of the 128-row kernel over a route plan."""
    H, I = 384, 256
    x = T.make_activations(M, H, DEV, seed=M)
    w1, s1 = T.make_fp8_block_weights(E, 2 * I, H, DEV, seed=1)
    w2, s2 = T.make_fp8_block_weights(E, H, I, DEV, seed=2)
    tw, ti = _route(M, E, k)
    kw = dict(use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2, block_shape=[128, 128])
    out = fg.fused_experts_impl(x, w1, w2, tw, ti, **kw)
    _parity(out, O.fused_moe_fp8_block_oracle(x, w1, w2, s1, s2, tw, ti), M)
    x2 = x.clone()
    assert torch.equal(fg.fused_experts_impl(x2, w1, w2, tw, ti, inplace=True, **kw), out)


@pytest.mark.parametrize("M,E,k,H,I", [(16384, 8, 2, 128, 128), (2600, 4, 2, 384, 1664), (900, 32, 4, 640, 1152)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_fp8_block_layer_odd_k_blocks_and_several_tiles_per_cta(M, E, k, H, I, dtype):
    """One K block or an odd number of them in a tile: the two accumulators, the stages and the scale slots do not start
    the next tile of the CTA where they started this one."""
    x = T.make_activations(M, H, DEV, seed=M, dtype=dtype)
    w1, s1 = T.make_fp8_block_weights(E, 2 * I, H, DEV, seed=1)
    w2, s2 = T.make_fp8_block_weights(E, H, I, DEV, seed=2)
    tw, ti = _route(M, E, k)
    out = fg.fused_experts_impl(x, w1, w2, tw, ti, use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2, block_shape=[128, 128])
    _parity(out, O.fused_moe_fp8_block_oracle(x, w1, w2, s1, s2, tw, ti), (M, H, I))


@pytest.mark.parametrize("M", [3, 700])  # a block per 16 groups of a token, a block per token
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_scattered_fp8_rows_are_the_quantisers(M, dtype):
    """Bytes and scales of the sorted rows against the stand-alone quantiser: zeros of either sign, subnormals, the type's
    largest, infinities and NaN among them, and every magnitude in between."""
    E, k, H, I = 4, 2, 8320, 128
    x = T.make_activations(M, H, DEV, seed=M, dtype=dtype)
    x *= torch.logspace(-30 if dtype == torch.bfloat16 else -6, 4, H // 128, device=DEV).repeat_interleave(128).to(dtype)
    big = torch.finfo(dtype).max
    for i, v in enumerate((0.0, -0.0, torch.finfo(dtype).tiny / 4, big, -big, float("inf"), -float("inf"), float("nan"))):
        x[i % M, 128 * i + i:128 * i + 128:7] = v
    x[M - 1, -128:] = -0.0
    ti = torch.stack([torch.arange(M, device=DEV) % E, (torch.arange(M, device=DEV) + 1) % E], 1).to(torch.int32)
    tw = torch.ones(M, k, device=DEV)
    w1, s1 = T.make_fp8_block_weights(E, 2 * I, H, DEV, seed=1)
    w2, s2 = T.make_fp8_block_weights(E, H, I, DEV, seed=2)
    sizes = (_lib.MODE_FP8_BLOCK, _lib.dtype_code(dtype), M, k, E, E, H, I, _lib.ACT_SILU)
    need, table = (ctypes.c_int64 * 4)(), (ctypes.c_int64 * (3 * 13))()
    _lib.check(_lib.lib().moe_layer_layout(*sizes, ctypes.addressof(need), ctypes.addressof(table)))
    ws = [torch.zeros(n, dtype=torch.uint8, device=DEV) for n in need]
    out = torch.empty_like(x)
    _lib.check(_lib.lib().moe_layer(
        sizes[0], sizes[1], x.data_ptr(), M, k, ti.data_ptr(), 0, tw.data_ptr(), w1.data_ptr(), s1.data_ptr(), w2.data_ptr(),
        s2.data_ptr(), out.data_ptr(), E, None, E, H, I, 0, _lib.ACT_SILU, 0.0, 0.0, 0.0, 0, None, 0, None,
        *[w.data_ptr() for w in ws], 1 | 2, _lib.status_word(torch.device(DEV)).data_ptr(), _lib.stream_of(x)))
    piece = lambda i, t: ws[table[3 * i]][table[3 * i + 1]:table[3 * i + 1] + table[3 * i + 2]].view(t)
    rows = piece(0, torch.int32).view(M, k).long()
    q, s = fg.per_token_group_quant_fp8(x, 128)
    got, scales = piece(5, torch.uint8).view(-1, H), piece(6, torch.float32).view(H // 128, -1)
    for j in range(k):
        assert torch.equal(got[rows[:, j]], q.view(torch.uint8))
        assert torch.equal(scales[:, rows[:, j]].t().contiguous().view(torch.int32), s.view(torch.int32))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_scattered_fp8_bytes_are_those_of_the_division(dtype):
    """Every pair of finite magnitudes (amax of the 128-group, |v| <= amax) of the type, about 5e8 of them, either sign: a group
    holds an amax and 127 of its values.  The kernel multiplies by a reciprocal and corrects; torch divides."""
    H, I, chunk = 7168, 128, 8192
    top = 0x7F7F if dtype == torch.bfloat16 else 0x7BFF  # bits of the largest finite value
    per_amax = torch.arange(1, top + 1, device=DEV).div(127, rounding_mode="floor") + 1  # groups for the values 0 .. amax
    amax = torch.repeat_interleave(torch.arange(1, top + 1, device=DEV), per_amax)
    first = torch.arange(amax.numel(), device=DEV) - torch.repeat_interleave(per_amax.cumsum(0) - per_amax, per_amax)
    sizes = (_lib.MODE_FP8_BLOCK, _lib.dtype_code(dtype), chunk, 1, 1, 1, H, I, _lib.ACT_SILU)
    need, table = (ctypes.c_int64 * 4)(), (ctypes.c_int64 * (3 * 13))()
    _lib.check(_lib.lib().moe_layer_layout(*sizes, ctypes.addressof(need), ctypes.addressof(table)))
    ws = [torch.zeros(n, dtype=torch.uint8, device=DEV) for n in need]
    ids, one = torch.zeros(chunk, dtype=torch.int32, device=DEV), torch.ones(chunk, device=DEV)
    w = torch.zeros(16, device=DEV)  # not read: the first two steps only
    piece = lambda i, t: ws[table[3 * i]][table[3 * i + 1]:table[3 * i + 1] + table[3 * i + 2]].view(t)
    lane, pairs = torch.arange(128, device=DEV), 0
    for g0 in range(0, amax.numel(), chunk * (H // 128)):
        a, f = amax[g0:g0 + chunk * (H // 128)], first[g0:g0 + chunk * (H // 128)]
        bits = torch.minimum(f[:, None] * 127 + (lane - 1), a[:, None])
        bits[:, 0] = a
        pairs += int((f[:, None] * 127 + (lane[1:] - 1) <= a[:, None]).sum())
        bits |= ((lane + f[:, None]) % 2) << 15
        x = torch.zeros((chunk * (H // 128), 128), dtype=dtype, device=DEV)
        x[:a.numel()] = torch.where(bits >= 0x8000, bits - 0x10000, bits).to(torch.int16).view(dtype)
        _lib.check(_lib.lib().moe_layer(
            sizes[0], sizes[1], x.data_ptr(), chunk, 1, ids.data_ptr(), 0, one.data_ptr(), w.data_ptr(), w.data_ptr(), w.data_ptr(),
            w.data_ptr(), x.data_ptr(), 1, None, 1, H, I, 0, _lib.ACT_SILU, 0.0, 0.0, 0.0, 0, None, 0, None,
            *[t.data_ptr() for t in ws], 1 | 2, _lib.status_word(torch.device(DEV)).data_ptr(), _lib.stream_of(x)))
        v = x.float()
        s = v.abs().amax(-1, keepdim=True).clamp(min=1e-10) * (1.0 / 448.0)
        want = (v / s).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)
        got = piece(5, torch.uint8).view(-1, 128)[:want.shape[0]]  # one expert: the rows are the tokens, in order
        assert torch.equal(got, want)
        assert torch.equal(piece(6, torch.float32).view(H // 128, -1)[:, :chunk].t().reshape(-1, 1), s)
    assert pairs == top * (top + 1) // 2 + top


@pytest.mark.parametrize("M,E,k,H,I", [
    (1, 1, 1, 128, 64), (1, 8, 8, 256, 192), (8, 2, 1, 2176, 128), (4, 8, 2, 1024, 2048),
    (3, 4, 3, 128, 64)])  # nine routes: the tile kernels
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_half_layer_few_routes(M, E, k, H, I, dtype):
    """One to eight routes (one K slice and several), a repeated call on the same stream, int64 ids, no route at all."""
    x, w1, w2, tw, ti = _half_layer(M, E, k, H, I, dtype)
    ref = O.fused_moe_half_oracle(x, w1, w2, tw, ti)
    out = fg.fused_experts_impl(x, w1, w2, tw, ti)
    _parity(out, ref, (M, E))
    assert torch.equal(fg.fused_experts_impl(x, w1, w2, tw, ti.long()), out)
    ti[0] = -1
    out = fg.fused_experts_impl(x, w1, w2, tw, ti)
    assert bool((out[0] == 0).all())
    if M > 1:
        _parity(out[1:], ref[1:], (M, E))


@pytest.mark.parametrize("M,k", [(1, 12), (4, 8), (32, 1), (33, 1), (11, 3)])
@pytest.mark.parametrize("spread", [1, 12])
def test_plan_of_few_routes(M, k, spread):
    """Up to 32 routes (one warp) and just above: all on one expert or spread, local experts only, ids out of range."""
    E, H, I = 12, 256, 128
    x = T.make_activations(M, H, DEV, seed=M)
    w1, s1 = T.make_int8_channel_weights(E, 2 * I, H, DEV, seed=1)
    w2, s2 = T.make_int8_channel_weights(E, H, I, DEV, seed=2)
    tw, ti = _route(M, E, k)
    if spread == 1:
        ti = torch.full_like(ti, 5)
    emap = torch.full((E,), -1, dtype=torch.int32, device=DEV)
    emap[4:9] = torch.arange(5, dtype=torch.int32, device=DEV).flip(0)
    ti[M // 2, k - 1] = -1
    keep = (ti >= 4) & (ti < 9)
    ref = O.fused_moe_w8a16_oracle(x, w1, w2, s1, s2, tw * keep, ti.clamp(min=0))
    loc = lambda w: w[4:9].flip(0).contiguous()
    out = fg.fused_experts_impl(x, loc(w1), loc(w2), tw, ti, use_int8_w8a16=True, per_channel_quant=True, w1_scale=loc(s1),
                                w2_scale=loc(s2), global_num_experts=E, expert_map=emap)
    _parity(out, ref, (M, k))
    assert bool((out[~keep.any(1)] == 0).all())


@pytest.mark.parametrize("M", [7, 300, 2500])
def test_layer_with_local_experts_and_weights_on_the_input(M):
    """expert_map (routes of other ranks get no rows), ids out of range, route weights applied on the input."""
    E, k, H, I = 12, 3, 256, 128
    x, w1, w2, tw, ti = _half_layer(M, E, k, H, I, torch.bfloat16)
    emap = torch.full((E,), -1, dtype=torch.int32, device=DEV)
    emap[4:8] = torch.arange(4, dtype=torch.int32, device=DEV)
    ti[M // 2, 1] = -1
    keep = (ti >= 4) & (ti < 8)
    ref = O.fused_moe_half_oracle(x, w1, w2, tw * keep, ti.clamp(min=0))
    out = fg.fused_experts_impl(x, w1[4:8].contiguous(), w2[4:8].contiguous(), tw, ti, global_num_experts=E, expert_map=emap)
    _parity(out, ref, M)
    assert bool((out[~keep.any(1)] == 0).all())
    if M > 100:
        full = ti.clamp(min=0)
        out = fg.fused_experts_impl(x, w1, w2, tw, full, apply_router_weight_on_input=True)
        ref = O.fused_moe_half_oracle(x, w1, w2, tw, full, apply_router_weight_on_input=True)
        _parity(out, ref, M)


@pytest.mark.parametrize("M,E,k,H,I", [
    (20, 4, 2, 192, 128), (90, 3, 1, 256, 384),      # 64-token tiles: a last K block of 64, several tiles of one expert
    (200, 2, 1, 320, 256), (1300, 4, 2, 128, 128),   # 160-token tiles: even splits with remainders
    (208, 16, 4, 448, 1920), (212, 16, 4, 448, 1920), (1500, 16, 4, 448, 1920)])  # either tile's last and first; many tiles per CTA
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_int8_weight_layer_tiles(M, E, k, H, I, dtype):
    x = T.make_activations(M, H, DEV, seed=M, dtype=dtype)
    w1, s1 = T.make_int8_channel_weights(E, 2 * I, H, DEV, seed=1, std=H**-0.5)
    w2, s2 = T.make_int8_channel_weights(E, H, I, DEV, seed=2, std=I**-0.5)
    tw, ti = _route(M, E, k)
    out = fg.fused_experts_impl(x, w1, w2, tw, ti, use_int8_w8a16=True, per_channel_quant=True, w1_scale=s1, w2_scale=s2)
    _parity(out, O.fused_moe_w8a16_oracle(x, w1, w2, s1, s2, tw, ti), (M, E))


@pytest.mark.parametrize("numel", [1, 31, 2048, 2049, 16384, 16385, 65536, 65537, 262144, 262145])
@pytest.mark.parametrize("E,bs", [(5, 16), (256, 128), (1024, 7)])
def test_align_slices(numel, E, bs):
    """Clusters of 8 and 16, 2 to 16 rounds of ids per warp; ids without a place; every slot written."""
    ids = T.make_align_ids(numel, 1, E, DEV, skewed=E > 5, seed=numel)
    if numel > 40:
        ids[7], ids[numel // 2] = -1, -3
    got = fg.moe_align_block_size(ids, bs, E)
    ref = O.moe_align_block_size_oracle(ids.cpu(), bs, E)
    for g, r in zip(got, ref):
        assert torch.equal(g.cpu(), torch.as_tensor(r))


@pytest.mark.parametrize("E", [511, 512])
@pytest.mark.parametrize("numel", [33, 2048, 2049, 16384, 16385, 65537])
def test_sorted_ids_either_side_of_the_lane_masks(E, numel):
    """Up to 511 experts the lanes of an expert are found by lane masks, beyond by votes: align, and the route plan of a layer
    whose tiles, rows and combine follow it."""
    ids = T.make_align_ids(numel, 1, E, DEV, skewed=numel % 2 == 1, seed=numel)
    ids[5], ids[numel // 2] = -1, E - 1
    got = fg.moe_align_block_size(ids, 32, E)
    ref = O.moe_align_block_size_oracle(ids.cpu(), 32, E)
    for g, r in zip(got, ref):
        assert torch.equal(g.cpu(), torch.as_tensor(r))
    H = I = 128
    k = 1 if numel % 2 else 2
    M = numel // k
    ti = ids[:M * k].view(M, k).contiguous()
    if k == 2:
        ti[:, 1] = (ti[:, 0].clamp(min=0) + 1) % E
    x, w1, w2, tw, _ = _half_layer(M, E, k, H, I, torch.bfloat16)
    out = fg.fused_experts_impl(x, w1, w2, tw, ti)
    keep = ti >= 0
    rows = torch.arange(0, M, max(1, M // 300), device=DEV)  # the oracle on some of the tokens
    ref = O.fused_moe_half_oracle(x[rows], w1, w2, (tw * keep)[rows], ti.clamp(min=0)[rows])
    _parity(out[rows], ref, (M, E))


@pytest.mark.parametrize("M", [5, 591, 592])  # 148 multiprocessors: the last size that reads tokens early, the first that does not
@pytest.mark.parametrize("fmt", ["half", "fp8_block", "fp8_channel"])
def test_tokens_and_weights_written_right_before_the_layer(fmt, M):
    """The scatter reads its tokens and the combine its plan and weights before their predecessors have ended.  Layers in place,
    one behind the other, each on what the last one wrote, equal layers with a synchronisation between, bit for bit."""
    E, k, H, I = 8, 2, 1024, 512
    kw = {}
    w1f, w2f = torch.randn(E, 2 * I, H, device=DEV) * 4 * H**-0.5, torch.randn(E, H, I, device=DEV) * 4 * I**-0.5
    if fmt == "half":
        w1, w2 = w1f.bfloat16(), w2f.bfloat16()
    elif fmt == "fp8_block":
        (w1, s1), (w2, s2) = (T.make_fp8_block_weights(E, n, kk, DEV, seed=n, std=4 * kk**-0.5) for n, kk in ((2 * I, H), (H, I)))
        kw = dict(use_fp8_w8a8=True, block_shape=[128, 128], w1_scale=s1, w2_scale=s2)
    else:
        s1, s2 = w1f.abs().amax(-1) / 448.0, w2f.abs().amax(-1) / 448.0
        w1, w2 = (w1f / s1[..., None]).to(torch.float8_e4m3fn), (w2f / s2[..., None]).to(torch.float8_e4m3fn)
        kw = dict(use_fp8_w8a8=True, per_channel_quant=True, w1_scale=s1, w2_scale=s2)
    routes = [_route(M, E, k, seed=i) for i in range(4)]
    xs = [T.make_activations(M, H, DEV, seed=i) for i in range(8)]
    want = []
    for x in xs:
        for tw, ti in routes:
            torch.cuda.synchronize()
            x = fg.fused_experts_impl(x, w1, w2, tw, ti, **kw)
        want.append(x)
    torch.cuda.synchronize()
    x, tw, ti = torch.empty_like(xs[0]), torch.empty_like(routes[0][0]), torch.empty_like(routes[0][1])
    got = []
    for src in xs:
        x.copy_(src)
        for a, b in routes:
            ti.copy_(b)
            tw.copy_(a)
            fg.fused_experts_impl(x, w1, w2, tw, ti, inplace=True, **kw)
        got.append(x.clone())
    assert _lib.read_status() == 0
    for g, w in zip(got, want):
        assert w.float().norm() > 0 and torch.equal(g, w)


@pytest.mark.parametrize("limit", [1, 8])
@pytest.mark.parametrize("numel", [0, 1, 2049, 4097, 16385, 65537, 262144])
@pytest.mark.parametrize("E,bs", [(5, 16), (256, 128), (1024, 7)])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_align_where_large_clusters_do_not_run(limit, numel, E, bs, dtype):
    """A partition of the GPU may hold no cluster of 16, or none of 8: other kernels, the same outputs."""
    ids = T.make_align_ids(numel, 1, E, DEV, skewed=E > 5, seed=numel).to(dtype)
    if numel > 40:
        ids[7], ids[numel // 2] = -1, -3
    cap = numel + E * (bs - 1)
    got = [torch.full((n,), -7, dtype=torch.int32, device=DEV) for n in (cap, -(-cap // bs), 1)]
    _lib.check(_lib.lib().moe_align_block_size_ex(
        ids.data_ptr(), int(dtype == torch.int64), numel, E, bs, got[0].data_ptr(), cap, got[1].data_ptr(), got[1].numel(),
        got[2].data_ptr(), limit, _lib.status_word(DEV).data_ptr(), _lib.stream_of(ids)))
    for g, r in zip(got, fg.moe_align_block_size(ids, bs, E)):
        assert torch.equal(g[:r.numel()], r)
    assert _lib.read_status() == 0


@pytest.mark.parametrize("fmt", ["half", "fp8_block", "int8_weight", "fp8_row", "int8_row"])
def test_layer_where_the_route_plan_does_not_run(fmt, monkeypatch):
    """The plan of more than 2048 routes needs a cluster; without one the layer goes through the align kernels."""
    M, E, k, H, I = 1100, 4, 2, 256, 128
    x, w1, w2, tw, ti = _half_layer(M, E, k, H, I, torch.bfloat16)
    kw = {}
    if fmt == "half":
        ref = O.fused_moe_half_oracle(x, w1, w2, tw, ti)
    elif fmt == "fp8_block":
        (w1, s1), (w2, s2) = T.make_fp8_block_weights(E, 2 * I, H, DEV, seed=1), T.make_fp8_block_weights(E, H, I, DEV, seed=2)
        kw = dict(use_fp8_w8a8=True, block_shape=[128, 128], w1_scale=s1, w2_scale=s2)
        ref = O.fused_moe_fp8_block_oracle(x, w1, w2, s1, s2, tw, ti)
    else:
        w1, s1 = T.make_int8_channel_weights(E, 2 * I, H, DEV, seed=1)
        w2, s2 = T.make_int8_channel_weights(E, H, I, DEV, seed=2)
        if fmt == "fp8_row":
            w1, w2 = w1.to(torch.float8_e4m3fn), w2.to(torch.float8_e4m3fn)
        option = {"int8_weight": "use_int8_w8a16", "fp8_row": "use_fp8_w8a8", "int8_row": "use_int8_w8a8"}[fmt]
        kw = {"per_channel_quant": True, "w1_scale": s1, "w2_scale": s2, option: True}
        ref = (O.fused_moe_w8a16_oracle(x, w1, w2, s1, s2, tw, ti) if fmt == "int8_weight" else
               O.fused_moe_row_scaled_oracle(x, w1, w2, s1.reshape(E, -1), s2.reshape(E, -1), tw, ti, fmt=fmt[:-4], per_token=True))

    class NoPlan:
        fused_experts = staticmethod(lambda *a: None)

    served = fg.fused_experts_impl(x, w1, w2, tw, ti, **kw)
    monkeypatch.setattr(_lib, "host", lambda: NoPlan)
    monkeypatch.setattr("flaggems_vllm_b200.fused_moe._workspace_bytes", lambda *a: None)
    staged = fg.fused_experts_impl(x, w1, w2, tw, ti, **kw)
    _parity(served, ref, fmt)
    _parity(staged, ref, fmt)


@pytest.mark.parametrize("fmt,M,kernels", [
    ("half", 2, 3),        # split K: align, GEMM 1, GEMM 2 with the sum
    ("half", 300, 5),      # plan, scatter, GEMM 1, GEMM 2, sum
    ("fp8_block", 300, 6),  # the padding rows of whole blocks are cleared besides
    ("int8_row", 300, 6),  # the intermediate has its own quantiser
    ("align", 64, 1),
    ("fp8_tensor_quant", 64, 3)])  # one scale for the tensor: its largest value, the scale, the quantiser
def test_launch_count_is_the_number_of_kernels(fmt, M, kernels):
    E, k, H, I = 4, 2, 256, 128
    x, w1, w2, tw, ti = _half_layer(M, E, k, H, I, torch.bfloat16)
    if fmt == "align":
        call = lambda: fg.moe_align_block_size(ti, 16, E)
    elif fmt == "fp8_tensor_quant":
        q, sc = torch.empty(x.shape, dtype=torch.uint8, device=DEV), torch.empty(1, device=DEV)
        call = lambda: _lib.check(_lib.lib().moe_rowwise_quant(x.data_ptr(), _lib.dtype_code(x.dtype), M, H, 3, None, None, 0,
                                                               q.data_ptr(), sc.data_ptr(), _lib.stream_of(x)))
    else:
        kw = {}
        if fmt == "fp8_block":
            (w1, s1), (w2, s2) = T.make_fp8_block_weights(E, 2 * I, H, DEV), T.make_fp8_block_weights(E, H, I, DEV)
            kw = dict(use_fp8_w8a8=True, block_shape=[128, 128], w1_scale=s1, w2_scale=s2)
        elif fmt == "int8_row":
            (w1, s1), (w2, s2) = T.make_int8_channel_weights(E, 2 * I, H, DEV), T.make_int8_channel_weights(E, H, I, DEV)
            kw = dict(use_int8_w8a8=True, per_channel_quant=True, w1_scale=s1, w2_scale=s2)
        call = lambda: fg.fused_experts_impl(x, w1, w2, tw, ti, **kw)
    call()
    before = _lib.LAUNCHES
    call()
    assert _lib.LAUNCHES - before == kernels


@pytest.mark.parametrize("M", [3, 300, 2500])
@pytest.mark.parametrize("staged", [False, True])
def test_expert_map_shorter_than_the_expert_count(M, staged, monkeypatch):
    """Ids beyond the map have no local expert; the kernels, which look up every id below the count, get a map that long."""
    E, k, H, I = 12, 3, 256, 128
    x, w1, w2, tw, ti = _half_layer(M, E, k, H, I, torch.bfloat16)
    emap = torch.tensor([-1, 1, 0, 3, -1, 2], dtype=torch.int32, device=DEV)
    order = [2, 1, 5, 3]  # global expert of local expert 0, 1, 2, 3
    keep = torch.isin(ti, torch.tensor(order, dtype=torch.int32, device=DEV))
    ref = O.fused_moe_half_oracle(x, w1, w2, tw * keep, ti)
    if staged:
        monkeypatch.setenv("FLAGGEMS_B200_PRESORT", "auto")  # any of the switches takes the staged pipeline
    out = fg.fused_experts_impl(x, w1[order].contiguous(), w2[order].contiguous(), tw, ti, global_num_experts=E, expert_map=emap)
    _parity(out, ref, M)
    assert bool((out[~keep.any(1)] == 0).all())


def test_fp8_expert_of_more_blocks_than_a_group_of_the_tile_order():
    """K = 7168: 18 blocks of 128 rows share a pass over the column tiles.  Experts of 41 (three groups of 14, 14, 13), 19 (10 and
    9), 18, one and no blocks; rows do not depend on the order, bit for bit."""
    counts, H, I = (41 * 128 - 5, 18 * 128 + 1, 18 * 128, 3, 0), 7168, 256
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32, device=DEV) for e, n in enumerate(counts)])
    ids = ids[torch.randperm(ids.numel(), generator=torch.Generator().manual_seed(3)).to(DEV)][:, None].contiguous()
    M, E = ids.shape[0], len(counts)
    x = T.make_activations(M, H, DEV, seed=4)
    tw = torch.rand((M, 1), device=DEV) + 0.5
    w1, s1 = T.make_fp8_block_weights(E, 2 * I, H, DEV, seed=1)
    w2, s2 = T.make_fp8_block_weights(E, H, I, DEV, seed=2)
    kw = dict(use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2, block_shape=[128, 128])
    out = fg.fused_experts_impl(x, w1, w2, tw, ids, **kw)
    _parity(out, O.fused_moe_fp8_block_oracle(x, w1, w2, s1, s2, tw, ids), counts)
    for m0 in range(0, M, 2000):  # at most nine blocks per expert
        part = slice(m0, m0 + 2000)
        assert torch.equal(fg.fused_experts_impl(x[part], w1, w2, tw[part], ids[part], **kw), out[part])


def _fixed_routes(counts, k, seed):
    """Expert e gets counts[e] routes of sum / k tokens, no token the same expert twice: slot j deals out the j-th part of a list."""
    flat = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(counts)])
    M = flat.numel() // k
    assert flat.numel() == M * k and max(counts) <= M
    ids = flat.view(k, M).t()[torch.randperm(M, generator=torch.Generator().manual_seed(seed))].contiguous().to(DEV)
    return torch.rand((M, k), generator=torch.Generator().manual_seed(seed)).to(DEV) + 0.5, ids


@pytest.mark.parametrize("fmt,k,counts", [
    ("half", 2, (128, 65, 62, 1, 0, 0, 0, 0)), ("half", 1, (64, 1, 0, 63)),                # tiles of 64 rows: two full ones, 65 rows, one
    ("half", 2, (129, 128, 1, 0, 0, 0, 0, 0)), ("half", 1, (128, 129, 257, 1, 0, 64, 65, 56)), ("half", 1, (380, 3, 0, 0)),  # 128 rows
    ("half", 1, (256, 257, 486, 1)), ("half", 1, (404, 4, 0, 0)),                          # 256 rows
    ("fp8", 1, (128, 129, 257, 1, 0, 64, 65, 56, 0, 0, 0, 0)), ("fp8", 1, (256, 257, 486, 1)),
    ("int8", 1, (128, 129, 257, 1, 0, 64, 65, 56, 0, 0, 0, 0)), ("int8", 1, (256, 257, 486, 1))])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_pair_tiles_full_and_one_row_over(fmt, k, counts, dtype):
    """Experts that fill a tile of the CTA pair exactly, have one row more, one row and none, in each tile size; rings and
    accumulators wrap from tile to tile.  A row does not depend on the tile it is in, bit for bit: half the tokens at a time,
    in tiles of other rows and, where the line is crossed, of another size."""
    E, H, I = len(counts), 4224, 2560
    tw, ti = _fixed_routes(counts, k, sum(counts))
    M = ti.shape[0]
    x = T.make_activations(M, H, DEV, seed=M, dtype=dtype)
    w1 = T.make_half_weights(E, 2 * I, H, DEV, seed=1, dtype=dtype, std=H**-0.5)
    w2 = T.make_half_weights(E, H, I, DEV, seed=2, dtype=dtype, std=I**-0.5)
    if fmt == "half":
        kw, ref = {}, O.fused_moe_half_oracle(x, w1, w2, tw, ti)
    else:
        top = 448.0 if fmt == "fp8" else 127.0
        s1, s2 = w1.float().abs().amax(-1) / top, w2.float().abs().amax(-1) / top
        cast = (lambda w: w.to(torch.float8_e4m3fn)) if fmt == "fp8" else (lambda w: w.round().to(torch.int8))
        w1, w2 = cast(w1.float() / s1[..., None]), cast(w2.float() / s2[..., None])
        kw = {"use_fp8_w8a8" if fmt == "fp8" else "use_int8_w8a8": True, "per_channel_quant": True, "w1_scale": s1, "w2_scale": s2}
        ref = O.fused_moe_row_scaled_oracle(x, w1, w2, s1, s2, tw, ti, fmt=fmt, per_token=True)
    out = fg.fused_experts_impl(x, w1, w2, tw, ti, **kw)
    _parity(out, ref, (fmt, counts))
    for part in (slice(0, M // 2), slice(M // 2, M)):
        assert torch.equal(fg.fused_experts_impl(x[part], w1, w2, tw[part], ti[part], **kw), out[part])


@pytest.mark.parametrize("fmt", ["fp8", "half", "fp8_row"])
@pytest.mark.parametrize("inplace", [False, True])
def test_scatter_and_combine_either_side_of_four_tokens_per_sm(fmt, inplace):
    """Parts of a token per block and the plan not waited for, below; a block per token, from there on: the same rows, bit for bit."""
    M, E, k, H, I = 4 * torch.cuda.get_device_properties(0).multi_processor_count, 16, 3, 1152, 128
    x = T.make_activations(M, H, DEV, seed=M)
    tw, ti = _route(M, E, k)
    if fmt == "half":
        w1, w2 = (T.make_half_weights(E, n, K, DEV, seed=n, std=K**-0.5) for n, K in ((2 * I, H), (H, I)))
        kw, ref = {}, O.fused_moe_half_oracle(x, w1, w2, tw, ti)
    elif fmt == "fp8":
        (w1, s1), (w2, s2) = (T.make_fp8_block_weights(E, n, K, DEV, seed=n) for n, K in ((2 * I, H), (H, I)))
        kw = dict(use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2, block_shape=[128, 128])
        ref = O.fused_moe_fp8_block_oracle(x, w1, w2, s1, s2, tw, ti)
    else:
        w1f, w2f = torch.randn(E, 2 * I, H, device=DEV) * H**-0.5, torch.randn(E, H, I, device=DEV) * I**-0.5
        s1, s2 = w1f.abs().amax(-1) / 448.0, w2f.abs().amax(-1) / 448.0
        w1, w2 = (w1f / s1[..., None]).to(torch.float8_e4m3fn), (w2f / s2[..., None]).to(torch.float8_e4m3fn)
        kw = dict(use_fp8_w8a8=True, per_channel_quant=True, w1_scale=s1, w2_scale=s2)
        ref = O.fused_moe_row_scaled_oracle(x, w1, w2, s1, s2, tw, ti, fmt="fp8", per_token=True)
    out = fg.fused_experts_impl(x.clone(), w1, w2, tw, ti, inplace=inplace, **kw)
    _parity(out, ref, fmt)
    assert torch.equal(fg.fused_experts_impl(x[:M - 1].clone(), w1, w2, tw[:M - 1], ti[:M - 1], inplace=inplace, **kw), out[:M - 1])


@pytest.mark.parametrize("M,N,K,columns,split", [
    (200, 256, 7168, 32, 8), (1000, 256, 7168, 64, 4), (2600, 256, 7168, 256, 4), (4000, 256, 7168, 256, 4), (8192, 256, 7168, 256, 2)])
def test_router_gemm_adds_the_partial_sums_of_each_split(M, N, K, columns, split):
    """The split of K is part of the result: undivided sums of K = 7168 are twice as far from 64-bit arithmetic."""
    c, s = ctypes.c_int(), ctypes.c_int()
    _lib.check(_lib.lib().moe_router_gemm_tile(M, N, K, 148, 8, ctypes.addressof(c), ctypes.addressof(s)))
    assert (c.value, s.value) == (columns, split)  # on a device of 148 multiprocessors
    x = T.make_activations(M, K, DEV, seed=M)
    w = torch.randn((N, K), generator=torch.Generator(device=DEV).manual_seed(N), device=DEV).to(torch.bfloat16)
    out = fg.router_gemm(x, w)
    ref = x.double() @ w.double().t()
    assert float((out.double() - ref).norm() / ref.norm()) < 4e-6 and _lib.read_status() == 0


@pytest.mark.parametrize("fmt,counts", [
    ("half", (128, 129, 3, 0)), ("half", (64, 64, 64, 67)),                   # 65 and 64 rows per expert: tiles of 256 and of 128
    ("half", (257, 256, 300, 1)), ("int8", (31, 64, 65, 0)), ("int8", (256, 257, 288, 1)), ("fp8", (128, 129, 257, 1))])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_other_activation_in_the_pair_tiles(fmt, counts, dtype):
    """GEMM1 has the 256-row kernel for it, GEMM2 the kernel of the plan's tiles; a row is the same in another batch, bit for bit."""
    E, H, I = len(counts), 1152, 1664
    tw, ti = _fixed_routes(counts, 1, 7)
    M = ti.shape[0]
    x = T.make_activations(M, H, DEV, seed=M, dtype=dtype)
    kw = dict(activation="swigluoai_uninterleave", gemm1_alpha=1.702, gemm1_beta=1.0, gemm1_clamp_limit=7.0)
    w1 = T.make_half_weights(E, 2 * I, H, DEV, seed=1, dtype=dtype, std=H**-0.5)
    w2 = T.make_half_weights(E, H, I, DEV, seed=2, dtype=dtype, std=I**-0.5)
    if fmt == "half":
        ref = O.fused_moe_half_oracle(x, w1, w2, tw, ti, act_fn=lambda z: O.swigluoai_oracle(z, 1.702, 1.0, 7.0))
    else:
        top = 448.0 if fmt == "fp8" else 127.0
        s1, s2 = w1.float().abs().amax(-1) / top, w2.float().abs().amax(-1) / top
        cast = (lambda w: w.to(torch.float8_e4m3fn)) if fmt == "fp8" else (lambda w: w.round().to(torch.int8))
        w1, w2 = cast(w1.float() / s1[..., None]), cast(w2.float() / s2[..., None])
        kw |= {"use_fp8_w8a8" if fmt == "fp8" else "use_int8_w8a8": True, "per_channel_quant": True, "w1_scale": s1, "w2_scale": s2}
        ref = O.fused_moe_row_scaled_oracle(x, w1, w2, s1, s2, tw, ti, fmt=fmt, per_token=True, activation="swigluoai_uninterleave")
    out = fg.fused_experts_impl(x, w1, w2, tw, ti, **kw)
    _parity(out, ref, (fmt, counts))
    half = slice(0, M // 2)
    assert torch.equal(fg.fused_experts_impl(x[half], w1, w2, tw[half], ti[half], **kw), out[half])
