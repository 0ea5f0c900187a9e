"""CPU-only checks: the C-ABI library loads and exports every declared symbol,
the Python entry points keep the reference's signatures, argument validation
raises the reference's error types before any device work."""

import ctypes
import inspect
import os
import re

import pytest
import torch

import flaggems_vllm
import flaggems_vllm_b200 as fg
from flaggems_vllm_b200 import _lib, build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_builds_and_exports_every_declared_symbol():
    path = build.build()
    handle = ctypes.CDLL(path)
    header = open(os.path.join(ROOT, "include", "moe_sm100.h")).read()
    declared = set(re.findall(r"^(?:int|unsigned long long|const char\*)\s+(moe_[a-z0-9_]+)\s*\(", header, flags=re.M))
    assert declared, "no declarations found in the header"
    for name in declared:
        assert hasattr(handle, name), f"{name} declared in the header but not exported"
    assert declared == set(_lib.SYMBOLS), "ctypes table and header disagree"
    assert handle.moe_abi_version() >= 1


def test_a_refused_call_counts_no_launch():
    before = _lib.LAUNCHES
    assert _lib.lib().moe_align_block_size(None, 0, 4, 8, 16, None, 64, None, 4, None, None, None) != 0
    assert _lib.lib().moe_layer_workspace(_lib.MODE_HALF, _lib.MOE_BF16, 0, 2, 8, 8, 512, 512, 0, None) != 0
    assert _lib.LAUNCHES == before


def _sig(fn):
    return [(n, p.kind, p.default) for n, p in inspect.signature(fn).parameters.items()]


def test_signatures_match_reference():
    # names, order, kinds and defaults of src/flaggems_vllm/ops/grouped_topk.py:1674-1684
    assert _sig(fg.grouped_topk) == [
        ("scores", inspect.Parameter.POSITIONAL_OR_KEYWORD, inspect._empty),
        ("n_group", inspect.Parameter.POSITIONAL_OR_KEYWORD, inspect._empty),
        ("topk_group", inspect.Parameter.POSITIONAL_OR_KEYWORD, inspect._empty),
        ("topk", inspect.Parameter.POSITIONAL_OR_KEYWORD, inspect._empty),
        ("renormalize", inspect.Parameter.POSITIONAL_OR_KEYWORD, inspect._empty),
        ("routed_scaling_factor", inspect.Parameter.POSITIONAL_OR_KEYWORD, inspect._empty),
        ("bias", inspect.Parameter.POSITIONAL_OR_KEYWORD, inspect._empty),
        ("scoring_func", inspect.Parameter.POSITIONAL_OR_KEYWORD, 0),
        ("is_padding", inspect.Parameter.POSITIONAL_OR_KEYWORD, None),
    ]
    # src/flaggems_vllm/ops/moe_align_block_size.py:896-902
    assert [(n, d) for n, _, d in _sig(fg.moe_align_block_size)] == [
        ("topk_ids", inspect._empty), ("block_size", inspect._empty), ("num_experts", inspect._empty),
        ("expert_map", None), ("pad_sorted_ids", False)]
    # src/flaggems_vllm/ops/fused_moe.py:2314-2344
    names = [n for n, _, _ in _sig(fg.fused_experts_impl)]
    assert names == [
        "hidden_states", "w1", "w2", "topk_weights", "topk_ids", "inplace", "activation",
        "apply_router_weight_on_input", "use_fp8_w8a8", "use_int8_w8a8", "use_int8_w8a16", "use_int4_w4a16",
        "ocp_mx_scheme", "per_channel_quant", "global_num_experts", "expert_map", "w1_scale", "w2_scale",
        "w1_zp", "w2_zp", "a1_scale", "a2_scale", "block_shape", "w1_bias", "w2_bias", "gemm1_alpha",
        "gemm1_beta", "gemm1_clamp_limit"]
    kinds = [k for _, k, _ in _sig(fg.fused_experts_impl)]
    assert kinds[:25] == [inspect.Parameter.POSITIONAL_OR_KEYWORD] * 25
    assert kinds[25:] == [inspect.Parameter.KEYWORD_ONLY] * 3
    assert inspect.signature(fg.fused_experts_impl).parameters["global_num_experts"].default == -1
    assert fg.ops_experts_impl is fg.fused_experts_impl
    assert flaggems_vllm.grouped_topk is fg.grouped_topk
    assert flaggems_vllm.ops_experts_impl is fg.fused_experts_impl
    assert "inplace" not in inspect.signature(fg.inplace_fused_experts).parameters
    # src/flaggems_vllm/ops/router_gemm.py:207, src/flaggems_vllm/ops/fp32_router_gemm.py:17,143
    assert [n for n, _, _ in _sig(fg.router_gemm)] == ["x", "weight"]
    assert [n for n, _, _ in _sig(fg.fp32_router_gemm)] == ["input", "router_weight"]
    assert [n for n, _, _ in _sig(fg.supports_fp32_router_gemm)] == [
        "hidden_size", "num_experts", "input_dtype", "weight_dtype"]
    assert flaggems_vllm.router_gemm is fg.router_gemm


_KIND = {inspect.Parameter.POSITIONAL_OR_KEYWORD: "positional", inspect.Parameter.POSITIONAL_ONLY: "positional",
         inspect.Parameter.KEYWORD_ONLY: "keyword_only", inspect.Parameter.VAR_POSITIONAL: "var_positional",
         inspect.Parameter.VAR_KEYWORD: "var_keyword"}


def test_signatures_match_the_reference_source():
    """Names, order, kinds and defaults of every public function of the path, against
    tests/golden/signatures.json, which tests/golden/make_signatures.py reads from the
    reference's source with ast."""
    import json

    with open(os.path.join(ROOT, "tests", "golden", "signatures.json")) as fh:
        ref = json.load(fh)
    assert len(ref) >= 14
    for name, info in ref.items():
        ours = [[n, _KIND[p.kind], None if p.default is inspect._empty else repr(p.default)]
                for n, p in inspect.signature(getattr(fg, name)).parameters.items()]
        assert ours == info["params"], f"{name} differs from {info['source']}"
        assert getattr(flaggems_vllm, name) is getattr(fg, name)


def test_grouped_topk_validation_errors():
    s = torch.zeros(4, 16)
    b = torch.zeros(16)
    with pytest.raises(ValueError, match="2D"):
        fg.grouped_topk(torch.zeros(16), 1, 1, 2, True, 1.0, b)
    with pytest.raises(ValueError, match="divisible"):
        fg.grouped_topk(s, 3, 1, 2, True, 1.0, b)
    with pytest.raises(ValueError, match="n_group"):
        fg.grouped_topk(torch.zeros(4, 64), 64, 1, 2, True, 1.0, torch.zeros(64))
    with pytest.raises(ValueError, match="topk"):
        fg.grouped_topk(torch.zeros(4, 64), 1, 1, 33, True, 1.0, torch.zeros(64))
    with pytest.raises(ValueError, match="scoring_func"):
        fg.grouped_topk(s, 1, 1, 2, True, 1.0, b, 2)
    with pytest.raises(ValueError, match="bias length"):
        fg.grouped_topk(s, 1, 1, 2, True, 1.0, torch.zeros(8))
    with pytest.raises(ValueError, match="Unsupported dtype"):
        fg.grouped_topk(s.double(), 1, 1, 2, True, 1.0, b)
    with pytest.raises(RuntimeError, match="no CPU path"):
        fg.grouped_topk(s, 1, 1, 2, True, 1.0, b)  # valid arguments, CPU tensors


def test_fused_experts_validation_errors():
    x = torch.zeros(4, 64, dtype=torch.bfloat16)
    w1 = torch.zeros(2, 256, 64, dtype=torch.bfloat16)
    w2 = torch.zeros(2, 64, 128, dtype=torch.bfloat16)
    tw = torch.zeros(4, 2)
    ti = torch.zeros(4, 2, dtype=torch.int32)
    with pytest.raises(ValueError, match="Unknown MoE activation"):
        fg.fused_experts_impl(x, w1, w2, tw, ti, activation="tanh")
    with pytest.raises(ValueError, match="Only 'silu'"):
        fg.fused_experts_impl(x, w1, w2, tw, ti, activation="gelu")
    with pytest.raises(ValueError, match="require swigluoai"):
        fg.fused_experts_impl(x, w1, w2, tw, ti, gemm1_alpha=1.0)
    with pytest.raises(NotImplementedError):
        fg.fused_experts_impl(x, w1, w2, tw, ti, ocp_mx_scheme="w_bogus")
    with pytest.raises(AssertionError, match="Hidden size mismatch"):
        fg.fused_experts_impl(torch.zeros(4, 32, dtype=torch.bfloat16), w1, w2, tw, ti)
    with pytest.raises(AssertionError, match="topk shape"):
        fg.fused_experts_impl(x, w1, w2, torch.zeros(4, 3), ti)
    with pytest.raises(AssertionError, match="contiguous"):
        fg.fused_experts_impl(torch.zeros(64, 4, dtype=torch.bfloat16).t(), w1, w2, tw, ti)
    with pytest.raises(AssertionError, match="weights expected"):
        fg.fused_experts_impl(x, w1, w2, tw, ti, use_int8_w8a8=True)  # bf16 weights are not int8 weights
    with pytest.raises(NotImplementedError, match="block-quantised INT8"):
        fg.fused_experts_impl(x, w1.to(torch.int8), w2.to(torch.int8), tw, ti, use_int8_w8a8=True, block_shape=[128, 128])
    with pytest.raises(NotImplementedError, match="block_shape"):
        fg.fused_experts_impl(x, w1, w2, tw, ti, use_fp8_w8a8=True, block_shape=[64, 64])
    with pytest.raises(ValueError, match="finite scalar gemm1_alpha"):
        fg.fused_experts_impl(x, w1, w2, tw, ti, activation="swigluoai_uninterleave")
    with pytest.raises(ValueError, match="gemm1_clamp_limit >= 0"):
        fg.fused_experts_impl(x, w1, w2, tw, ti, activation="swigluoai_uninterleave", gemm1_alpha=1.702,
                              gemm1_beta=1.0, gemm1_clamp_limit=-1.0)
    with pytest.raises(RuntimeError, match="no CPU path"):
        fg.fused_experts_impl(x, w1, w2, tw, ti)


def test_router_gemm_validation_errors():
    x, w = torch.zeros(2, 16, dtype=torch.bfloat16), torch.zeros(4, 16, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="2D"):
        fg.router_gemm(x[0], w)
    with pytest.raises(ValueError, match="shape"):
        fg.router_gemm(x, w[:, :8])
    with pytest.raises(ValueError, match="CUDA device"):
        fg.fp32_router_gemm(x, w.float())
    assert fg.supports_fp32_router_gemm(6144, 128, torch.bfloat16, torch.float32)
    assert not fg.supports_fp32_router_gemm(7168, 256, torch.bfloat16, torch.float32)
    assert not fg.supports_fp32_router_gemm(6144, 128, torch.bfloat16, torch.bfloat16)


def test_align_rejects_cpu_tensors_and_bad_dtypes():
    with pytest.raises(RuntimeError, match="no CPU path"):
        fg.moe_align_block_size(torch.zeros(4, 2, dtype=torch.int32), 16, 8)


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", str(tmp_path / "nope.so"))
    with pytest.raises(RuntimeError, match="no CPU or Triton fallback"):
        _lib.lib()


def test_product_package_never_imports_the_oracle():
    pkg = os.path.join(ROOT, "flaggems_vllm_b200")
    for fn in os.listdir(pkg):
        if fn.endswith(".py"):
            src = open(os.path.join(pkg, fn)).read()
            assert "oracle" not in src, f"{fn} mentions the oracle"


def test_small_batch_slice_count_model():
    """The K-slice count asked of the small-batch GEMMs: never below what one unit can hold, never
    above 16, and the choices the measurements were taken with."""
    from flaggems_vllm_b200 import fused_moe

    H, I = 4096, 14336  # one token of the Mixtral shape: two experts
    assert fused_moe.small_k_slices(_lib.MODE_HALF, True, H, I, 2, 148) == 2      # 896 units, 7 per CTA at most
    assert fused_moe.small_k_slices(_lib.MODE_HALF, False, I, H, 2, 148) == 9     # 576 units: four full waves
    assert fused_moe.small_k_slices(_lib.MODE_W8A16, True, 2048, 768, 8, 148) == 1  # 96 units fit one wave
    for mode in (_lib.MODE_HALF, _lib.MODE_FP8_BLOCK, _lib.MODE_W8A16):
        for K in (128, 512, 2048, 7168, 14336):
            for blocks in (1, 2, 8, 64):
                for gemm1 in (True, False):
                    S = fused_moe.small_k_slices(mode, gemm1, K, 1024, blocks, 148)
                    chunks = K // (64 if mode == _lib.MODE_HALF else 128)
                    need = -(-chunks // (16 if mode == _lib.MODE_W8A16 else 32))
                    assert 1 <= S <= 16 and (S >= need or need > 16) and S <= max(chunks, 1)


@pytest.mark.parametrize("sms,largest", [(148, 8), (148, 4), (70, 8), (32, 2), (16, 1)])
def test_router_tile_keeps_to_the_clusters_of_the_device(sms, largest):
    columns, split = ctypes.c_int(), ctypes.c_int()
    for M in (5, 64, 200, 1000, 8192):
        for N, K in ((8, 4096), (33, 72), (128, 2048), (256, 7168), (1024, 512)):
            _lib.check(_lib.lib().moe_router_gemm_tile(M, N, K, sms, largest, ctypes.addressof(columns), ctypes.addressof(split)))
            assert columns.value in (32, 64, 128, 256) and 1 <= split.value <= min(largest, -(-K // 64))
    _lib.check(_lib.lib().moe_router_gemm_tile(200, 256, 7168, sms, largest, ctypes.addressof(columns), ctypes.addressof(split)))
    assert split.value == largest  # a small product wants every SM it can get
    assert _lib.lib().moe_router_gemm_tile(200, 256, 7168, 0, 8, ctypes.addressof(columns), ctypes.addressof(split)) != 0


def test_kernel_choice_at_the_benchmark_configurations(monkeypatch):
    """Host policy (no device work): which schedule serves the configurations of the benchmark plan."""
    from flaggems_vllm_b200 import fused_moe as fm

    for var in ("FLAGGEMS_B200_GENERIC_GEMM", "FLAGGEMS_B200_TC_WIDE", "FLAGGEMS_B200_TC_PAIR", "FLAGGEMS_B200_TC_PAIR_WIDE",
                "FLAGGEMS_B200_PRESORT", "FLAGGEMS_B200_TMA_OUT", "FLAGGEMS_B200_SMALL_M"):
        monkeypatch.delenv(var, raising=False)
    bf16 = torch.bfloat16
    # DeepSeek-V3 shape, FP8 block scales: always the 128-row tcgen05 kernel, never the small-batch schedule
    for M in (1, 32, 128, 1024, 8192):
        numel = M * 8
        assert fm._choose_kernel(_lib.MODE_FP8_BLOCK, bf16, 7168, 2048, numel, 256) == fm.KERNEL_TC
        assert not fm._use_small_path(_lib.MODE_FP8_BLOCK, bf16, 7168, 2048, numel, 8)
        assert fm._presort_rows(_lib.MODE_FP8_BLOCK, fm.KERNEL_TC, numel, 256) == (M >= 4096)
        assert fm._sorted_output(_lib.MODE_FP8_BLOCK, fm.KERNEL_TC, numel, 256) == (M >= 2048)
    # Mixtral shape, bf16: small-batch schedule up to 8 routes, the 256x256 tile from 256 rows per expert on
    assert fm._use_small_path(_lib.MODE_HALF, bf16, 4096, 14336, 2, 2)
    assert not fm._use_small_path(_lib.MODE_HALF, bf16, 4096, 14336, 32, 2)
    assert fm._choose_kernel(_lib.MODE_HALF, bf16, 4096, 14336, 512, 8) == fm.KERNEL_TC
    assert fm._choose_kernel(_lib.MODE_HALF, bf16, 4096, 14336, 2048, 8) == fm.KERNEL_TC_WIDE
    assert not fm._sorted_output(_lib.MODE_HALF, fm.KERNEL_TC_WIDE, 8192, 8)
    # Qwen3 shape, weight-only int8: small-batch schedule up to 16 routes, the converter kernel beyond
    assert fm._use_small_path(_lib.MODE_W8A16, bf16, 2048, 768, 8, 8)
    assert not fm._use_small_path(_lib.MODE_W8A16, bf16, 2048, 768, 512, 8)
    assert fm._choose_kernel(_lib.MODE_W8A16, bf16, 2048, 768, 32768, 128) == fm.KERNEL_TC
    # shapes the tensor-core kernels do not serve fall to the generic kernel; the switches override
    assert fm._choose_kernel(_lib.MODE_HALF, torch.float32, 4096, 14336, 2048, 8) == fm.KERNEL_GENERIC
    assert fm._choose_kernel(_lib.MODE_FP8_BLOCK, bf16, 7168 + 64, 2048, 64, 256) == fm.KERNEL_GENERIC
    monkeypatch.setenv("FLAGGEMS_B200_TC_PAIR", "1")
    assert fm._choose_kernel(_lib.MODE_FP8_BLOCK, bf16, 7168, 2048, 65536, 256) == fm.KERNEL_TC_PAIR
    monkeypatch.setenv("FLAGGEMS_B200_GENERIC_GEMM", "1")
    assert fm._choose_kernel(_lib.MODE_FP8_BLOCK, bf16, 7168, 2048, 65536, 256) == fm.KERNEL_GENERIC


@pytest.mark.parametrize("mode", [_lib.MODE_HALF, _lib.MODE_FP8_BLOCK, _lib.MODE_W8A16, _lib.MODE_FP8_ROW, _lib.MODE_INT8_ROW])
@pytest.mark.parametrize("tokens", [1, 40, 1500])
def test_layer_buffers_lie_apart(mode, tokens):
    """Buffers of the layer call share four workspaces: aligned, inside them, at least 256 bytes between neighbours."""
    need, table = (ctypes.c_int64 * 4)(), (ctypes.c_int64 * 39)()
    _lib.check(_lib.lib().moe_layer_layout(mode, _lib.MOE_BF16, tokens, 2, 8, 8, 512, 512, _lib.ACT_SILU,
                                           ctypes.addressof(need), ctypes.addressof(table)))
    for ws in range(4):
        used = sorted((table[i + 1], table[i + 2]) for i in range(0, 39, 3) if table[i] == ws and table[i + 2] > 0)
        assert used
        for (at, n), (after, _) in zip(used, used[1:] + [(need[ws], 0)]):
            assert at % 256 == 0 and at + n + 256 <= after


@pytest.mark.parametrize("tokens,topk,experts,served", [
    (32768, 8, 256, True), (32769, 8, 256, False), (32768, 9, 256, False), (65535, 4, 256, True), (65536, 1, 256, False),
    (4096, 8, 1024, True), (4096, 8, 1025, False), (8, 32, 64, True), (8, 33, 64, False)])
def test_layer_call_serves_what_its_declaration_says(tokens, topk, experts, served):
    need = (ctypes.c_int64 * 4)()
    for mode in (_lib.MODE_HALF, _lib.MODE_FP8_BLOCK, _lib.MODE_W8A16, _lib.MODE_FP8_ROW, _lib.MODE_INT8_ROW):
        rc = _lib.lib().moe_layer_workspace(mode, _lib.MOE_BF16, tokens, topk, experts, experts, 256, 128, _lib.ACT_SILU,
                                            ctypes.addressof(need))
        assert (rc == 0) == served


def _layer_pieces(mode, tokens, topk, E, H, I, act=_lib.ACT_SILU):
    need, table = (ctypes.c_int64 * 4)(), (ctypes.c_int64 * 39)()
    _lib.check(_lib.lib().moe_layer_layout(mode, _lib.MOE_BF16, tokens, topk, E, E, H, I, act, ctypes.addressof(need),
                                           ctypes.addressof(table)))
    return [table[i + 2] for i in range(0, 39, 3)]


@pytest.mark.parametrize("tokens,topk,E,H,I,split", [
    (1, 2, 8, 4096, 14336, True), (2, 2, 8, 4096, 14336, False),                                   # 0.70 GB, 1.41 GB
    (1, 1, 16, 5120, 8192, True), (3, 1, 16, 5120, 8192, True), (4, 1, 16, 5120, 8192, False),     # 0.25, 0.75, 1.01 GB
    (1, 6, 64, 2048, 1408, True), (3, 2, 8, 2048, 4096, True), (4, 2, 8, 2048, 4096, True),
    (8, 1, 8, 256, 128, True), (9, 1, 8, 256, 128, False), (1, 8, 128, 2048, 768, True)])
def test_few_routes_of_half_precision_keep_k_slices_summed_in_fp32(tokens, topk, E, H, I, split):
    """Up to eight routes and 1 GB of weights: the schedule that adds its K slices' sums in fp32 (only it has counters)."""
    assert (_layer_pieces(_lib.MODE_HALF, tokens, topk, E, H, I)[12] > 0) == split


def test_warps_agree_on_a_wait_before_they_act_as_one():
    """A bounded wait gives up by the clock, and lanes may read it on either side of the limit.  Where a warp goes on with
    instructions that it executes as one (tensor memory, mma.sync, barriers), the lanes vote on the answer first."""
    csrc = os.path.join(ROOT, "flaggems_vllm_b200", "csrc")
    # barriers that consumers, converters and epilogues wait for; the issuing warps wait for others
    waits = {"gemm_tc.cu": ("tmem_full", "acc_full", "xch_bar"), "gemm_wt.cu": ("tmem_full",), "gemm_w8t.cu": ("tmem_full", "r_full", r"done\[s\]\), ph,"),
             "gemm_w8.cu": ("tmem_full", "r_full", "b_empty"), "router_gemm.cu": ("done",)}
    for name, barriers in waits.items():
        lines = open(os.path.join(csrc, name)).read().split("\n")
        for barrier in barriers:
            found = [i for i, line in enumerate(lines) if re.search(r"mbar_wait\w*(<\w+>)?\([^;]*\b" + barrier, line)]
            assert found, (name, barrier)
            for i in found:
                voted = "warp_agrees(mbar_wait" in lines[i] or "warp_agrees(ready)" in lines[i + 1]
                assert voted, f"{name}:{i + 1}: {lines[i].strip()}"
    # a warp that has given up still meets the others at the named barriers of the tiles and units that are left; the split-K
    # kernel's lanes go on without waiting
    tc, small = (open(os.path.join(csrc, n)).read() for n in ("gemm_tc.cu", "gemm_small.cu"))
    assert "(alive || TMAOUT); tile += tile_step" in tc and "for (int u = u_begin; u < u_end; ++u)" in small
    assert "if (alive) alive = mbar_wait(&aux->full[st]" in small


@pytest.mark.parametrize("mode,act,E,topk,tokens,tile", [
    # half precision: 64-row tiles while no expert can have more than two of them, 256 beyond 100 rows per expert
    ("half", "silu", 8, 2, 100, 64), ("half", "silu", 8, 2, 128, 64), ("half", "silu", 8, 2, 129, 128), ("half", "silu", 4, 2, 65, 64),
    ("half", "silu", 4, 2, 66, 128), ("half", "silu", 64, 6, 128, 64), ("half", "silu", 64, 6, 129, 128), ("half", "silu", 8, 2, 403, 128),
    ("half", "silu", 8, 2, 404, 256), ("half", "silu", 8, 2, 16384, 256),
    ("half", "swigluoai", 8, 2, 9, 128), ("half", "swigluoai", 8, 2, 259, 128), ("half", "swigluoai", 8, 2, 260, 256),
    ("fp8_row", "silu", 128, 8, 33, 128), ("fp8_row", "silu", 128, 8, 1039, 128), ("fp8_row", "silu", 128, 8, 1040, 256),
    ("int8_row", "silu", 128, 8, 1039, 128), ("int8_row", "silu", 128, 8, 1040, 256),
    ("fp8_row", "swigluoai", 128, 8, 100, 256), ("int8_row", "swigluoai", 128, 8, 1500, 256)])
def test_pair_tiles_where_their_lines_lie(mode, act, E, topk, tokens, tile):
    """The lines that hold under skewed routing, which the host cannot see: read from the room for tiles in the plan."""
    code = {"half": _lib.MODE_HALF, "fp8_row": _lib.MODE_FP8_ROW, "int8_row": _lib.MODE_INT8_ROW}[mode]
    H = 512
    pieces = _layer_pieces(code, tokens, topk, E, H, 256, _lib.ACT_SILU if act == "silu" else _lib.ACT_SWIGLUOAI)
    rows, used = pieces[11] // (2 * H), min(tokens * topk, E)
    assert {t for t in (64, 128, 256) if rows // t + used + 1 == pieces[1] // 16} == {tile}
