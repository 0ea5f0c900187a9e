"""Failure handling on a real GPU without faulting or hanging it: a bounded wait that is made
to run out sets the status bit and the context stays usable."""

import ctypes

import pytest
import torch

import flaggems_vllm_b200 as fg
from flaggems_vllm_b200 import _lib, fused_moe
from flaggems_vllm_b200 import testing as T

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_a_wait_that_runs_out_sets_the_status_bit_and_the_gpu_still_answers():
    L = _lib.lib()
    dev = torch.device(DEV)
    status = _lib.status_word(dev)
    assert fg.read_status(dev) == 0
    gave_up = torch.zeros(1, dtype=torch.int32, device=dev)
    st = torch.cuda.current_stream().cuda_stream
    # one warp waits 1 ms on a barrier nobody arrives at
    _lib.check(L.moe_debug_wait_timeout(status.data_ptr(), 1_000_000, gave_up.data_ptr(), st))
    torch.cuda.synchronize()
    assert int(gave_up.item()) == 1
    assert fg.read_status(dev) & _lib.ST_WAIT_TIMEOUT
    assert fg.read_status(dev) == 0  # reading cleared it
    # the context is alive: a layer runs and reports nothing
    M, E, H, I, k = 8, 8, 256, 256, 2
    x = T.make_activations(M, H, DEV)
    w1 = T.make_half_weights(E, 2 * I, H, DEV, seed=1, std=H**-0.5)
    w2 = T.make_half_weights(E, H, I, DEV, seed=2, std=I**-0.5)
    logits, _ = T.make_router_inputs(M, E, DEV)
    tw, ti = fg.grouped_topk(torch.softmax(logits, -1), 1, 1, k, True, 1.0, torch.zeros(E, device=DEV), 0)
    out = fg.fused_experts_impl(x, w1, w2, tw.to(torch.bfloat16), ti)
    torch.cuda.synchronize()
    assert torch.isfinite(out.float()).all() and fg.read_status(dev) == 0


def test_wait_limit_setter_round_trip():
    L = _lib.lib()
    old = L.moe_set_wait_limit_ns(0)
    assert old > 0
    assert L.moe_set_wait_limit_ns(5_000_000) == old
    assert L.moe_set_wait_limit_ns(old) == 5_000_000
    assert L.moe_set_wait_limit_ns(0) == old


def test_status_check_mode_raises(monkeypatch):
    """FLAGGEMS_B200_CHECK_STATUS=1: the layer reads the status word and raises when a kernel reported a problem."""
    monkeypatch.setenv("FLAGGEMS_B200_CHECK_STATUS", "1")
    M, E, H, I, k = 8, 8, 256, 256, 2
    x = T.make_activations(M, H, DEV)
    w1 = T.make_half_weights(E, 2 * I, H, DEV, seed=1, std=H**-0.5)
    w2 = T.make_half_weights(E, H, I, DEV, seed=2, std=I**-0.5)
    logits, _ = T.make_router_inputs(M, E, DEV)
    tw, ti = fg.grouped_topk(torch.softmax(logits, -1), 1, 1, k, True, 1.0, torch.zeros(E, device=DEV), 0)
    fg.fused_experts_impl(x, w1, w2, tw.to(torch.bfloat16), ti)  # clean: no exception
    bad = ti.clone()
    bad[0, 0] = E + 3  # an expert id outside the table: skipped by align, reported in the status word
    with pytest.raises(fg.MoeKernelError, match="status word"):
        fg.fused_experts_impl(x, w1, w2, tw.to(torch.bfloat16), bad)
    assert fg.read_status() == 0


class _GuardedAllocator:
    """Stands in for torch.empty inside the layer: every workspace sits between two guard bands
    filled with a byte pattern, so a kernel that writes outside its buffer is caught."""

    GUARD = 4096  # bytes on either side (keeps the 16-byte / 1024-byte alignments the kernels ask for)
    PATTERN = 0xA5

    def __init__(self):
        self.real_empty = torch.empty
        self.blocks = []

    def __call__(self, *size, dtype=None, device=None, **kw):
        if len(size) == 1 and not isinstance(size[0], int):
            size = tuple(size[0])
        dtype = dtype or torch.get_default_dtype()
        if device is None or torch.device(device).type != "cuda" or kw:
            return self.real_empty(tuple(size), dtype=dtype, device=device, **kw)
        n = 1
        for s in size:
            n *= int(s)
        nbytes = n * self.real_empty((), dtype=dtype).element_size()
        padded = (nbytes + 255) // 256 * 256
        whole = torch.full((padded + 2 * self.GUARD,), self.PATTERN, dtype=torch.uint8, device=device)
        self.blocks.append((whole, padded))
        return whole[self.GUARD:self.GUARD + nbytes].view(dtype).view(size)

    def check(self):
        assert self.blocks, "no workspace was allocated through the guarded allocator"
        for whole, padded in self.blocks:
            lo, hi = whole[:self.GUARD], whole[self.GUARD + padded:]
            assert bool((lo == self.PATTERN).all()) and bool((hi == self.PATTERN).all()), \
                f"a kernel wrote outside a {padded}-byte workspace"
        return len(self.blocks)


_MODES = {"bf16": _lib.MODE_HALF, "fp8": _lib.MODE_FP8_BLOCK, "w8a16": _lib.MODE_W8A16, "fp8_row": _lib.MODE_FP8_ROW,
          "int8_row": _lib.MODE_INT8_ROW}


def _layer_inputs(mode, M):
    E, H, I, k = 8, 512, 512, 2
    x = T.make_activations(M, H, DEV, seed=M)
    logits, _ = T.make_router_inputs(M, E, DEV, seed=M + 1)
    tw, ti = fg.grouped_topk(torch.softmax(logits, -1), 1, 1, k, True, 1.0, torch.zeros(E, device=DEV), 0)
    if mode == "bf16":
        w1 = T.make_half_weights(E, 2 * I, H, DEV, seed=1, std=H**-0.5)
        w2 = T.make_half_weights(E, H, I, DEV, seed=2, std=I**-0.5)
        return x, w1, w2, tw, ti, None, None
    if mode == "fp8":
        w1, s1 = T.make_fp8_block_weights(E, 2 * I, H, DEV, seed=1)
        w2, s2 = T.make_fp8_block_weights(E, H, I, DEV, seed=2)
        return x, w1, w2, tw, ti, s1, s2
    w1, s1 = T.make_int8_channel_weights(E, 2 * I, H, DEV, seed=1)
    w2, s2 = T.make_int8_channel_weights(E, H, I, DEV, seed=2)
    if mode == "fp8_row":
        w1, w2 = w1.to(torch.float8_e4m3fn), w2.to(torch.float8_e4m3fn)
    return x, w1, w2, tw, ti, s1, s2


@pytest.mark.parametrize("mode", ["bf16", "fp8", "w8a16"])
@pytest.mark.parametrize("M", [1, 5, 200, 1500])
def test_guard_bands_around_every_workspace_stay_intact(monkeypatch, mode, M):
    """The staged pipeline: all its buffers (sorted ids, expert ids, quantised rows and scales, the
    sorted copies, the intermediate, y, the row index, split-K partial sums) are allocated with guard
    bands on both sides; after the layer every band still holds its pattern.  The sizes cover the
    small-batch schedule, the 128-row kernels with row stores and the staged TMA output."""
    x, w1, w2, tw, ti, s1, s2 = _layer_inputs(mode, M)
    ref, out = torch.empty_like(x), torch.empty_like(x)

    def staged(result):
        fused_moe.run_chunk(x, w1, w2, tw, ti, result, mode=_MODES[mode], w1_scale=s1, w2_scale=s2,
                            global_num_experts=w1.shape[0], expert_map=None, apply_router_weight_on_input=False, keep={})

    staged(ref)
    guard = _GuardedAllocator()
    monkeypatch.setattr(torch, "empty", guard)
    try:
        staged(out)
        torch.cuda.synchronize()
    finally:
        monkeypatch.undo()
    assert guard.check() >= 4
    assert torch.equal(out, ref) and fg.read_status(torch.device(DEV)) == 0


def _native_layer(mode, M, weight_on_input, fill, stages=63):
    """moe_layer on workspaces of the test's own, every byte of them `fill` before: (out, workspaces, pieces)."""
    x, w1, w2, tw, ti, s1, s2 = _layer_inputs(mode, M)
    (E, N, H), k, band = w1.shape, ti.shape[1], _GuardedAllocator.GUARD
    sizes = (_MODES[mode], _lib.dtype_code(x.dtype), M, k, E, E, H, N // 2, _lib.ACT_SILU)
    need, table = (ctypes.c_int64 * 4)(), (ctypes.c_int64 * (3 * 13))()
    _lib.check(_lib.lib().moe_layer_layout(*sizes, ctypes.addressof(need), ctypes.addressof(table)))
    pieces = [(table[3 * i], band + table[3 * i + 1], table[3 * i + 2]) for i in range(13)]
    ws = [torch.full((n + 2 * band,), fill, dtype=torch.uint8, device=DEV) for n in need]
    out = torch.empty_like(x)
    kind = 1 if mode == "fp8_row" else 0
    _lib.check(_lib.lib().moe_layer(
        sizes[0], sizes[1], x.data_ptr(), M, k, ti.data_ptr(), 0, tw.data_ptr(), w1.data_ptr(), _lib.ptr(s1), w2.data_ptr(),
        _lib.ptr(s2), out.data_ptr(), E, None, E, H, N // 2, int(weight_on_input), _lib.ACT_SILU, 0.0, 0.0, 0.0, kind, None, kind,
        None, *[w.data_ptr() + band for w in ws], stages, _lib.status_word(DEV).data_ptr(), _lib.stream_of(x)))
    torch.cuda.synchronize()
    return out, ws, pieces


@pytest.mark.parametrize("mode", list(_MODES))
@pytest.mark.parametrize("M", [1, 5, 200, 1500])
@pytest.mark.parametrize("weight_on_input", [False, True])
def test_gaps_between_the_buffers_of_the_layer_call_stay_intact(mode, M, weight_on_input):
    """The layer call keeps its buffers in four workspaces.  Every byte outside the buffers, 256 or more behind
    each and 4 KB around the workspaces, still holds its pattern afterwards, and what the workspaces held before changes no
    result.  The sizes cover the few-route plan and split-K schedule, occupied rows only, whole blocks and staged stores."""
    out, ws, pieces = _native_layer(mode, M, weight_on_input, _GuardedAllocator.PATTERN)
    for i, w in enumerate(ws):
        outside = torch.ones(w.numel(), dtype=torch.bool, device=DEV)
        used = [(at, n) for at_ws, at, n in pieces if at_ws == i and n > 0]
        assert used and all(at % 256 == 0 for at, _ in used)
        for at, n in used:
            assert bool(outside[at:at + n].all()), "pieces overlap"
            outside[at:at + n] = False
        for at, n in used:
            assert bool(outside[at + n:at + n + 256].all()), "no gap behind a piece"
        assert bool((w[outside] == _GuardedAllocator.PATTERN).all()), f"a kernel wrote outside its buffer in workspace {i}"
    assert torch.equal(out, _native_layer(mode, M, weight_on_input, 0xFF)[0])  # 0xFF: NaN in every float type
    assert torch.isfinite(out).all() and fg.read_status(torch.device(DEV)) == 0


@pytest.mark.parametrize("M", [600, 1500])
def test_padding_rows_are_zero_whatever_the_workspaces_held(M):
    """From 128 rows per expert on, the FP8 GEMMs multiply whole blocks: the padding rows of both operands are zeros,
    with finite scales, although every byte of the workspaces was 0xFF (NaN) before."""
    _, ws, pieces = _native_layer("fp8", M, False, 0xFF, stages=1 | 2 | 4)
    view = lambda i, t: ws[pieces[i][0]][pieces[i][1]:pieces[i][1] + pieces[i][2]].view(t)
    H = I = 512
    x_rows, act = view(5, torch.uint8).view(-1, H), view(8, torch.uint8).view(-1, I)
    x_scales, act_scales = (view(i, torch.float32).view(4, -1) for i in (6, 10))
    tiles = view(1, torch.int32).view(-1, 4)[:int(view(2, torch.int32)[0])].tolist()
    padding = [r for row0, n, _, _ in tiles for r in range(row0 + (n >> 16), row0 + (n & 0xFFFF))]
    assert len(padding) > 8
    assert bool((x_rows[padding] == 0).all()) and bool((x_scales[:, padding] == 0).all())
    assert bool(((act[padding] & 0x7F) == 0).all()) and bool(torch.isfinite(act_scales[:, padding]).all())
