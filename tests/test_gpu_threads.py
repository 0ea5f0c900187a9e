"""Other Python threads keep running while a launch waits for a place in the device's queue.

The stream is kept busy by a kernel of bounded length and then filled with more launches than the queue holds, so
that the thread that launches is made to wait inside the native call.  A thread that launches for another stream,
or for another rank that this one's work depends on, must be able to run meanwhile."""

import threading
import time

import pytest
import torch

import flaggems_vllm_b200 as fg
from flaggems_vllm_b200 import _lib, testing as T

pytestmark = pytest.mark.gpu
DEV = "cuda"
BUSY_CYCLES = 1_500_000_000  # 0.8 s at 1.9 GHz
LAUNCHES = 4000              # the queue holds about a thousand


def _align():
    ids = T.make_align_ids(8, 2, 8, DEV, seed=1)
    return lambda: fg.moe_align_block_size(ids, 16, 8)


def _router():
    x, w = T.make_activations(2, 256, DEV, seed=1), T.make_half_weights(1, 8, 256, DEV, seed=2)[0]
    return lambda: fg.router_gemm(x, w)


def _grouped():
    logits, bias = T.make_router_inputs(2, 64, DEV, seed=1)
    return lambda: fg.grouped_topk(logits, 8, 4, 4, True, 1.0, bias, 1)


def _topk():
    logits, _ = T.make_router_inputs(2, 8, DEV, seed=1)
    w = torch.empty((2, 2), device=DEV)
    ids, rows = (torch.empty((2, 2), dtype=torch.int32, device=DEV) for _ in range(2))
    return lambda: fg.topk_softmax(w, ids, rows, logits, True)


def _layer():
    x = T.make_activations(2, 256, DEV, seed=1)
    w1 = T.make_half_weights(4, 256, 256, DEV, seed=2)
    w2 = T.make_half_weights(4, 256, 128, DEV, seed=3)
    tw = torch.full((2, 2), 0.5, device=DEV)
    ti = torch.tensor([[0, 1], [2, 3]], dtype=torch.int32, device=DEV)
    return lambda: fg.fused_experts_impl(x, w1, w2, tw, ti)


@pytest.mark.parametrize("make", [_align, _router, _grouped, _topk, _layer])
def test_other_threads_run_while_a_launch_waits_for_the_queue(make):
    call = make()
    for _ in range(3):
        call()
    torch.cuda.synchronize()
    waits = []

    def fill():
        torch.cuda._sleep(BUSY_CYCLES)
        for _ in range(LAUNCHES):
            t = time.perf_counter()
            call()
            waits.append(time.perf_counter() - t)

    worker = threading.Thread(target=fill)
    gap, last = 0.0, time.perf_counter()
    worker.start()
    while worker.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
    worker.join()
    torch.cuda.synchronize()
    assert max(waits) > 0.2, "the queue never filled: this run says nothing"
    # a thread that asks for the lock gets it after one switch interval (5 ms); the queue stays full for longer than 200 ms
    assert gap < 0.1, f"no other thread ran for {gap:.3f} s while a launch waited {max(waits):.3f} s"
    assert _lib.read_status() == 0
