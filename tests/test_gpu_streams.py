"""Calls on another stream than the current one: what a call allocates for itself stays its own until that stream is done with it."""
import numpy as np
import pytest
import torch

from lisa_b200 import ops
from tests import util
from tests.gpu_util import dev_bf16, dev_u32

pytestmark = pytest.mark.gpu

SLEEP = 50_000_000  # clocks of the sleeping kernel: some 30 ms


def _affine(cuda, rng, n, k, bits=4, gs=64, experts=None):
    return [f(a, cuda) for f, a in zip((dev_u32, dev_bf16, dev_bf16), util.affine_weights(rng, n, k, bits, gs, experts=experts))]


def _fill(cuda, nbytes):
    """Takes and overwrites what the current stream's pool has free at this size."""
    return [torch.full((nbytes,), 0xff, dtype=torch.uint8, device=cuda) for _ in range(8)]


def test_swiglu_without_act_keeps_its_scratch_until_the_other_stream_is_done(cuda):
    rng = np.random.default_rng(0)
    m, n, k = 5, 256, 4096
    lin = _affine(cuda, rng, n, k)
    gate, up = (dev_bf16(util.activations(rng, m, k), cuda) for _ in range(2))
    want, _ = ops.quantized_matmul_swiglu(gate, up, *lin)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP)
    y, _ = ops.quantized_matmul_swiglu(gate, up, *lin, stream=side)
    kept = _fill(cuda, m * k * 2)  # (before the side stream has run the call)
    torch.cuda.current_stream().synchronize()
    side.synchronize()
    assert torch.equal(y, want) and len(kept) == 8


def test_workspaces_and_copies_of_the_other_stream(cuda):
    rng = np.random.default_rng(1)
    rows, experts, n, k = 40, 4, 128, 256
    lin = _affine(cuda, rng, n, k, experts=experts)
    wide = dev_bf16(util.activations(rng, rows, 2 * k), cuda)
    x = wide[:, ::2]  # not contiguous: the call copies it
    ids = torch.sort(torch.from_numpy(rng.integers(0, experts, rows))).values.to(cuda)  # int64: copied too
    want = ops.gather_qmm(x, *lin, None, ids, True, 64, 4, True)
    pair = ops.gather_qmm_siblings(x, [lin, lin], ids)
    dense = ops.quantized_matmul(x, *(t[0] for t in lin))
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP)
    got = ops.gather_qmm(x, *lin, None, ids, True, 64, 4, True, stream=side)
    got_pair = ops.gather_qmm_siblings(x, [lin, lin], ids, stream=side.cuda_stream)
    got_dense = ops.quantized_matmul(x, *(t[0] for t in lin), stream=side)
    kept = [_fill(cuda, size) for size in (rows * 16 + 256, rows * k * 2, rows * 4)]
    torch.cuda.current_stream().synchronize()
    side.synchronize()
    assert torch.equal(got, want) and torch.equal(got_dense, dense) and len(kept) == 3
    assert all(torch.equal(a, b) for a, b in zip(got_pair, pair))


def test_outputs_belong_to_the_current_stream(cuda):
    """As before: an output's memory comes from the pool of the caller's stream, whatever stream the call runs on."""
    rng = np.random.default_rng(2)
    lin = _affine(cuda, rng, 128, 256)
    x = dev_bf16(util.activations(rng, 1, 256), cuda)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    y = ops.quantized_matmul(x, *lin, stream=side)
    side.synchronize()
    assert torch.cuda.current_stream() == torch.cuda.default_stream()
    address = y.data_ptr()
    del y
    assert torch.empty((1, 128), dtype=torch.bfloat16, device=cuda).data_ptr() == address


def test_a_launch_that_waits_for_its_stream_lets_other_threads_run(cuda):
    """A stream's queue takes some thousand launches; the next one waits for the GPU.  It waits without the interpreter's lock."""
    import threading
    import time

    rng = np.random.default_rng(3)
    lin = _affine(cuda, rng, 128, 256)
    x = dev_bf16(util.activations(rng, 1, 256), cuda)
    out = ops.quantized_matmul(x, *lin)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(40 * SLEEP)  # about a second

    def fill():
        for _ in range(6000):
            ops.quantized_matmul(x, *lin, out=out, stream=side)

    worker, gap, last = threading.Thread(target=fill), 0.0, time.perf_counter()
    worker.start()
    start = last
    while worker.is_alive():
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
        time.sleep(0)
    side.synchronize()
    took = time.perf_counter() - start
    assert took > 0.4, "the queue took everything: the test shows nothing"
    assert gap < 0.25, f"the other thread stood for {gap:.2f} s of {took:.2f}"
