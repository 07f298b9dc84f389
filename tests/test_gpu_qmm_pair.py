"""The prefill GEMM on pairs of SMs (qmm_pair.cu) against the oracle, at the edges of its tiling: pairs that share a tile's k, token tiles of every
kind, outputs that are stored row by row, groups that do not fill a k-block, tables with an empty tail, the GGUF form."""
import numpy as np
import pytest
import torch

from lisa_b200 import ops
from oracle import oracle as O
from tests import util
from tests.gpu_util import dev_bf16, dev_f32, dev_i32, dev_u8, dev_u32, host_bf16_bits

pytestmark = pytest.mark.gpu

TOL = 1e-2


# two, three and four pairs a tile (few tiles of much k); one pair with a token tile above 256 and a ragged second one; odd rows (2-byte stores);
# an odd number of groups of 32; k that ends inside a k-block, inside a packed stage, in the first half of a k-block
@pytest.mark.parametrize("ns,k,m,bits,gs", [
    ((7000,), 2560, 9, 4, 64), ((1032,), 2048, 300, 4, 64), ((4100,), 4096, 100, 4, 64), ((4096,), 4096, 16, 2, 64), ((256,), 4096, 16, 4, 64), ((2000,), 9728, 40, 4, 128),
    ((1001,), 4096, 33, 4, 64), ((18944,), 128, 290, 4, 64), ((18001,), 192, 301, 2, 64), ((129,), 1056, 50, 4, 32), ((77,), 1120, 270, 4, 32), ((257, 3, 1000), 320, 65, 4, 64),
    ((512, 511), 2048, 31, 2, 128), ((300,), 96, 9, 4, 32)])
def test_edges(cuda, ns, k, m, bits, gs):
    rng = np.random.default_rng(sum(ns) + k + m)
    x = util.activations(rng, m, k)
    host = [util.affine_weights(rng, n, k, bits, gs) for n in ns]
    dev = [(dev_u32(w, cuda), dev_bf16(s, cuda), dev_bf16(b, cuda)) for w, s, b in host]
    launches = ops.launch_count()
    ys = ops.quantized_matmul_siblings(dev_bf16(x, cuda), dev, True, gs, bits) if len(ns) > 1 else [ops.quantized_matmul(dev_bf16(x, cuda), *dev[0], True, gs, bits)]
    assert ops.launch_count() - launches == 1
    for n, (w, s, b), y in zip(ns, host, ys):
        rows = np.unique(np.concatenate([np.arange(min(n, 3)), np.arange(max(n - 3, 0), n), rng.integers(0, n, 64), np.array([r for r in (127, 128, 255, 256) if r < n], dtype=int)]))
        truth = O.affine_matmul(x, *(np.ascontiguousarray(a[rows]) for a in (w, s, b)), gs, bits, round_weight_bf16=True, f64=True)
        err, l2 = util.parity(O.bf16_to_f32(host_bf16_bits(y))[:, rows], truth)
        assert err <= TOL and l2 <= 3e-3, (n, err, l2)
    assert ops.device_status() == 0


# runs of every length in one table (none, one row, more than a tile), rows whose id is outside it, one and two linears, odd rows
@pytest.mark.parametrize("experts,n,k,gs,counts,tail,linears", [
    (6, 264, 512, 64, (0, 1, 70, 129, 0, 64), 0, 1), (4, 131, 1056, 32, (200, 0, 1, 0), 5, 2), (3, 256, 4096, 64, (0, 0, 40), 30, 1), (2, 72, 320, 64, (700, 391), 0, 2),
    (8, 512, 256, 128, (0, 0, 0, 500, 0, 0, 0, 0), 17, 1)])
def test_grouped_edges(cuda, experts, n, k, gs, counts, tail, linears):
    rng = np.random.default_rng(experts + n + k)
    ids = np.repeat(np.arange(experts + 1), (*counts, tail)).astype(np.int32)
    rows = ids.size
    assert rows > 8 * experts
    x = util.activations(rng, rows, k)
    host = [util.affine_weights(rng, n, k, 4, gs, experts=experts) for _ in range(linears)]
    dev = [(dev_u32(w, cuda), dev_bf16(s, cuda), dev_bf16(b, cuda)) for w, s, b in host]
    ys = ops.gather_qmm_siblings(dev_bf16(x, cuda), dev, dev_i32(ids, cuda), gs, 4)
    live = rows - tail
    for t, y in zip(host, ys):
        got = O.bf16_to_f32(host_bf16_bits(y))
        assert not got[live:].any()
        err, l2 = util.parity(got[:live], O.bf16_to_f32(O.gather_qmm(x[:live], *t, ids[:live], gs, 4)))
        assert err <= TOL and l2 <= 4e-3, (err, l2)
    assert ops.device_status() == 0


# one to four pairs a tile, two planes of a ragged number of tokens, rows that are no whole tile
@pytest.mark.parametrize("name,fmt,rows,k,tokens", [("Q4K", O.Q4_K, 256, 4096, 33), ("Q4K", O.Q4_K, 2048, 8192, 40), ("Q4K", O.Q4_K, 512, 2048, 300), ("Q4K", O.Q4_K, 136, 256, 600),
                                                    ("Q2K", O.Q2_K, 1000, 4096, 45), ("Q2K", O.Q2_K, 4096, 8192, 64), ("Q2K", O.Q2_K, 264, 1024, 600)])
def test_gguf_edges(cuda, name, fmt, rows, k, tokens):
    rng = np.random.default_rng(rows + k + tokens)
    w = util.gguf_weights(rng, fmt, rows, k)
    x = rng.normal(0, 1, size=(tokens, k)).astype(np.float32)
    y = ops.packed_matmul(name, dev_u8(w, cuda), dev_f32(x, cuda)).cpu().numpy()
    pick = np.unique(np.concatenate([np.arange(0, rows, 37), [rows - 1]]))
    truth = x.astype(np.float64) @ O.gguf_decode(fmt, np.ascontiguousarray(w[pick])).reshape(pick.size, k).astype(np.float64).T
    err, l2 = util.parity(y[:, pick], truth)
    assert err <= 2e-4 and l2 <= 1e-4, (err, l2)  # two bf16 planes per operand: 16 significant bits
    assert ops.device_status() == 0
