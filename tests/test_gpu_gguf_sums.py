"""GGUF matvecs of f32 activations: sums as good as f32 ones, and a row's bits by its length alone."""
import numpy as np
import pytest
import torch

from lisa_b200 import ops
from oracle import oracle as O
from tests import util
from tests.gpu_util import dev_f32, dev_u8

pytestmark = pytest.mark.gpu


def _inputs(rng, tokens, k, kind):
    x = rng.normal(0, 1, size=(tokens, k)).astype(np.float32)
    if kind == "outlier":
        x[0, 5] = 3e4
    if kind == "tails":
        x[:, ::32] *= 2.0 ** 12
    return x


# one token only where the three-byte grid of the header does not hold (Q2_K rows that are no whole stages)
@pytest.mark.parametrize("name,fmt,rows,k,tokens", [
    ("Q2K", O.Q2_K, 256, 8960, 1), ("Q2K", O.Q2_K, 2400, 2816, 1), ("Q2K", O.Q2_K, 136, 18432, 2), ("Q2K", O.Q2_K, 1208, 1280, 4), ("Q2K", O.Q2_K, 64, 7168, 8),
    ("Q2K", O.Q2_K, 2304, 3072, 19), ("Q4K", O.Q4_K, 24, 768, 2), ("Q4K", O.Q4_K, 1208, 1280, 4), ("Q4K", O.Q4_K, 64, 7168, 8), ("Q4K", O.Q4_K, 2304, 3072, 19)])
@pytest.mark.parametrize("kind", ["normal", "outlier", "tails"])
def test_error_against_f64_is_that_of_f32_sums(cuda, name, fmt, rows, k, tokens, kind):
    rng = np.random.default_rng(rows + k + tokens)
    w = util.gguf_weights(rng, fmt, rows, k)
    x = _inputs(rng, tokens, k, kind)
    truth = x.astype(np.float64) @ O.gguf_decode(fmt, w).reshape(rows, k).astype(np.float64).T
    err, l2 = util.parity(ops.packed_matvec(name, dev_u8(w, cuda), dev_f32(x, cuda)).cpu().numpy(), truth)
    # one rounding is 2^-24 = 0.6e-7; the warp-per-row kernel's f32 sums measure 0.8 to 1.5e-7.  With an outlier the sums are its few roundings,
    # all in one accumulator.
    assert l2 <= (1.6e-7 if kind == "normal" else 3e-7), l2
    assert err <= 2e-6, err


@pytest.mark.parametrize("name,fmt,experts,rows,k,tokens,top_k", [("Q2K", O.Q2_K, 4, 256, 2304, 1, 2), ("Q2K", O.Q2_K, 8, 64, 1024, 90, 4), ("Q4K", O.Q4_K, 8, 64, 1024, 90, 4)])
def test_expert_error_against_f64_is_that_of_f32_sums(cuda, name, fmt, experts, rows, k, tokens, top_k):
    rng = np.random.default_rng(rows + k)
    w = util.gguf_weights(rng, fmt, rows, k, experts=experts)
    x = rng.normal(0, 1, size=(tokens, 1, k)).astype(np.float32)
    ids = np.stack([rng.permutation(experts)[:top_k] for _ in range(tokens)]).astype(np.int32)
    truth = np.einsum("tk,tjrk->tjr", x[:, 0].astype(np.float64), O.gguf_decode(fmt, w).reshape(experts, rows, k).astype(np.float64)[ids])
    _, l2 = util.parity(ops.expert_matvec(name, dev_u8(w, cuda), dev_f32(x, cuda), torch.from_numpy(ids).to(cuda)).cpu().numpy(), truth)
    assert l2 <= 1.6e-7, l2


@pytest.mark.parametrize("name,fmt,k", [("Q2K", O.Q2_K, 256), ("Q2K", O.Q2_K, 2048), ("Q2K", O.Q2_K, 2816), ("Q2K", O.Q2_K, 18432), ("Q4K", O.Q4_K, 768), ("Q4K", O.Q4_K, 2048),
                                        ("Q4K", O.Q4_K, 7168), ("Q4K", O.Q4_K, 18432)])
def test_bits_of_a_row_do_not_depend_on_the_matrix_or_the_batch(cuda, name, fmt, k):
    """A shard of the rows, or some of the tokens, gives what the whole gives, bit for bit: plans differ in clusters, tasks, token sets and rounds."""
    rng = np.random.default_rng(k)
    rows, tokens = 9216, 24
    w = dev_u8(util.gguf_weights(rng, fmt, rows, k), cuda)
    x = dev_f32(rng.normal(0, 1, size=(tokens, k)).astype(np.float32), cuda)
    full = ops.packed_matvec(name, w, x)
    for r0, r1 in ((0, 8), (4608, 9216), (1024, 3496)):
        part = w[r0:r1].contiguous()
        for t0, t1 in ((0, 24), (3, 5), (7, 10), (11, 16), (16, 24)):
            assert torch.equal(ops.packed_matvec(name, part, x[t0:t1].contiguous()), full[t0:t1, r0:r1]), (r0, r1, t0, t1)
    if k % 1024 and name == "Q2K":  # (a single token of whole stages is on the grid of the header)
        assert torch.equal(ops.packed_matvec(name, w[:2304].contiguous(), x[9:10].contiguous()), full[9:10, :2304])


# a row's sums of sixteen parts fit a CTA, or not (one CTA per slot: more slots than SMs)
@pytest.mark.parametrize("rows,k,tokens", [(512, 2304, 20), (8192, 5376, 60)])
def test_bits_of_an_expert_row_do_not_depend_on_the_slots(cuda, rows, k, tokens):
    rng = np.random.default_rng(5)
    experts, top_k = 3, 3
    w = dev_u8(util.gguf_weights(rng, O.Q2_K, rows, k, experts=experts), cuda)
    x = dev_f32(rng.normal(0, 1, size=(tokens, 1, k)).astype(np.float32), cuda)
    ids = torch.from_numpy(rng.integers(0, experts, size=(tokens, top_k)).astype(np.int32)).to(cuda)
    full = ops.expert_matvec("Q2K", w, x, ids)
    assert torch.equal(ops.expert_matvec("Q2K", w, x[4:5].contiguous(), ids[4:5].contiguous()), full[4:5])
    assert torch.equal(ops.expert_matvec("Q2K", w[:, 64:128].contiguous(), x, ids), full[..., 64:128])


def test_small_activations_are_not_zeros(cuda):
    rng = np.random.default_rng(6)
    for name, fmt in (("Q2K", O.Q2_K), ("Q4K", O.Q4_K)):
        w = util.gguf_weights(rng, fmt, 64, 1024)
        for tokens in (1, 3):
            x = (rng.normal(0, 1, size=(tokens, 1024)) * 2.0 ** -110).astype(np.float32)
            truth = x.astype(np.float64) @ O.gguf_decode(fmt, w).reshape(64, 1024).astype(np.float64).T
            _, l2 = util.parity(ops.packed_matvec(name, dev_u8(w, cuda), dev_f32(x, cuda)).cpu().numpy(), truth)
            # (the three bytes of a single token keep 12 of their 22 bits at 2^-110)
            assert l2 <= (2.0 ** -10 if tokens == 1 else 1e-6), (name, tokens, l2)
