"""GGUF matvecs of f32 activations: sums as good as f32 ones."""
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
