"""Operators that take the activations as they are -- 8-bit codes, group sizes 32 and 128, three to eight rows, the routed block -- on inputs where a
coarse grid of the activations shows: in every 32 of k one element is `ratio` times the rest, and the weights are zero there.  And the bound of
the grid where there is one: 2- and 4-bit codes with group size 64 at one and two rows.  The default dispatch runs, whatever kernel that is."""
import numpy as np
import pytest

from lisa_b200 import ops
from lisa_b200.quant import QuantizedLinear, SwitchGlu
from oracle import oracle as O
from tests import util
from tests.gpu_util import dev_bf16, dev_f32, dev_u32, host_bf16_bits

pytestmark = pytest.mark.gpu


def _tails(rng, m, k, ratio):
    """Activations and the places of their large elements."""
    hot = np.arange(0, k, 32) + rng.integers(0, 32, size=k // 32)
    x = O.bf16_to_f32(util.activations(rng, m, k))
    x[:, hot] *= ratio
    return O.f32_to_bf16(x.astype(np.float32)), hot


def _without(w, hot, bits):
    """The packed rows with code 0 at those places."""
    w, per = w.copy(), 32 // bits
    for c in hot:
        w[..., c // per] &= ~np.uint32(((1 << bits) - 1) << (bits * (c % per)))
    return w


@pytest.mark.parametrize("bits,gs", [(8, 32), (8, 64), (8, 128), (4, 32), (4, 128), (2, 32), (2, 128)])
@pytest.mark.parametrize("n,k", [(264, 1280), (72, 4352)])
@pytest.mark.parametrize("m", [1, 2, 5])
@pytest.mark.parametrize("ratio", [2.0 ** 10, 2.0 ** 16])
def test_heavy_tails(cuda, bits, gs, n, k, m, ratio):
    rng = np.random.default_rng(n + k + bits + gs + m)
    w, s, _ = util.affine_weights(rng, n, k, bits, gs)
    x, hot = _tails(rng, m, k, ratio)
    w, b = _without(w, hot, bits), np.zeros_like(s)
    y = ops.quantized_matmul(dev_bf16(x, cuda), dev_u32(w, cuda), dev_bf16(s, cuda), dev_bf16(b, cuda), True, gs, bits)
    truth = O.affine_matmul(x, w, s, b, gs, bits, round_weight_bf16=False, f64=True).astype(np.float64)
    terms = np.abs(O.bf16_to_f32(x).astype(np.float64)) @ np.abs(O.affine_dequantize(w, s, b, gs, bits, out_f32=True).astype(np.float64)).T
    # the rounding of the output, and of f32 sums over the terms that are not zero
    assert np.all(np.abs(O.bf16_to_f32(host_bf16_bits(y)) - truth) <= 2.0 ** -8 * np.abs(truth) + 2.0 ** -16 * terms)


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("n,k", [(264, 1280), (72, 4352)])
@pytest.mark.parametrize("m", [1, 2, 3, 8])
@pytest.mark.parametrize("ratio", [2.0 ** 6, 2.0 ** 10])
def test_heavy_tails_of_group_size_64(cuda, bits, n, k, m, ratio):
    """One and two rows: an element is off by at most 2^-14 of its group's largest power of two (include/lisa_cuda.h)."""
    rng = np.random.default_rng(n + k + bits + m)
    w, s, _ = util.affine_weights(rng, n, k, bits, 64)
    x, hot = _tails(rng, m, k, ratio)
    w, b = _without(w, hot, bits), np.zeros_like(s)
    y = ops.quantized_matmul(dev_bf16(x, cuda), dev_u32(w, cuda), dev_bf16(s, cuda), dev_bf16(b, cuda), True, 64, bits)
    truth = O.affine_matmul(x, w, s, b, 64, bits, round_weight_bf16=False, f64=True).astype(np.float64)
    xf = np.abs(O.bf16_to_f32(x).astype(np.float64))
    wabs = np.abs(O.affine_dequantize(w, s, b, 64, bits, out_f32=True).astype(np.float64))
    step = 2.0 ** (np.floor(np.log2(xf.reshape(m, k // 64, 64).max(axis=2))) - 14) if m <= 2 else np.zeros((m, k // 64))
    bound = np.einsum("ngk,mg->mn", wabs.reshape(n, k // 64, 64), step) + 2.0 ** -8 * np.abs(truth) + 2.0 ** -16 * (xf @ wabs.T)
    assert np.all(np.abs(O.bf16_to_f32(host_bf16_bits(y)) - truth) <= bound)


@pytest.mark.parametrize("scale", [2.0 ** -100, 2.0 ** -118])
@pytest.mark.parametrize("bits,gs,m", [(8, 64, 1), (8, 64, 4), (4, 128, 2), (4, 128, 8), (4, 32, 1), (2, 128, 3)])
def test_small_activations_are_not_zeros(cuda, bits, gs, m, scale):
    """Groups of very small elements: the kernels' grids follow them down to the range of a float."""
    rng = np.random.default_rng(bits + gs + m)
    n, k = 64, 512
    w, s, b = util.affine_weights(rng, n, k, bits, gs)
    x = O.f32_to_bf16((O.bf16_to_f32(util.activations(rng, m, k)) * np.float32(scale)).astype(np.float32))
    y = ops.quantized_matmul(dev_bf16(x, cuda), dev_u32(w, cuda), dev_bf16(s, cuda), dev_bf16(b, cuda), True, gs, bits)
    truth = O.bf16_to_f32(x).astype(np.float64) @ O.affine_dequantize(w, s, b, gs, bits, out_f32=True).astype(np.float64).T
    err = np.abs(O.bf16_to_f32(host_bf16_bits(y)).astype(np.float64) - truth)
    # (2^-122 is the grid of four bytes at its lower end, 2^-133 the smallest bf16)
    assert np.all(err <= 2.0 ** -8 * np.abs(truth) + 2.0 ** -12 * np.sqrt(np.mean(truth * truth)) + 2.0 ** -117)
    assert np.linalg.norm(err) <= (2.0 ** -7 if scale > 2.0 ** -110 else 0.05) * np.linalg.norm(truth)


@pytest.mark.parametrize("gs", [32, 64, 128])
@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("tokens", [1, 3, 9])
def test_routed_block_with_heavy_tails(cuda, gs, bits, tokens):
    rng = np.random.default_rng(bits + gs + tokens)
    experts, top_k, hidden, inter = 8, 4, 1024, 384
    x, hot = _tails(rng, tokens, hidden, 2.0 ** 10)
    lins = []
    for n, k in ((inter, hidden), (inter, hidden), (hidden, inter)):
        w, s, b = util.affine_weights(rng, n, k, bits, gs, experts=experts)
        if k == hidden:
            w, b = _without(w, hot, bits), np.zeros_like(b)
        lins.append(QuantizedLinear(dev_u32(w, cuda), dev_bf16(s, cuda), dev_bf16(b, cuda), gs, bits))
    block = SwitchGlu(*lins, top_k)
    tx, logits = dev_bf16(x, cuda), dev_f32(rng.normal(size=(tokens, experts)).astype(np.float32), cuda)
    idx, weights = ops.moe_route(logits, top_k)
    g, u, d = ((l.weight, l.scales, l.biases) for l in lins)
    want = ops.moe_down_combine(ops.moe_gate_up_act(tx, idx, g, u, gs, bits), idx, weights, d, gs, bits).float()  # f32 throughout
    got = block.forward(tx, logits).float()
    # gate, up, their SwiGLU and down are rounded to bf16 in both: a rounding that falls the other way moves a result by 2^-8
    assert float((got - want).norm() / want.norm()) <= 2.0 ** -7
