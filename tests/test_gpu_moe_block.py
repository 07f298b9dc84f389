"""The routed block as one call: what its two forms accept, and what it refuses before a launch."""
import numpy as np
import pytest
import torch

from lisa_b200 import _cabi, ops
from lisa_b200.quant import QuantizedLinear, SwitchGlu
from tests import util
from tests.gpu_util import dev_bf16, dev_f32, dev_u32

pytestmark = pytest.mark.gpu


def _block(cuda, rng, experts, hidden, inter, gs=64, bits=4, top_k=2):
    shapes = [(inter, hidden), (inter, hidden), (hidden, inter)]
    return SwitchGlu(*[QuantizedLinear(*(f(a, cuda) for f, a in zip((dev_u32, dev_bf16, dev_bf16), util.affine_weights(rng, n, k, bits, gs, experts=experts))), gs, bits)
                       for n, k in shapes], top_k)


def test_per_slot_form_takes_what_its_two_steps_take(cuda):
    """Group sizes that are multiples of the codes of a word (moe_gate_up_act, moe_down_combine), and scales at any address."""
    rng = np.random.default_rng(3)
    tokens, experts, hidden, inter = 3, 4, 384, 192
    x, logits = dev_bf16(util.activations(rng, tokens, hidden), cuda), dev_f32(rng.normal(size=(tokens, experts)).astype(np.float32), cuda)
    for gs, shift in ((96, 0), (64, 1)):
        block = _block(cuda, rng, experts, hidden, inter, gs)
        for lin in (block.gate, block.up, block.down):
            odd = torch.empty(lin.scales.numel() + shift, dtype=torch.bfloat16, device=cuda)[shift:].view(lin.scales.shape)
            lin.scales = odd.copy_(lin.scales)
        g, u, d = ((l.weight, l.scales, l.biases) for l in (block.gate, block.up, block.down))
        idx, weights = ops.moe_route(logits, block.top_k)
        want = ops.moe_down_combine(ops.moe_gate_up_act(x, idx, g, u, gs, 4), idx, weights, d, gs, 4)
        assert torch.equal(block.forward(x, logits), want)


def _swap(lin, **kw):
    return QuantizedLinear(kw.get("weight", lin.weight), kw.get("scales", lin.scales), kw.get("biases", lin.biases), lin.group_size, lin.bits)


@pytest.mark.parametrize("tokens", [1, 32])
def test_every_mismatched_tensor_is_refused_on_the_host(cuda, tokens):
    """Both forms: an expert, row or column too few in any of the nine tensors, other bits, another group size."""
    rng = np.random.default_rng(4)
    experts, hidden, inter = 4, 256, 128
    block = _block(cuda, rng, experts, hidden, inter)
    x, logits = dev_bf16(util.activations(rng, tokens, hidden), cuda), dev_f32(rng.normal(size=(tokens, experts)).astype(np.float32), cuda)
    assert block.forward(x, logits).shape == (tokens, hidden)
    before = ops.launch_count()
    bad = []
    for part in ("gate", "up", "down"):
        lin = getattr(block, part)
        for field in ("weight", "scales", "biases"):
            t = getattr(lin, field)
            bad += [{part: _swap(lin, **{field: v})} for v in (t[:-1], t[:, :-8], t[..., :-1], t[0], t[..., ::2])]
        bad.append({part: _swap(lin, scales=lin.scales.to(torch.float8_e4m3fn))})
    other = _block(cuda, rng, experts, hidden, inter * 2)
    bad += [{"up": other.up}, {"down": other.down}, {"up": _block(cuda, rng, experts, hidden, inter, 64, 2).up}, {"down": _block(cuda, rng, experts, hidden, inter, 128).down},
            {"up": _block(cuda, rng, experts - 1, hidden, inter).up}]
    for change in bad:
        with pytest.raises(_cabi.LisaError) as err:
            SwitchGlu(**{"gate": block.gate, "up": block.up, "down": block.down, **change}, top_k=2).forward(x, logits)
        assert err.value.code == _cabi.ERR_BAD_ARG
    for args in ((x[:, :-64].contiguous(), logits), (x, logits[:, :-1].contiguous()), (x, logits[0]), (x.reshape(-1)[:-hidden // 2], logits)):
        with pytest.raises(_cabi.LisaError):
            block.forward(*args)
    assert ops.launch_count() == before
