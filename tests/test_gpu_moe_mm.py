"""The routed block of a batch of tokens (moe_mm.cu) against the oracle's block, at the edges of its sort and its tiling."""
import numpy as np
import pytest

from lisa_b200 import ops
from lisa_b200.quant import QuantizedLinear, SwitchGlu
from oracle import oracle as O
from tests import util
from tests.gpu_util import dev_bf16, dev_f32, dev_u32, host_bf16_bits

pytestmark = pytest.mark.gpu


# runs of less and more than eight rows (one and several entries), ragged last steps, row blocks that are no multiple of eight, cuts, both
# group sizes, the largest one-block sort, sixteen warps a CTA (rows of much k)
@pytest.mark.parametrize("tokens,experts,top_k,hidden,inter,bits,gs", [
    (5, 8, 8, 128, 128, 4, 64), (33, 16, 2, 640, 384, 4, 64), (64, 128, 16, 256, 128, 4, 64), (61, 64, 8, 2048, 768, 4, 64), (16, 16, 6, 1152, 640, 2, 64),
    (9, 16, 4, 4096, 1152, 4, 64), (12, 32, 8, 1024, 512, 4, 128), (40, 40, 8, 1280, 768, 2, 128), (33, 1024, 1, 128, 128, 2, 64)])
def test_edges(cuda, tokens, experts, top_k, hidden, inter, bits, gs):
    rng = np.random.default_rng(tokens + experts + hidden + inter)
    host = [util.affine_weights(rng, n, k, bits, gs, experts=experts) for n, k in ((inter, hidden), (inter, hidden), (hidden, inter))]
    block = SwitchGlu(*[QuantizedLinear(dev_u32(w, cuda), dev_bf16(s, cuda), dev_bf16(b, cuda), gs, bits) for w, s, b in host], top_k)
    x = util.activations(rng, tokens, hidden)
    logits = rng.normal(size=(tokens, experts)).astype(np.float32)
    logits[:, 0] += 2.0  # one long run
    got = O.bf16_to_f32(host_bf16_bits(block.forward(dev_bf16(x, cuda), dev_f32(logits, cuda))))
    want, _ = O.moe_forward(x, logits, *host, top_k, gs, bits, round_weight_bf16=False)
    err, l2 = util.parity(got, O.bf16_to_f32(want))
    # gate, up, their product, down and the fold are rounded to bf16 on both sides: where a sum in another order falls to the other side, down's row and the
    # fold move by an ulp, 2^-7 each at most; few do, so that the norm of the differences is below that of one rounding (2^-9 to each side)
    assert err <= 2.0 ** -6 and l2 <= 2.0 ** -8, (err, l2)
    assert ops.device_status() == 0
