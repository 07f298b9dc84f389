"""The byte-dot-product GGUF matvec (gguf_dp.cu) against the oracle, at the edges of its tiling."""
import numpy as np
import pytest

from lisa_b200 import ops
from oracle import oracle as O
from tests import util
from tests.gpu_util import dev_f32, dev_u8

pytestmark = pytest.mark.gpu


# octets of rows (part of one, one, several per CTA), ragged last steps (blocks that are no multiple of two or four; Q2_K rows that are
# not whole 16-byte pieces), rows that start in the middle of a sector, k cut into parts
@pytest.mark.parametrize("name,fmt", [("Q2K", O.Q2_K), ("Q4K", O.Q4_K)])
@pytest.mark.parametrize("rows,k,tokens", [(8, 256, 1), (16, 512, 2), (24, 768, 1), (40, 1024, 3), (1208, 1280, 1), (40, 2816, 8), (64, 7168, 1), (16, 18432, 2)])
def test_edges(cuda, name, fmt, rows, k, tokens):
    rng = np.random.default_rng(rows + k + tokens)
    w = util.gguf_weights(rng, fmt, rows, k)
    x = rng.normal(0, 1, size=(tokens, k)).astype(np.float32)
    x[0, 5] = 3e4
    y = ops.packed_matvec(name, dev_u8(w, cuda), dev_f32(x, cuda)).cpu().numpy()
    err, l2 = util.parity(y, x.astype(np.float64) @ O.gguf_decode(fmt, w).reshape(rows, k).astype(np.float64).T)
    assert err <= 1e-4 and l2 <= 1e-5, (err, l2)
