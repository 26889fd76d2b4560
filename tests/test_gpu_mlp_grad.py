"""The gradient kernel of the learned warm start at the edges of its tiles (128 samples) and of
its grid (one CTA per SM: from 152 tiles on a CTA sums over several), against the CPU oracle,
which rounds the same operands to BF16.  What is left between the two is the order of FP32 sums
(1e-6) and operands on whose rounding the two fall on different sides: one BF16 ulp (2^-8) of
one term each.  Two such flips in a row of one sample, the smallest sum there is, are 2^-7 of
it; 2e-2 of a block's largest entry holds two and a half of them."""
import numpy as np
import pytest

from oracle import oracle
from test_gpu_mlp import net_with, rel
from test_mlp_oracle import data, random_net

pytestmark = pytest.mark.gpu

BLOCKS = {"W1": (0, 256), "b1": (256, 320), "W2": (320, 4416), "b2": (4416, 4480), "W3": (4480, 8576),
          "b3": (8576, 8640), "W4": (8640, 8704), "b4": (8704, 8705)}


@pytest.mark.parametrize("n", [1, 2, 31, 127, 128, 129, 300, 128 * 152, 128 * 152 + 1, 128 * 304 + 65])
def test_gradient_tiles(lib, n):
    p, norm = random_net(21)
    x, t = data(n, 22)
    m = net_with(p, norm)
    g, loss = m.gradients(x, t)
    again, loss2 = m.gradients(x, t)
    m.close()
    assert np.array_equal(g, again) and loss == loss2   # sums in a fixed order
    _, ref, l_ref = oracle.mlp_eval(p, norm, x, t, bf16=True, grad=True)
    for name, (a, b) in BLOCKS.items():
        assert rel(g[a:b], ref[a:b]) < 2e-2, name
    assert abs(loss - l_ref) <= 1e-3 * l_ref
