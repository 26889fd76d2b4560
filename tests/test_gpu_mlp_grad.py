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


def test_kept_scratch(lib):
    """One object called from several threads with batches that grow, shrink and exceed what it
    keeps (2^20 samples): each call's result is that of the call made alone."""
    from concurrent.futures import ThreadPoolExecutor

    p, norm = random_net(23)
    sizes = [40_000, 3, 5_000, 100_000, 129, (1 << 20) + 1]
    batches = [data(n, 30 + n) for n in sizes]
    alone = []
    for x, t in batches:
        m = net_with(p, norm)
        alone.append((m.gradients(x, t), m.predict(x)))
        m.close()
    m = net_with(p, norm)
    with ThreadPoolExecutor(4) as pool:
        got = list(pool.map(lambda b: (m.gradients(*b), m.predict(b[0])), batches * 2))
    m.close()
    for (a, ya), (b, yb) in zip(alone * 2, got):
        assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(ya, yb)
