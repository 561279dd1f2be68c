"""The input gradient of a float32 layer of few columns: a sum of at most twelve products, rounded as one chain of fused multiply-adds up to four columns
and as two (every other column each) above, which is closer to the exact sum."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import seeded

pytestmark = pytest.mark.gpu


def _chain(a, b):
    # products of two float32 numbers are exact in float64, so one rounding to float32 a step is a fused multiply-add's (but for ties made by rounding twice)
    s = np.float32(0.0)
    for x, y in zip(a, b):
        s = (x.astype(np.float64)[:, None] * y.astype(np.float64) + s).astype(np.float32)
    return s


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("m,k", [(33, 132), (256, 784)])
def test_grad_x_rounds_as_its_chains(m, k, n):
    x, w, dy = seeded((m, k), 1), seeded((k, n), 2, 0.1), seeded((m, n), 3)
    gx = em.linear_backward(em.Tensor(x), em.Tensor(w), em.Tensor(dy))[0].to_np()
    chains = 2 if n > 4 else 1
    same = sum(_chain(dy.T[c::chains], w.T[c::chains]) for c in range(chains))
    assert np.mean(gx != same) <= 1e-4
    exact = dy.astype(np.float64) @ w.astype(np.float64).T
    assert np.linalg.norm(gx - exact) <= 1.0001 * np.linalg.norm(same - exact)
