"""The kernels of a small classifier step: float32 projections to at most 12 columns, and cross-entropy of few classes and rows,
at the edges of what sends a call to them, against float64."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import bf16_round, seeded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 3, 4, 5, 257, 2049])
@pytest.mark.parametrize("k", [4, 252, 256, 784, 1028, 2052])
@pytest.mark.parametrize("n,bias", [(1, True), (2, False), (5, True), (7, True), (10, True), (12, False), (13, True)])
def test_narrow_projection(m, k, n, bias):
    x, w = seeded((m, k), 1), seeded((k, n), 2)
    b = seeded((n,), 3) if bias else None
    y = em.linear_forward(em.Tensor(x), em.Tensor(w), em.Tensor(b) if bias else None).to_np()
    x, w = x.astype(np.float64), w.astype(np.float64)
    ref = x @ w + (b if bias else 0.0)
    # float32 products and sums of k terms, in whatever order: at most k / 8 + 32 roundings on a term's way (tiles add slabs one after the other)
    bound = (k / 8 + 32) * 2.0**-24 * (np.abs(x) @ np.abs(w) + (np.abs(b) if bias else 0.0))
    assert (np.abs(y - ref) <= bound).all()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 100, 195, 196, 255, 256, 257, 1000])  # 195 x 12: the last of that width in one block
@pytest.mark.parametrize("cols", [1, 2, 10, 12, 24, 25, 31, 32, 33])
def test_small_cross_entropy(rows, cols, dtype):
    x = seeded((rows, cols), 4, 3.0)
    x = bf16_round(x) if dtype == "bfloat16" else x
    y = np.eye(cols, dtype=np.float32)[np.random.default_rng(5).integers(cols, size=rows)]
    loss = em.loss.CrossEntropyLoss()
    value = loss(em.Tensor(x, dtype), em.Tensor(y, dtype))
    z = x.astype(np.float64)
    z -= z.max(-1, keepdims=True)
    lp = z - np.log(np.exp(z).sum(-1, keepdims=True))
    # exponents are rounded to float32 (values up to 32), the exponential is good to 2^-22; bfloat16 results to 2^-9
    rel = 32 * 2.0**-23 + 2.0**-21 + (2.0**-8 if dtype == "bfloat16" else 0.0)
    assert (np.abs(loss.probs.to_np() - np.exp(lp)) <= rel * np.exp(lp) + 1e-30).all()
    ref = -(y * lp).sum() / rows
    assert abs(value - ref) <= 4e-6 * max(1.0, abs(ref))


@pytest.mark.parametrize("k", [2**31 - 1024 - 4, 2**31 - 1024])
def test_narrow_projection_of_a_longest_contraction(k):
    """On either side of the last contraction that the kernel takes, whose counter stays below 2^31 past the end."""
    torch = pytest.importorskip("torch")
    from ember_b200 import _lib

    x, w, y = (torch.zeros(n, device="cuda") for n in (k, k, 1))
    at = torch.tensor([0, 3, 1024, 2**30 + 5, k - 1029, k - 1], device="cuda")
    x[at], w[at] = torch.arange(1.0, 7.0, device="cuda"), 0.5
    torch.cuda.synchronize()
    _lib.check(_lib.lib().ember_linear_fwd(x.data_ptr(), w.data_ptr(), None, y.data_ptr(), 1, 1, k, 0, 0, 0, 0, 0, None))
    em._core._sync()
    assert y.item() == 10.5
