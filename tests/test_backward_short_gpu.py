"""The single-pass backward at 128 columns takes dQ out of tensor memory in halves up to two query tiles and in whole rows above: both sides of the
line against float64, with a single row, partial tiles and columns that are not the kernel's own."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import bf16_round, seeded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("lq,lk,d", [(1, 1, 128), (1, 300, 72), (127, 128, 120), (129, 700, 96), (255, 257, 128), (256, 256, 128), (256, 1000, 112), (257, 257, 128), (258, 600, 80)])
def test_gradients_on_both_sides_of_the_line(lq, lk, d, causal):
    shape = lambda n: (1, 3, n, d)  # noqa: E731
    q, k, v = (bf16_round(seeded(shape(n), i, 0.5)) for i, n in enumerate((lq, lk, lk)))
    g = bf16_round(seeded(shape(lq), 9))
    tq, tk, tv, tg = (em.Tensor(x, "bfloat16") for x in (q, k, v, g))
    o, lse = em.attention_forward(tq, tk, tv, None, causal)
    got = em.attention_backward(tq, tk, tv, o, lse, tg, None, causal)
    q, k, v, g = (x[0].astype(np.float64) for x in (q, k, v, g))
    s = np.einsum("hqd,hkd->hqk", q, k) * d ** -0.5
    if causal:
        s = np.where(np.arange(lk)[None, :] > np.arange(lq)[:, None] + lk - lq, -np.inf, s)
    p = np.exp(s - s.max(-1, keepdims=True))
    p /= p.sum(-1, keepdims=True)
    dp = np.einsum("hqd,hkd->hqk", g, v)
    ds = p * (dp - (p * dp).sum(-1, keepdims=True)) * d ** -0.5
    exact = (np.einsum("hqk,hkd->hqd", ds, k), np.einsum("hqk,hqd->hkd", ds, q), np.einsum("hqk,hqd->hkd", p, g))
    # what P (dP - delta) is rounded to: P, dS and the results to bf16 (2^-9 each), delta by o's rounding. Of one key alone dS is 0 but for delta's.
    size = np.einsum("hqk,hqk->hqk", p, np.abs(dp) + (p * np.abs(dp)).sum(-1, keepdims=True)) * d ** -0.5
    bounds = (np.einsum("hqk,hkd->hqd", size, np.abs(k)), np.einsum("hqk,hqd->hkd", size, np.abs(q)), np.einsum("hqk,hqd->hkd", p, np.abs(g)))
    # delta sums d products o g of o rounded to 2^-9 of itself: |g| |o| 2^-9 a row at most, of which d ** -0.5 p |k| reaches dq
    delta = p * (np.abs(g) * np.abs(np.einsum("hqk,hkd->hqd", p, v))).sum(-1, keepdims=True) * d ** -0.5 * 2.0 ** -9
    extra = (np.einsum("hqk,hkd->hqd", delta, np.abs(k)), np.einsum("hqk,hqd->hkd", delta, np.abs(q)), 0.0)
    for name, a, e, b, x in zip(("dq", "dk", "dv"), got, exact, bounds, extra):
        assert (np.abs(a.to_np()[0] - e) <= 4 * 2.0 ** -9 * b + x + 1e-30).all(), name
