"""Float32 attention where two CTAs share a block's tiles of the other side, against float64: odd numbers of tiles, a second half without a tile or that a
row does not see, rows that see nothing, columns between the kernels' own, and launches in which some blocks are shared and others are not."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import seeded

pytestmark = pytest.mark.gpu


def _exact(q, k, v, causal):
    q, k, v = (a.astype(np.float64) for a in (q, k, v))
    s = np.einsum("bqd,bkd->bqk", q, k) * q.shape[-1] ** -0.5
    if causal:
        s[:, np.triu(np.ones(s.shape[1:], bool), 1 + s.shape[2] - s.shape[1])] = -np.inf
    top = s.max(-1, keepdims=True)
    e = np.exp(s - top)
    total = e.sum(-1, keepdims=True)
    return (e / total) @ v, (top + np.log(total))[..., 0], (e / total) @ np.abs(v)


@pytest.mark.parametrize("units,lq,lk,d,causal", [
    (1, 512, 512, 64, True), (1, 512, 512, 64, False), (4, 385, 385, 128, True), (8, 130, 700, 64, True), (2, 257, 577, 40, True), (1, 647, 647, 63, True),
    (5, 300, 311, 80, True), (16, 306, 306, 128, True), (6, 333, 450, 96, False), (4, 451, 451, 100, False), (2, 1, 3005, 64, False), (2, 703, 2984, 64, False),
    (74, 100, 900, 64, False), (12, 880, 880, 72, True), (9, 1097, 1097, 64, True), (7, 1301, 1301, 128, True), (25, 337, 371, 72, True), (5, 1900, 2011, 96, True)])
def test_forward(units, lq, lk, d, causal):
    q, k, v = (seeded((1, units, n, d), i) for i, n in enumerate((lq, lk, lk), 1))
    out, lse = em.attention_forward(*(em.Tensor(a) for a in (q, k, v)), None, causal)
    exact, exact_lse, weighed = _exact(q[0], k[0], v[0], causal)
    # a score is d products in float32, rounded by 2^-24 of up to the sum of their magnitudes, below 2 sqrt(d) for these values; its error is the
    # relative error of its weight. The sums over keys add a tile at a time: at most lk / 64 roundings, and the exponential's 4.
    score, sums = 4.0 * np.sqrt(d) * 2.0 ** -24 * 4, (lk / 64 + 8) * 2.0 ** -24
    assert np.abs(lse.to_np()[0] - exact_lse).max() <= score + sums + np.abs(exact_lse).max() * 2.0 ** -23
    assert (np.abs(out.to_np()[0] - exact) <= (2 * score + 2 * sums) * weighed + 1e-30).all()


@pytest.mark.parametrize("units,lq,lk,d,causal", [
    (1, 512, 512, 64, True), (1, 289, 289, 48, False), (2, 114, 246, 64, False), (3, 271, 271, 63, True), (4, 241, 241, 128, True), (1, 442, 442, 100, False),
    (9, 62, 361, 48, False), (4, 53, 1203, 64, True), (2, 1021, 272, 40, False), (5, 471, 449, 96, False), (6, 822, 822, 64, True), (14, 346, 346, 64, True),
    (6, 662, 662, 96, True), (7, 235, 235, 72, False), (14, 121, 326, 128, True), (1, 1301, 1301, 128, True), (8, 289, 289, 48, True)])
def test_backward(units, lq, lk, d, causal):
    q, k, v, g = (seeded((1, units, n, d), i) for i, n in enumerate((lq, lk, lk, lq), 1))
    tq, tk, tv, tg = (em.Tensor(a) for a in (q, k, v, g))
    out, lse = em.attention_forward(tq, tk, tv, None, causal)
    got = [t.to_np()[0] for t in em.attention_backward(tq, tk, tv, out, lse, tg, None, causal)]
    q, k, v, g = (a[0].astype(np.float64) for a in (q, k, v, g))
    s = np.einsum("bqd,bkd->bqk", q, k) * d ** -0.5
    if causal:
        s[:, np.triu(np.ones((lq, lk), bool), 1 + lk - lq)] = -np.inf
    p = np.exp(s - s.max(-1, keepdims=True))
    p /= p.sum(-1, keepdims=True)
    dp = np.einsum("bqd,bkd->bqk", g, v)
    delta = (p * dp).sum(-1, keepdims=True)
    ds = p * (dp - delta) * d ** -0.5
    # as above: the weights' relative error, and that of dP - delta against their magnitudes; then sums of up to max(lq, lk) terms, a tile at a time
    score = 4.0 * np.sqrt(d) * 2.0 ** -24 * 4 + (lk / 64 + 8) * 2.0 ** -24
    size = p * (np.einsum("bqd,bkd->bqk", abs(g), abs(v)) + (p * abs(dp)).sum(-1, keepdims=True)) * d ** -0.5
    rel = 2 * score + (max(lq, lk) / 64 + 8) * 2.0 ** -24
    exact = (ds @ k, ds.transpose(0, 2, 1) @ q, p.transpose(0, 2, 1) @ g)
    bounds = (size @ abs(k), size.transpose(0, 2, 1) @ abs(q), p.transpose(0, 2, 1) @ abs(g))
    for name, a, e, b in zip(("dq", "dk", "dv"), got, exact, bounds):
        assert (np.abs(a - e) <= rel * b + 1e-30).all(), name


def test_largest_scores_in_either_half():
    """One key holds nearly all of a row's weight, in the first CTA's keys for some rows and in the second's for others."""
    lq, lk, d = 256, 1024, 64
    k, v = seeded((1, 2, lk, d), 1), seeded((1, 2, lk, d), 2)
    chosen = (np.arange(lq) * 37) % lk
    q = 40 * k[:, :, chosen]
    out, _ = em.attention_forward(*(em.Tensor(a) for a in (q, k, v)), None, False)
    np.testing.assert_allclose(out.to_np()[0], _exact(q[0], k[0], v[0], False)[0], rtol=0, atol=2e-4)


def test_repeats_bit_for_bit():
    q, k, v = (em.Tensor(seeded((1, 12, 880, 64), i)) for i in range(3))
    def run():
        out, lse = em.attention_forward(q, k, v, None, True)
        short = [em.Tensor(seeded((1, 6, 622, 64), i)) for i in range(4)]
        o2, l2 = em.attention_forward(*short[:3], None, True)
        return [t.to_np() for t in (out, lse, *em.attention_backward(*short[:3], o2, l2, short[3], None, True))]

    first = run()
    for _ in range(3):
        assert all(np.array_equal(a, b) for a, b in zip(first, run()))
