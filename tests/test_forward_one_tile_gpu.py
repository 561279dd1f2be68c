"""One query tile per CTA of the bf16 forward: two threads share a row and agree on its maximum. Against the two-tile form (bit for
bit) and float64, where the maximum keeps moving past the rescale threshold, with either sign of the scale and ragged ends."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import bf16_round, seeded
from ember_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [16, 64, 80, 128])
@pytest.mark.parametrize("lq,lk,causal", [(1, 1, False), (128, 129, True), (130, 64, False), (70, 1000, True), (300, 512, False)])
@pytest.mark.parametrize("sign,growth", [(1.0, 0.0), (-1.0, 0.0), (1.0, 40.0), (-1.0, 40.0)])
def test_one_tile_form(lq, lk, d, causal, sign, growth):
    q, k, v = (bf16_round(seeded((1, 2, n, d), s, 0.5)) for n, s in ((lq, 1), (lk, 2), (lk, 3)))
    scale = sign / np.sqrt(d)
    if growth:  # one component raises the scores along the keys, by `growth` from the first to the last
        q[..., 0] = 4.0
        k[..., 0] = bf16_round((np.arange(lk) / lk * growth / (4.0 * scale)).astype(np.float32))
    L = _lib.lib()
    before = L.ember_set_forward_block_rows(128)
    try:
        got = {}
        for rows in (128, 256):
            L.ember_set_forward_block_rows(rows)
            o, lse = em.attention_forward(*(em.Tensor(x, "bfloat16") for x in (q, k, v)), float(scale), causal)
            got[rows] = o.to_np(), lse.to_np()
    finally:
        L.ember_set_forward_block_rows(before)
    assert np.array_equal(got[128][0], got[256][0]) and np.array_equal(got[128][1], got[256][1])
    s = (q.astype(np.float64) @ k.astype(np.float64).swapaxes(-1, -2)) * scale
    if causal:
        s[..., np.arange(lk)[None, :] > np.arange(lq)[:, None] + lk - lq] = -np.inf
    m = s.max(-1, keepdims=True)
    with np.errstate(invalid="ignore"):
        p = np.exp(s - m)
    l = p.sum(-1, keepdims=True)
    seen = np.isfinite(l[..., 0])  # rows of more queries than keys under the mask see nothing
    ref = (p / l) @ v.astype(np.float64)
    # weights and results are rounded to 8 bits: 2^-9 of the largest value each; sums and exponents in float32 beside that
    assert np.abs(got[128][0] - ref)[seen].max() <= 1.05 * 2.0**-8 * np.abs(v).max()
    ref_lse = (m + np.log(l))[..., 0]
    assert np.abs(got[128][1] - ref_lse)[seen].max() <= 1e-4 + 2e-6 * np.abs(ref_lse[seen]).max()
