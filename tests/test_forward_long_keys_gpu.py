"""The bf16 forward over many key tiles: from the second one on, a tile's weights are written over those that the product before them has read, and
the softmax warps learn of that product's end early (asked while they still compute) or late (waited for). CTAs alone on the chip and two or three to an
SM's turn, maxima that move (every other tile's weights are rescaled) or stand still. Both forms give the same bits, call after call."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import bf16_round, seeded
from ember_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("units,lq,lk,d,causal", [(1, 128, 4096, 128, False), (2, 640, 3001, 64, True), (150, 128, 1500, 128, False), (37, 1280, 1280, 80, True)])
@pytest.mark.parametrize("growth", [0.0, 200.0])
def test_both_forms_repeat_and_agree(units, lq, lk, d, causal, growth):
    q, k, v = (bf16_round(seeded((1, units, n, d), s, 0.5)) for n, s in ((lq, 1), (lk, 2), (lk, 3)))
    if growth:  # one component raises the scores along the keys, by `growth` from the first to the last
        q[..., 0] = 4.0
        k[..., 0] = bf16_round((np.arange(lk) / lk * growth / 4.0 * np.sqrt(d)).astype(np.float32))
    tq, tk, tv = (em.Tensor(x, "bfloat16") for x in (q, k, v))
    L = _lib.lib()
    before = L.ember_set_forward_block_rows(128)
    try:
        got = []
        for rows in (128, 128, 128, 256, 256):
            L.ember_set_forward_block_rows(rows)
            o, lse = em.attention_forward(tq, tk, tv, None, causal)
            got.append((o.to_np(), lse.to_np()))
    finally:
        L.ember_set_forward_block_rows(before)
    for o, lse in got[1:]:
        assert np.array_equal(o, got[0][0]) and np.array_equal(lse, got[0][1])
    for u in {0, units // 2, units - 1}:
        s = (q[0, u].astype(np.float64) @ k[0, u].astype(np.float64).T) / np.sqrt(d)
        if causal:
            s[np.arange(lk)[None, :] > np.arange(lq)[:, None] + lk - lq] = -np.inf
        m = s.max(-1, keepdims=True)
        p = np.exp(s - m)
        l = p.sum(-1, keepdims=True)
        # weights and results are rounded to 8 bits: 2^-9 of the largest value each; sums and exponents in float32 beside that
        assert np.abs(got[0][0][0, u] - (p / l) @ v[0, u].astype(np.float64)).max() <= 1.05 * 2.0 ** -8 * np.abs(v[0, u]).max()
        exact = (m + np.log(l))[:, 0]
        assert np.abs(got[0][1][0, u] - exact).max() <= 1e-4 + 2e-6 * np.abs(exact).max()
