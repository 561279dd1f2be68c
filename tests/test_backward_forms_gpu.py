"""The single-pass backward's forms at 64 columns: dQ beside dP above eight query tiles, in dP's columns below. Both against float64 around the
line and with partial tiles."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import bf16_round, seeded

pytestmark = pytest.mark.gpu


def _exact(q, k, v, g, scale, causal):
    s = np.einsum("hqd,hkd->hqk", q, k, dtype=np.float64) * scale
    if causal:
        lq, lk = s.shape[1:]
        s = np.where(np.arange(lk)[None, :] > np.arange(lq)[:, None] + lk - lq, -np.inf, s)
    p = np.exp(s - s.max(-1, keepdims=True))
    p /= p.sum(-1, keepdims=True)
    dp = np.einsum("hqd,hkd->hqk", g, v, dtype=np.float64)
    ds = p * (dp - (p * dp).sum(-1, keepdims=True)) * scale
    return np.einsum("hqk,hkd->hqd", ds, k), np.einsum("hqk,hqd->hkd", ds, q), np.einsum("hqk,hqd->hkd", p, g)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("lq,lk,d", [(1024, 1024, 64), (1025, 1300, 64), (1151, 1152, 56), (1153, 1537, 64), (1024, 1100, 56)])
def test_gradients_on_both_sides_of_the_line(lq, lk, d, causal):
    shape = lambda n: (1, 2, n, d)  # noqa: E731
    q, k, v = (bf16_round(seeded(shape(n), i, 0.5)) for i, n in enumerate((lq, lk, lk)))
    g = bf16_round(seeded(shape(lq), 9))
    tq, tk, tv, tg = (em.Tensor(x, "bfloat16") for x in (q, k, v, g))
    o, lse = em.attention_forward(tq, tk, tv, None, causal)
    got = em.attention_backward(tq, tk, tv, o, lse, tg, None, causal)
    exact = _exact(*(x[0].astype(np.float64) for x in (q, k, v, g)), d ** -0.5, causal)
    for name, a, e in zip(("dq", "dk", "dv"), got, exact):
        a = a.to_np()[0]
        # weights and score gradients are bf16 operands (2^-9 each) and so are the results and delta's o: 1e-2 of the norm is above their sum
        assert np.linalg.norm(a - e) <= 1e-2 * np.linalg.norm(e), name
        assert np.abs(a - e).max() <= 2e-2 * np.abs(e).max(), name
