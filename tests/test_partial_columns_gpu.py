"""Head dimensions that leave 16 or more of a tile's 64 or 128 columns empty: products stop after the last 16
columns in use and the dQ accumulator holds only the 32-column chunks in use. Every such dimension, so that the
last chunk and the last 16 columns are full, half full and nearly empty, over lengths that end inside a tile,
forward and both backward forms, against the CPU oracle.

bf16 tolerance of the attention tests: 2e-2 of the largest value (operands, probabilities and results in bf16)."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import bf16_round, seeded
from ember_b200 import _lib
from oracle import cpu_oracle

pytestmark = pytest.mark.gpu
TOL = 2e-2


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dim", [8, 16, 24, 32, 40, 48, 56, 72, 80, 88, 96, 104, 112, 120])
def test_forward_and_both_backwards(dim, causal):
    B, H, Lq, Lk = 1, 2, 130, 300
    q, k, v, g = (bf16_round(seeded((B, H, n, dim), s, 0.5)) for s, n in enumerate((Lq, Lk, Lk, Lq), 1))
    tq, tk, tv, tg = (em.Tensor(a, "bfloat16") for a in (q, k, v, g))
    o, lse = em.attention_forward(tq, tk, tv, None, causal)
    ref_o, ref_l = cpu_oracle.attention_fwd(q, k, v, None, causal)
    assert np.abs(o.to_np() - ref_o).max() <= TOL * np.abs(ref_o).max() and np.abs(lse.to_np() - ref_l).max() <= TOL
    ref = cpu_oracle.attention_bwd(q, k, v, g, None, causal)
    L = _lib.lib()
    for deterministic in (0, 1):
        before = L.ember_set_deterministic(deterministic)
        try:
            got = em.attention_backward(tq, tk, tv, o, lse, tg, None, causal)
        finally:
            L.ember_set_deterministic(before)
        for a, r, name in zip(got, ref, ("dq", "dk", "dv")):
            assert np.abs(a.to_np() - r).max() <= TOL * np.abs(r).max(), (name, deterministic)
