"""Float32 attention at the edges of its kernels' tiles, against the CPU oracle. The units and lengths
put the launch in each of its row-per-thread forms (a few long rows to many short ones), the lengths
leave remainders of one row and one short of a tile, and the head dimensions fill 32, 64 and 128
columns exactly, partly, and with rows that are no whole number of 16-byte pieces.

Tolerance: a result is a chain of sums of n = lk (or d) float32 terms; with operands of order one the
rounding of such a sum is about sqrt(n) * 2^-24 of its terms' root sum of squares, so 64 * 2^-24 of the
largest reference magnitude covers n up to a thousand with room for the exponentials' 2^-22."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import seeded
from oracle import cpu_oracle

pytestmark = pytest.mark.gpu

REL = 64 * 2.0 ** -24


@pytest.mark.parametrize("units,lq,lk,d,causal", [
    (1, 1, 1, 4, False), (2, 15, 17, 32, True), (3, 65, 129, 33, False), (2, 64, 64, 64, True), (1, 127, 200, 128, False),
    (80, 97, 97, 64, True), (80, 129, 63, 36, False), (40, 257, 257, 128, True),
    (80, 191, 193, 64, False), (80, 193, 193, 20, True),
])
def test_float32_tiles_match_the_oracle(units, lq, lk, d, causal):
    q, k, v = (seeded((1, units, n, d), s) for n, s in ((lq, 1), (lk, 2), (lk, 3)))
    g = seeded((1, units, lq, d), 4)
    tq, tk, tv, tg = (em.Tensor(x) for x in (q, k, v, g))
    o, lse = em.attention_forward(tq, tk, tv, None, causal)
    grads = em.attention_backward(tq, tk, tv, o, lse, tg, None, causal)
    ro, rl = cpu_oracle.attention_fwd(q, k, v, None, causal)
    ref = (ro, rl, *cpu_oracle.attention_bwd(q, k, v, g, None, causal))
    for name, got, want in zip(("o", "lse", "dq", "dk", "dv"), (o, lse, *grads), ref):
        assert np.abs(got.to_np() - want).max() <= REL * max(1.0, np.abs(want).max()), name
