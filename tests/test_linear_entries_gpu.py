"""Projections whose head-major operand has sequences that are no multiple of the 128-row tiles (64-row
contraction steps in the weight gradient), on the tensor-core kernel, against the CPU oracle: one row past a
tile, one short of it, entries shorter than a tile, the shortest that the rule lets through, and a
non-finite element in the last row of an entry.

Tolerance: bfloat16 results, half a unit in the last place (2^-9 of the value) plus the float32 sum's rounding."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import bf16_round, seeded
from ember_b200 import _lib
from oracle import cpu_oracle

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -8


def heads_first(a, batch, seq, parts, heads, dim):
    return np.ascontiguousarray(a.reshape(batch, seq, parts, heads, dim).transpose(2, 0, 3, 1, 4))


def close(got, ref, name):
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max(), name


@pytest.mark.parametrize("batch,seq,heads,dim", [(1, 129, 2, 64), (2, 127, 1, 128), (3, 40, 2, 64), (20, 8, 1, 64), (2, 65, 3, 128),
                                                 (4, 200, 2, 64), (2, 500, 4, 64), (1, 257, 2, 128), (3, 64, 2, 64)])
def test_both_projections_of_a_block(batch, seq, heads, dim):
    m, e = batch * seq, heads * dim
    for x_heads, y_heads, n in ((0, heads, 3 * e), (heads, 0, e)):
        if m > 128:
            assert _lib.lib().ember_linear_kernel_name(0, m, n, e, _lib.EMBER_BF16, x_heads, y_heads, seq, dim) == b"sm100_tcgen05"
        x, w, b, g = (bf16_round(seeded(s, i)) for i, s in enumerate(((m, e), (e, n), (n,), (m, n)), 1))
        lay_x = (lambda a: heads_first(a, batch, seq, 1, heads, dim)[0]) if x_heads else (lambda a: a.reshape(batch, seq, -1))
        lay_y = (lambda a: heads_first(a, batch, seq, n // e, heads, dim)) if y_heads else (lambda a: a.reshape(batch, seq, -1))
        tx, tw, tb, tg = (em.Tensor(a, "bfloat16") for a in (lay_x(x), w, b, lay_y(g)))
        close(em.linear_forward(tx, tw, tb, x_heads=x_heads, y_heads=y_heads).to_np(), lay_y(cpu_oracle.linear_fwd(x, w, b)), "y")
        rx, rw, rb = cpu_oracle.linear_bwd(x, w, g)
        for got, ref, name in zip(em.linear_backward(tx, tw, tg, x_heads=x_heads, y_heads=y_heads), (lay_x(rx), rw, rb), ("grad_x", "grad_w", "grad_b")):
            close(got.to_np().reshape(ref.shape), ref, name)


def test_an_infinity_stays_in_its_row_and_column():
    """The boxes past an entry's end read zeros for both operands: an infinity in the next entry's first row
    must not meet the padding of this one's."""
    batch, seq, heads, dim = 2, 70, 1, 64
    m, e = batch * seq, heads * dim
    x, w, g = (bf16_round(seeded(s, i)) for i, s in enumerate(((m, e), (e, 3 * e), (m, 3 * e)), 1))
    x[seq, 5] = np.inf
    g[seq] = np.abs(g[seq]) + 1
    tx, tw = em.Tensor(x.reshape(batch, seq, e), "bfloat16"), em.Tensor(w, "bfloat16")
    tg = em.Tensor(heads_first(g, batch, seq, 3, heads, dim), "bfloat16")
    _, gw, _ = em.linear_backward(tx, tw, tg, y_heads=heads)
    gw = gw.to_np()
    assert np.all(gw[5] == np.inf) and np.isfinite(np.delete(gw, 5, 0)).all()
    y = em.linear_forward(tx, tw, None, y_heads=heads).to_np().transpose(1, 3, 0, 2, 4).reshape(m, 3 * e)
    assert not np.isfinite(y[seq]).any() and np.isfinite(np.delete(y, seq, 0)).all()


def test_chained_launches_see_each_other():
    """Kernels of a chain start while the one before drains: a block's passes repeated on the same buffers, each
    reading what the launch before wrote and writing what it read, give the same bits as with a wait after each."""
    block = em.nn.MultiHeadAttention(256, 4, causal=True, dtype="bfloat16", seed=1)
    x = em.Tensor(bf16_round(seeded((2, 190, 256), 1)), "bfloat16")
    L = _lib.lib()
    before = L.ember_set_deterministic(1)
    try:
        results = []
        for wait in (True, False, False):
            y, grads = x, []
            for _ in range(6):
                y = block(y)
                if wait:
                    y.to_np()
                g = block.backward(y)
                if wait:
                    g.to_np()
                grads += [g, *block.gradients()]
            results.append([y.to_np()] + [t.to_np() for t in grads])
    finally:
        L.ember_set_deterministic(before)
    for other in results[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(results[0], other))
