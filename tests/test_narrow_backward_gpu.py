"""Gradients of a float32 layer of few columns in one launch, against float64: edges of the 128-column tiles and of the clusters' rows, every
width, gradients left out, and results that lie over an operand (which take the kernels for each gradient)."""
import ctypes

import numpy as np
import pytest

import ember_b200 as em
from conftest import seeded
from ember_b200 import _lib

pytestmark = pytest.mark.gpu


def _exact(x, w, dy):
    x, w, dy = (a.astype(np.float64) for a in (x, w, dy))
    return dy @ w.T, x.T @ dy, dy.sum(0)


def _close(got, exact, terms, bound):
    # sums of `terms` products in float32, in any order: each addition rounds by 2^-24 of what it has summed up
    assert (np.abs(got - exact) <= terms * 2.0 ** -24 * bound + 1e-30).all()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("m,k", [(1, 4), (31, 128), (33, 132), (65, 124), (256, 784), (511, 260), (1030, 2048), (130, 19204), (70, 38000)])
def test_gradients(m, k, n):
    x, w, dy = seeded((m, k), 1), seeded((k, n), 2, 0.1), seeded((m, n), 3)
    for need_x, need_b in ((True, True), (False, True), (True, False), (False, False)):
        got = em.linear_backward(em.Tensor(x), em.Tensor(w), em.Tensor(dy), need_grad_x=need_x, need_grad_b=need_b)
        ax, aw, ay = np.abs(x).astype(np.float64), np.abs(w).astype(np.float64), np.abs(dy).astype(np.float64)
        bounds = (ay @ aw.T, ax.T @ ay, ay.sum(0))
        for g, e, terms, bound, wanted in zip(got, _exact(x, w, dy), (n, m, m), bounds, (need_x, True, need_b)):
            assert (g is not None) == wanted
            if wanted:
                _close(g.to_np(), e, terms + 1, bound)


def test_rows_past_the_end_are_not_summed():
    # the last rows of a cluster's share are read four at a time; what follows them belongs to the next share, or is not there at all
    m, k, n = 70, 64, 10
    x, w, dy = seeded((m, k), 1), seeded((k, n), 2), seeded((m, n), 3)
    x[41], dy[41] = np.inf, 0.0  # 0 * inf: NaN in every element of grad_w that row 41 belongs to, whatever else is added
    gx, gw, gb = em.linear_backward(em.Tensor(x), em.Tensor(w), em.Tensor(dy))
    assert np.isnan(gw.to_np()).all() and np.isfinite(gx.to_np()).all() and np.isfinite(gb.to_np()).all()


@pytest.mark.parametrize("over", ["x", "dy"])
def test_results_over_operands_keep_their_order(over):
    """grad_x over x or over grad_y (same size here): grad_w and grad_b read both before grad_x is written."""
    m, k, n = 96, 8, 8
    x, w, dy = seeded((m, k), 1), seeded((k, n), 2), seeded((m, n), 3)
    tx, tw, ty = em.Tensor(x), em.Tensor(w), em.Tensor(dy)
    dw, db = em.Tensor.empty((k, n)), em.Tensor.empty((n,))
    dx = tx if over == "x" else ty
    p = lambda t: ctypes.c_void_p(t.ptr)  # noqa: E731
    _lib.check(_lib.lib().ember_linear_bwd(p(tx), p(tw), p(ty), p(dx), p(dw), p(db), m, n, k, 0, 0, 0, 0, 0, None))
    ex, ew, eb = _exact(x, w, dy)
    np.testing.assert_allclose(dx.to_np(), ex, rtol=0, atol=1e-4)
    np.testing.assert_allclose(dw.to_np(), ew, rtol=0, atol=1e-4)
    np.testing.assert_allclose(db.to_np(), eb, rtol=0, atol=1e-4)
