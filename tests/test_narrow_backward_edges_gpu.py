"""Gradients of a float32 layer of few columns where its one launch can go wrong: infinities in the last rows of a block's share, results between guard
bands, both sides of every line of the rule that chooses it, tall and wide layers whose blocks share no rows, a caller's stream and a captured graph."""
import ctypes

import numpy as np
import pytest

import ember_b200 as em
from conftest import Guarded, seeded
from ember_b200 import _lib

pytestmark = pytest.mark.gpu


def _call(torch, x, w, dy, dx, dw, db, stream):
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())  # noqa: E731
    (m, k), n = x.shape, w.shape[1]
    _lib.check(_lib.lib().ember_linear_bwd(p(x), p(w), p(dy), p(dx), p(dw), p(db), m, n, k, _lib.EMBER_F32, 0, 0, 0, 0, ctypes.c_void_p(stream.cuda_stream)))


@pytest.fixture
def gpu():
    torch = pytest.importorskip("torch")
    _lib.check(_lib.lib().ember_set_device(0))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        yield torch, stream
    torch.cuda.synchronize()


def _inputs(torch, m, k, n):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    new = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    return new(m, k), 0.1 * new(k, n), new(m, n)


def _check(x, w, dy, dx, dw, db, sums):
    x, w, dy = x.double(), w.double(), dy.double()
    m, n = dy.shape
    # sums of products in float32: `sums` (or n, or m) roundings of up to the sum of the magnitudes by 2^-24 each, and the result's own
    for got, exact, size, terms in ((dx, dy @ w.T, dy.abs() @ w.abs().T, n), (dw, x.T @ dy, x.abs().T @ dy.abs(), sums), (db, dy.sum(0), dy.abs().sum(0), m)):
        if got is not None:
            assert bool(((got - exact).abs() <= (terms + 1) * 2.0 ** -24 * size + 1e-30).all())


@pytest.mark.parametrize("row", [34, 35, 69])
def test_infinity_at_the_end_of_a_share(row):
    # 70 rows are shared by two blocks, [0, 35) and [35, 70); warps read four at a time, the last ones again past the end
    m, k, n, c = 70, 64, 10, 3
    x, w, dy = seeded((m, k), 1), seeded((k, n), 2), seeded((m, n), 3)
    dy[row, c] = np.inf
    gx, gw, gb = (t.to_np() for t in em.linear_backward(em.Tensor(x), em.Tensor(w), em.Tensor(dy)))
    assert np.array_equal(gw[:, c], np.sign(x[row]) * np.inf) and gb[c] == np.inf and np.array_equal(gx[row], np.sign(w[:, c]) * np.inf)
    rest, rows = np.arange(n) != c, np.arange(m) != row
    np.testing.assert_allclose(gw[:, rest], (x.T.astype(np.float64) @ dy[:, rest]), rtol=0, atol=m * 2.0 ** -24 * (np.abs(x).T @ np.abs(dy[:, rest])).max())
    np.testing.assert_allclose(gb[rest], dy[:, rest].astype(np.float64).sum(0), rtol=1e-6, atol=1e-6)
    np.testing.assert_allclose(gx[rows], dy[rows].astype(np.float64) @ w.T, rtol=0, atol=n * 2.0 ** -24 * (np.abs(dy[rows]) @ np.abs(w).T).max())


@pytest.mark.parametrize("n", [1, 5, 7, 8, 12])
@pytest.mark.parametrize("m,k", [(1, 4), (33, 124), (70, 132), (130, 260), (300, 1028)])
def test_nothing_is_written_outside_the_results(gpu, m, k, n):
    torch, stream = gpu
    x, w, dy = _inputs(torch, m, k, n)
    got = [Guarded(torch, s, torch.float32, "cuda") for s in ((m, k), (k, n), (n,))]
    _call(torch, x, w, dy, *(g.t for g in got), stream)
    stream.synchronize()
    for g, name in zip(got, ("grad_x", "grad_w", "grad_b")):
        g.check(name)
    _check(x, w, dy, *(g.t for g in got), m)


# rows to 16384; with 8 and 12 columns to 4096 where there are fewer than 512 inputs, and without grad_x more than 16 above 32768 inputs; 12 columns and
# grad_w alone
@pytest.mark.parametrize("m,k,n,need", [
    (16384, 64, 5, "xb"), (16385, 64, 5, "xb"), (4096, 508, 8, "xb"), (4097, 508, 8, "xb"), (4097, 512, 8, "xb"), (4097, 508, 12, "x"), (4097, 508, 9, "b"),
    (16, 32768, 8, "b"), (16, 32772, 8, "b"), (17, 32772, 8, "b"), (16, 32772, 8, "xb"), (16, 32772, 12, ""), (17, 32772, 12, "b"), (95, 220, 12, ""), (95, 222, 11, "xb")])
def test_both_sides_of_the_rule(gpu, m, k, n, need):
    torch, stream = gpu
    x, w, dy = _inputs(torch, m, k, n)
    dx, dw, db = torch.empty_like(x) if "x" in need else None, torch.empty_like(w), torch.empty(n, device="cuda") if "b" in need else None
    _call(torch, x, w, dy, dx, dw, db, stream)
    stream.synchronize()
    _check(x, w, dy, dx, dw, db, m)


@pytest.mark.parametrize("m,k,n", [(2048, 38000, 3), (1030, 40004, 12)])
def test_tall_and_wide(gpu, m, k, n):
    # more than two tiles of 128 columns an SM: a block has all rows, a warp every eighth four of them, which are added up before they meet its sums
    torch, stream = gpu
    x, w, dy = _inputs(torch, m, k, n)
    dx, dw, db = torch.empty_like(x), torch.empty_like(w), torch.empty(n, device="cuda")
    _call(torch, x, w, dy, dx, dw, db, stream)
    stream.synchronize()
    _check(x, w, dy, dx, dw, db, (m + 31) // 32 + 4 + 3)


def test_captured_and_replayed_on_new_values(gpu):
    torch, stream = gpu
    m, k, n = 256, 784, 10
    x, w, dy = _inputs(torch, m, k, n)
    dx, dw, db = torch.empty_like(x), torch.empty_like(w), torch.empty(n, device="cuda")
    _call(torch, x, w, dy, dx, dw, db, stream)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        dy.mul_(0.5)  # a kernel before, and what it writes is what the gradients are of
        _call(torch, x, w, dy, dx, dw, db, stream)
        total = dx.sum(1)  # a kernel behind
    for seed in (1, 2):
        x.copy_(torch.randn(m, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)))
        graph.replay()
        stream.synchronize()
        _check(x, w, dy, dx, dw, db, m)
        assert bool(torch.equal(total, dx.sum(1)))
