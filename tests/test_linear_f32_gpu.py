"""Float32 Linear products on the tensor cores (operands as three bf16 planes): edges of the 256-row tiles, of both tile widths and of
the contraction's parts, rows that are no multiple of 8 columns, head-major operands, and the calls left to the
CUDA-core kernel, against float64.

Tolerance: 1e-5 of the largest result, as for the CUDA-core products: partial sums of 64 terms carry up to 4 truncations of 2^-23,
adding k / 64 of them in float32 sqrt(k / 64) * 2^-24 of the terms, products of planes leave out less than 2^-24."""
import ctypes

import numpy as np
import pytest

import ember_b200 as em
from conftest import Guarded, seeded
from ember_b200 import _lib

pytestmark = pytest.mark.gpu


def kernels(m, n, k, *layout):
    """Which kernels take the three products: "t" the tensor cores, "s" the CUDA cores."""
    name = _lib.lib().ember_linear_kernel_name
    return "".join({b"sm100_tcgen05": "t", b"simt_f32": "s"}[name(p, m, n, k, _lib.EMBER_F32, *(layout or (0, 0, 0, 0)))] for p in range(3))


def check(m, n, k, x=None, w=None, b=None, g=None, tol=1e-5):
    x, w, b, g = (a if a is not None else seeded(s, i) for i, (a, s) in enumerate(((x, (m, k)), (w, (k, n)), (b, (n,)), (g, (m, n))), 1))
    tx, tw, tb, tg = (em.Tensor(a) for a in (x, w, b, g))
    got = [t.to_np() for t in (em.linear_forward(tx, tw, tb), *em.linear_backward(tx, tw, tg))]
    x, w, b, g = (a.astype(np.float64) for a in (x, w, b, g))
    for name, a, r in zip(("y", "grad_x", "grad_w", "grad_b"), got, (x @ w + b, g @ w.T, x.T @ g, g.sum(0))):
        assert np.abs(a - r).max() <= tol * np.abs(r).max(), name
    return got


@pytest.mark.parametrize("m,n,k", [(768, 512, 512), (513, 768, 1032), (255, 1000, 2048), (257, 1024, 1023), (1000, 1001, 1025), (2049, 520, 515),
                                   (300, 4097, 700), (4096, 384, 640), (700, 2056, 1030), (8192, 129, 1024), (2300, 2310, 2320),
                                   (3000, 72, 4000), (6000, 640, 200)])
def test_edges(m, n, k):
    assert kernels(m, n, k) == "ttt"
    check(m, n, k)


@pytest.mark.parametrize("batch,seq,heads,dim", [(2, 512, 8, 64), (3, 300, 4, 128), (8, 129, 8, 64), (1, 1000, 16, 64), (20, 40, 12, 64)])
def test_head_major_operands(batch, seq, heads, dim):
    m, e = batch * seq, heads * dim
    assert kernels(m, 3 * e, e, 0, heads, seq, dim) == "ttt" and kernels(m, e, e, heads, 0, seq, dim) == "ttt"
    x, g3, g1 = seeded((batch, seq, e), 1), seeded((3, batch, heads, seq, dim), 2), seeded((batch, seq, e), 3)
    w3, b3, w1 = seeded((e, 3 * e), 4), seeded((3 * e,), 5), seeded((e, e), 6)
    o = seeded((batch, heads, seq, dim), 7)
    rows = lambda a: a.astype(np.float64).reshape(-1, batch, heads, seq, dim).transpose(1, 3, 0, 2, 4).reshape(m, -1)  # noqa: E731
    y = em.linear_forward(em.Tensor(x), em.Tensor(w3), em.Tensor(b3), y_heads=heads).to_np()
    grads = [t.to_np() for t in em.linear_backward(em.Tensor(x), em.Tensor(w3), em.Tensor(g3), y_heads=heads)]
    y1 = em.linear_forward(em.Tensor(o), em.Tensor(w1), None, x_heads=heads).to_np()
    grads1 = [t.to_np() for t in em.linear_backward(em.Tensor(o), em.Tensor(w1), em.Tensor(g1), x_heads=heads)]
    x64, w3d, w1d, g = x.reshape(m, e).astype(np.float64), w3.astype(np.float64), w1.astype(np.float64), rows(g3)
    g1d, o64 = g1.reshape(m, e).astype(np.float64), rows(o)
    for a, r in ((rows(y), x64 @ w3d + b3), (grads[0].reshape(m, e), g @ w3d.T), (grads[1], x64.T @ g), (grads[2], g.sum(0)),
                 (y1.reshape(m, e), o64 @ w1d), (rows(grads1[0]), g1d @ w1d.T), (grads1[1], o64.T @ g1d)):
        assert np.abs(a - r).max() <= 1e-5 * np.abs(r).max()


@pytest.mark.parametrize("m,n,k", [(1, 64, 64), (3, 68, 65), (4, 1000, 512), (5, 64, 2048), (8, 1540, 100), (9, 204, 8192), (13, 2048, 513), (16, 6144, 1030), (16, 64, 1023), (2, 4100, 4099),
                                   (1, 8192, 8192), (16, 4096, 512), (12, 512, 100), (16, 2048, 100), (11, 516, 127), (9, 128, 200)])
def test_few_rows(m, n, k):
    """The kernel that streams w: every number of rows' form, contractions that leave rounds and the cluster's parts uneven."""
    check(m, n, k)


def test_one_hot_rows_pick_rows_of_w_bit_for_bit():
    """Three planes hold a float32 exactly, and so does the sum of its products with one."""
    w = seeded((1024, 1032), 1)
    x = np.zeros((600, 1024), np.float32)
    x[np.arange(600), (7 * np.arange(600)) % 1024] = 1
    assert np.array_equal(em.linear_forward(em.Tensor(x), em.Tensor(w), None).to_np(), w[(7 * np.arange(600)) % 1024])


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 2e38])
@pytest.mark.parametrize("where", ["x", "w", "g"])
def test_values_that_the_planes_cannot_hold(where, value):
    """They reach the results they belong to and no others, and nothing else loses precision."""
    m, n, k = 520, 1000, 1024
    a = {"x": seeded((m, k), 1), "w": seeded((k, n), 2), "g": seeded((m, n), 3)}
    a[where][7, 9] = value
    tx, tw, tg = (em.Tensor(a[i]) for i in "xwg")
    got = [t.to_np() for t in (em.linear_forward(tx, tw, None), *em.linear_backward(tx, tw, tg, need_grad_b=False)[:2])]
    x, w, g = (a[i].astype(np.float64) for i in "xwg")
    with np.errstate(all="ignore"):
        for q, r in zip(got, (x @ w, g @ w.T, x.T @ g)):
            near = np.abs(np.abs(r) / np.finfo(np.float32).max - 1) < 1e-3  # whose rounding decides
            r = np.where(np.abs(r) > np.finfo(np.float32).max, np.sign(r) * np.inf, r)
            fine = np.isfinite(r)
            assert np.array_equal(np.isfinite(q)[~near], fine[~near]) and np.array_equal(q[~fine & ~near], r[~fine & ~near].astype(np.float32), equal_nan=True)
            small = np.abs(r) < 1e6
            assert np.abs(q[small] - r[small]).max() <= 1e-5 * np.abs(r[small]).max()


def test_tiny_values_keep_their_precision():
    check(520, 1000, 1024, x=seeded((520, 1024), 1) * np.float32(1e-33))


def test_tiny_rows_and_columns_keep_their_precision():
    """A row of x, one of g and a column of w far below the rest, down to where bf16 has no digits left: each result by its own largest value."""
    for size in (1e-33, 1e-36, 1e-38):
        x, w, g = seeded((520, 1024), 1), seeded((1024, 1000), 2), seeded((520, 1000), 3)
        x[7] *= np.float32(size)
        g[5] *= np.float32(size)
        w[:, 11] *= np.float32(size)
        y, gx, gw = (t.to_np() for t in (em.linear_forward(em.Tensor(x), em.Tensor(w), None), *em.linear_backward(em.Tensor(x), em.Tensor(w), em.Tensor(g), need_grad_b=False)[:2]))
        x, w, g = (a.astype(np.float64) for a in (x, w, g))
        for a, r in ((y[7], np.delete(x[7] @ w, 11)), (np.delete(y[:, 11], 7), np.delete(x, 7, 0) @ w[:, 11]), (gx[5], g[5] @ w.T), (gw, x.T @ g)):
            a = np.delete(a, 11) if a.shape == (1000,) else a
            assert np.abs(a - r).max() <= 1e-5 * np.abs(r).max()


@pytest.mark.parametrize("m,n,k", [(8192, 1000, 64), (512, 50000, 96)])
def test_sums_of_one_sign(m, n, k):
    """Nonnegative operands: every truncation is in one direction. An accumulator of 64 terms takes four additions of full size, at 1/4 to 4/4
    of its sum, that lose half a unit of 2^-23 at most on average: 2.5 * 2^-24."""
    assert kernels(m, n, k)[0] == "t"
    x, w = np.abs(seeded((m, k), 1)), np.abs(seeded((k, n), 2))
    y = em.linear_forward(em.Tensor(x), em.Tensor(w), None).to_np()[::16]
    r = x[::16].astype(np.float64) @ w.astype(np.float64)
    assert np.sqrt(((y / r - 1) ** 2).mean()) <= 2.5 * 2.0 ** -24


def test_small_products_keep_their_precision():
    """Operands of 1e-18: their products are near the smallest float32, those of their parts below it."""
    x, w = seeded((520, 1024), 1) * np.float32(1e-18), seeded((1024, 1000), 2) * np.float32(1e-18)
    r = x.astype(np.float64) @ w.astype(np.float64)
    assert np.abs(em.linear_forward(em.Tensor(x), em.Tensor(w), None).to_np() - r).max() <= 1e-5 * np.abs(r).max()


def test_without_memory_for_the_planes():
    L = _lib.lib()
    L.ember_selftest_fail_scratch(2)
    check(520, 1000, 1024)
    assert L.ember_selftest_fail_scratch(0) == 0


@pytest.mark.parametrize("m,n,k", [(513, 768, 1032), (1000, 1001, 1025), (300, 4097, 700), (3000, 72, 4000), (2049, 520, 515), (13, 2048, 513), (16, 4100, 512), (3, 68, 65)])
def test_nothing_is_written_outside_the_results(m, n, k):
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    dev = torch.device("cuda", 0)
    x, w, b, g = (torch.from_numpy(seeded(shape, i)).to(dev) for i, shape in enumerate(((m, k), (k, n), (n,), (m, n)), 1))
    y, gx, gw, gb = (Guarded(torch, shape, torch.float32, dev) for shape in ((m, n), (m, k), (k, n), (n,)))
    s = torch.cuda.Stream(device=dev)
    s.wait_stream(torch.cuda.current_stream(dev))
    sp = ctypes.c_void_p(s.cuda_stream)
    _lib.check(L.ember_linear_fwd(x.data_ptr(), w.data_ptr(), b.data_ptr(), y.t.data_ptr(), m, n, k, 0, 0, 0, 0, 0, sp))
    _lib.check(L.ember_linear_bwd(x.data_ptr(), w.data_ptr(), g.data_ptr(), gx.t.data_ptr(), gw.t.data_ptr(), gb.t.data_ptr(), m, n, k, 0, 0, 0, 0, 0, sp))
    s.synchronize()
    for name, t, r in (("y", y, x.double() @ w.double() + b.double()), ("grad_x", gx, g.double() @ w.double().T), ("grad_w", gw, x.double().T @ g.double()), ("grad_b", gb, g.double().sum(0))):
        t.check(name)
        assert (t.t.double() - r).abs().max() <= 1e-5 * r.abs().max(), name


def test_results_repeat_bit_for_bit():
    first = check(3000, 200, 2048)
    for _ in range(3):
        assert all(np.array_equal(a, b) for a, b in zip(first, check(3000, 200, 2048)))
