"""Float32 attention on the tensor cores (operands as three bf16 parts): edges of its 128-row blocks and 64-row tiles,
head dimensions that fill the parts' columns partly, rows at any alignment, and the calls that it has to leave to the
CUDA-core kernels (values that the parts cannot hold, no memory for them), against float64.

Tolerance: products of parts leave out less than 2^-24 of a product and the tensor core's additions lose up to 2^-23 each of
a partial sum of 64 terms or fewer (at most 4 additions of full size), partial sums are then added in float32: of a sum of n
terms of order one that is about (4 + sqrt(n / 64)) * 2^-23 of its terms' root sum of squares. 64 * 2^-24 of the largest result
covers n up to 5000 with the exponentials' 2^-22 and a few units for the log-sum-exp."""
import ctypes

import numpy as np
import pytest

import ember_b200 as em
from conftest import Guarded, seeded
from ember_b200 import _lib

pytestmark = pytest.mark.gpu
REL = 64 * 2.0 ** -24


def reference(q, k, v, g, scale, causal):
    q, k, v, g = (x.astype(np.float64) for x in (q, k, v, g))
    s = np.einsum("uid,ujd->uij", q, k) * scale
    if causal:
        s[:, np.triu(np.ones(s.shape[1:], bool), 1 + s.shape[2] - s.shape[1])] = -np.inf
    m = s.max(-1, keepdims=True)
    p = np.exp(s - m)
    lse = (m + np.log(p.sum(-1, keepdims=True)))
    p = np.exp(s - lse)
    o = np.einsum("uij,ujd->uid", p, v)
    ds = p * (np.einsum("uid,ujd->uij", g, v) - (g * o).sum(-1, keepdims=True)) * scale
    return o, lse[..., 0], np.einsum("uij,ujd->uid", ds, k), np.einsum("uij,uid->ujd", ds, q), np.einsum("uij,uid->ujd", p, g)


def run(q, k, v, g, scale, causal):
    tq, tk, tv, tg = (em.Tensor(x[None]) if not isinstance(x, em.Tensor) else x for x in (q, k, v, g))
    o, lse = em.attention_forward(tq, tk, tv, scale, causal)
    grads = em.attention_backward(tq, tk, tv, o, lse, tg, scale, causal)
    return [t.to_np()[0] for t in (o, lse, *grads)]


def on_the_cuda_cores(*args):
    """The same without memory for the parts, and how many of the two calls (forward, backward) asked for it: those on the tensor cores."""
    L = _lib.lib()
    L.ember_selftest_fail_scratch(8)
    got = run(*args)
    return got, 8 - L.ember_selftest_fail_scratch(0)


def inputs(units, lq, lk, d, seed=1, std=0.5):
    return [seeded((units, n, d), seed + i, std) for i, n in enumerate((lq, lk, lk, lq))]


def close(got, want, rel=REL):
    for name, a, b in zip(("o", "lse", "dq", "dk", "dv"), got, want):
        assert np.abs(a - b).max() <= rel * max(1e-30, np.abs(b).max()), name


@pytest.mark.parametrize("units,lq,lk,d,causal", [
    (2, 640, 640, 64, True), (1, 1, 4097, 64, True), (2, 129, 577, 64, False), (1, 511, 513, 64, True), (3, 385, 1025, 64, True),
    (1, 1300, 1290 + 10, 40, False), (2, 200, 1152, 33, True), (1, 600, 1217, 61, False), (1, 1100, 1100, 8, True), (1, 1090, 1090, 3, False),
    (1, 512, 512, 128, True), (2, 127, 641, 128, False), (1, 65, 1023, 80, True), (2, 300, 700, 96, True), (1, 577, 577, 101, False), (1, 640, 576, 72, False),
    (160, 256, 256, 64, True), (40, 256, 256, 128, False), (1, 600, 641, 65, False), (2, 450, 520, 88, True), (1, 513, 600, 97, True),
])
def test_edges_of_blocks_and_tiles(units, lq, lk, d, causal):
    x = inputs(units, lq, lk, d)
    want = reference(*x, d ** -0.5, causal)
    close(run(*x, d ** -0.5, causal), want)
    cores, asked = on_the_cuda_cores(*x, d ** -0.5, causal)
    assert asked == 2
    close(cores, want)


@pytest.mark.parametrize("units,lq,lk,d,causal", [(2, 513, 640, 64, True), (1, 1300, 1300, 40, False), (1, 577, 600, 101, False), (2, 300, 700, 96, True), (1, 1090, 1090, 3, False)])
def test_nothing_is_written_outside_the_results(units, lq, lk, d, causal):
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    dev = torch.device("cuda", 0)
    x = inputs(units, lq, lk, d)
    q, k, v, g = (torch.from_numpy(a).to(dev) for a in x)
    o, lse, dq, dk, dv = (Guarded(torch, shape, torch.float32, dev) for shape in ((units, lq, d), (units, lq), (units, lq, d), (units, lk, d), (units, lk, d)))
    n = L.ember_attention_workspace_bytes(_lib.EMBER_OP_BWD, units, lq, lk, d, 0, 0)
    ws = Guarded(torch, (n,), torch.uint8, dev)
    s = torch.cuda.Stream(device=dev)
    s.wait_stream(torch.cuda.current_stream(dev))
    sp = ctypes.c_void_p(s.cuda_stream)
    ptr = lambda t: (t.t if isinstance(t, Guarded) else t).data_ptr()  # noqa: E731
    _lib.check(L.ember_attention_fwd(*map(ptr, (q, k, v, o, lse)), units, lq, lk, d, d ** -0.5, int(causal), 0, sp))
    _lib.check(L.ember_attention_bwd(*map(ptr, (q, k, v, o, lse, g, dq, dk, dv)), units, lq, lk, d, d ** -0.5, int(causal), 0, ptr(ws), n, sp))
    s.synchronize()
    for t in (o, lse, dq, dk, dv, ws):
        t.check()
    close([t.t.cpu().numpy() for t in (o, lse, dq, dk, dv)], reference(*x, d ** -0.5, causal))


def test_captured_calls():
    """Under stream capture the parts' memory becomes nodes of the graph: replays give the bits of plain calls, on the inputs of the day."""
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    dev = torch.device("cuda", 0)
    units, n, d, m, e = 4, 700, 64, 700, 1024
    q, k, v, g = (torch.empty((units, n, d), device=dev) for _ in range(4))
    x, w, b = torch.empty((m, e), device=dev), torch.empty((e, e), device=dev), torch.empty((e,), device=dev)
    out = [torch.empty((units, n, d), device=dev) for _ in range(4)] + [torch.empty((units, n), device=dev), torch.empty((m, e), device=dev)]
    ws = torch.empty(L.ember_attention_workspace_bytes(_lib.EMBER_OP_BWD, units, n, n, d, 0, 0), device=dev, dtype=torch.uint8)
    s = torch.cuda.Stream(device=dev)

    def calls():
        sp = ctypes.c_void_p(s.cuda_stream)
        o, dq, dk, dv, lse, y = (t.data_ptr() for t in out)
        a = [t.data_ptr() for t in (q, k, v)]
        _lib.check(L.ember_attention_fwd(*a, o, lse, units, n, n, d, 0.125, 1, 0, sp))
        _lib.check(L.ember_attention_bwd(*a, o, lse, g.data_ptr(), dq, dk, dv, units, n, n, d, 0.125, 1, 0, ws.data_ptr(), ws.numel(), sp))
        _lib.check(L.ember_linear_fwd(x.data_ptr(), w.data_ptr(), b.data_ptr(), y, m, e, e, 0, 0, 0, 0, 0, sp))

    def fill(seed):
        gen = torch.Generator(device=dev).manual_seed(seed)
        for t in (q, k, v, g, x, w, b):
            t.normal_(generator=gen)
        torch.cuda.synchronize()

    fill(1)
    calls()
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        calls()
    for seed in (2, 3):
        fill(seed)
        for t in out:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in out]
        calls()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, out))


@pytest.mark.parametrize("d", [64, 96, 40])
@pytest.mark.parametrize("scale", [-0.3, 0.0, 2.0])
def test_any_scale(d, scale):
    x = inputs(2, 600, 700, d)
    close(run(*x, scale, True), reference(*x, scale, True))


@pytest.mark.parametrize("d", [64, 128, 40])
def test_rows_off_the_16_byte_grid(d):
    """Views one element into a buffer: every operand's rows start at odd multiples of 4 bytes."""
    x = inputs(2, 520, 530, d)
    off = []
    for a in x:
        flat = np.concatenate([np.zeros(1, np.float32), a.ravel()])
        off.append(em.Tensor(flat).view(1, (1, *a.shape)))
    close(run(*off, d ** -0.5, True), reference(*x, d ** -0.5, True))


@pytest.mark.parametrize("d", [64, 128])
def test_lengths_of_one_visible_key(d):
    """Row 0 of a square causal call sees one key: its output is that key's value, bit for bit (three parts hold a float32 exactly)."""
    q, k, v, g = inputs(1, 640, 640, d)
    o = run(q, k, v, g, d ** -0.5, True)[0]
    assert np.array_equal(o[0, 0], v[0, 0])


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("which", [0, 1, 2, 3])
@pytest.mark.parametrize("value", [np.inf, np.nan, 3e38])
def test_values_that_the_parts_cannot_hold(d, which, value):
    """One such element anywhere: infinities and NaN where a call without memory for the parts (the CUDA-core kernels alone) has
    them, and the same numbers elsewhere."""
    x = inputs(2, 520, 600, d)
    x[which][1, 300, 5] = value
    got = run(*x, d ** -0.5, False)
    want, asked = on_the_cuda_cores(*x, d ** -0.5, False)
    assert asked == 2
    if value == 3e38:  # times score gradients that are nothing but the rounding of what cancels there: not dq and dk
        got, want = ([t[0], t[1], t[4]] for t in (got, want))
    for a, b in zip(got, want):
        fine = np.isfinite(b)
        assert np.array_equal(fine, np.isfinite(a)) and np.array_equal(a[~fine], b[~fine], equal_nan=True)
        for u in range(2):  # the element's own unit by its own largest value
            f = fine[u]
            assert not f.any() or np.abs(a[u][f].astype(np.float64) - b[u][f]).max() <= REL * np.abs(b[u][f].astype(np.float64)).max()


@pytest.mark.parametrize("d", [64, 128])
def test_tensors_of_tiny_values_keep_their_precision(d):
    """Upstream gradients of 1e-33: their low parts would fall under bf16's smallest values."""
    q, k, v, g = inputs(2, 520, 600, d)
    g *= np.float32(2e-33)
    close(run(q, k, v, g, d ** -0.5, False), reference(q, k, v, g, d ** -0.5, False))


def peaked(units, lq, lk, d, size):
    """q and k of elements of +-size, query i along key i + lk - lq."""
    rng = np.random.default_rng(5)
    k = np.where(rng.standard_normal((units, lk, d)) < 0, -1, 1) * rng.uniform(0.75, 1.25, (units, lk, d)) * size
    k = k.astype(np.float32)
    return (k[:, lk - lq:] * np.float32(1.37)).astype(np.float32), k


@pytest.mark.parametrize("units,lq,lk,d", [(2, 520, 600, 64), (2, 520, 600, 128), (1, 600, 600, 40), (1, 200, 512, 64), (64, 128, 128, 64)])
@pytest.mark.parametrize("size", [10.0, 30.0, 1e3, 1e5, 1e8, 4e14])
def test_large_scores_leave_the_largest_a_weight_of_one(units, lq, lk, d, size):
    """Elements of +-size: query i scores about twice what any other key gets with key i + lk - lq, whose weight is 1 to the last bit where forward
    and backward round scores alike. That key's value is the output, its gradient the upstream gradient. Scores' rounding errors may reach
    the weight where the two run on different kernels, up to the 2^12 at which those calls stay on the CUDA cores: 2^-10 then (a few units
    of 2^-23 of a score)."""
    q, k = peaked(units, lq, lk, d, size)
    v, g = seeded((units, lk, d), 2), seeded((units, lq, d), 3)
    scale = 0.25 if d == 40 else 0.125
    s = (q[0].astype(np.float64) @ k[0].T.astype(np.float64)) * scale
    best = s[np.arange(lq), np.arange(lq) + lk - lq]
    s[np.arange(lq), np.arange(lq) + lk - lq] = -np.inf
    assert (best - s.max(1)).min() > 40
    o, lse, dq, dk, dv = run(q, k, v, g, scale, False)
    rel = 2.0 ** -10 if units == 64 or lq == 200 else 2.0 ** -20
    assert np.abs(o - v[:, lk - lq:]).max() <= 2.0 ** -20 * np.abs(v).max()
    assert np.abs(lse[0] - best).max() <= 2.0 ** -20 * best.max()
    assert np.abs(dv[:, lk - lq:] - g).max() <= rel * np.abs(g).max()
    assert np.isfinite(dq).all() and np.isfinite(dk).all()


@pytest.mark.parametrize("d", [64, 128, 40])
def test_tiny_rows_keep_their_precision(d):
    """A row of upstream gradients, one of values and a key whose every weight is about e^-85, far below the rest: each row of results that
    they alone make by its own largest value. 2^-14 for the key: its scores' rounding errors, 85 * 2^-23 each, reach its weights."""
    q, k, v, g = inputs(2, 520, 600, d)
    g[1, 5] *= np.float32(2e-37)
    q[:, :, 0], k[0, 9] = 4, 0
    k[0, 9, 0] = -79 / (4 * d ** -0.5)
    o, lse, dq, dk, dv = run(q, k, v, g, d ** -0.5, False)
    ro, rl, rq, rk, rv = reference(q, k, v, g, d ** -0.5, False)
    for a, b, rel in ((dq[1, 5], rq[1, 5], REL), (dv[0, 9], rv[0, 9], 2.0 ** -14), (o, ro, REL), (dk, rk, REL)):
        assert np.abs(a - b).max() <= rel * np.abs(b).max()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("sizes", [(1, 1, 1e-18, 1e-18), (1e-18, 1e15, 1e-10, 1e-20), (1, 1, 1e-30, 1e5), (1e6, 1e-7, 1e7, 1e7), (1, 1, 1, 1e-33)])
def test_sizes_of_the_tensors(d, sizes):
    """Score gradients near both ends of float32."""
    q, k, v, g = (a * np.float32(s) for a, s in zip(inputs(2, 520, 600, d), sizes))
    for a, b in zip(run(q, k, v, g, d ** -0.5, True), reference(q, k, v, g, d ** -0.5, True)):
        assert np.abs(a - b).max() <= REL * np.abs(b).max() + 2.0 ** -140  # 2^9 of the smallest float32


@pytest.mark.parametrize("d", [64, 96, 128])
def test_scores_of_one_sign(d):
    """Nonnegative q and k: every truncation of a score's partial sums is in one direction. An accumulator of 64 terms takes four additions of
    full size, at 1/4 to 4/4 of its sum, which lose half a unit of 2^-23 at most on average: 2.5 * 2^-24 of a score."""
    q, k, v, g = (np.abs(a) for a in inputs(4, 1024, 1024, d, std=1.0))
    lse = run(q, k, v, g, d ** -0.5, False)[1]
    want = reference(q, k, v, g, d ** -0.5, False)[1]
    score = np.einsum("uid,ud->ui", q.astype(np.float64), k.astype(np.float64).mean(1)) * d ** -0.5
    assert np.sqrt(((lse - want) ** 2).mean()) <= 2.5 * 2.0 ** -24 * np.sqrt((score ** 2).mean())


@pytest.mark.parametrize("n", [256, 600])
@pytest.mark.parametrize("size", [10.0, 30.0, 1e5])
def test_large_scores_with_the_units_in_pieces(n, size):
    """Forward one unit a call, backward all of them, which may go to different kernels: as above, 2^-10 of the scores' rounding errors up to
    2^12, none beyond it nor where both directions take the same kernels whatever the number of units."""
    units, d = 32, 64
    q, k = peaked(units, n, n, d, size)
    v, g = seeded((units, n, d), 2), seeded((units, n, d), 3)
    pieces = [[t.to_np() for t in em.attention_forward(*(em.Tensor(x[None, u:u + 1]) for x in (q, k, v)), 0.125, False)] for u in range(units)]
    o, lse = (em.Tensor(np.concatenate([p[i] for p in pieces], 1)) for i in range(2))
    dv = em.attention_backward(*(em.Tensor(x[None]) for x in (q, k, v)), o, lse, em.Tensor(g[None]), 0.125, False)[2].to_np()[0]
    assert np.abs(o.to_np()[0] - v).max() <= 2.0 ** -20 * np.abs(v).max()
    assert np.abs(dv - g).max() <= (2.0 ** -10 if n == 256 and size == 10 else 2.0 ** -20) * np.abs(g).max()


def test_zeros_stay_on_the_tensor_cores_and_give_means():
    q, k, v, g = inputs(2, 520, 600, 64)
    q[:] = 0
    close(run(q, k, v, g, 0.125, False), reference(q, k, v, g, 0.125, False))


def test_without_memory_for_the_parts():
    x = inputs(2, 600, 600, 64)
    got, asked = on_the_cuda_cores(*x, 0.125, True)
    assert asked == 2
    close(got, reference(*x, 0.125, True))


@pytest.mark.parametrize("d", [64, 128])
def test_results_repeat_bit_for_bit(d):
    x = inputs(3, 700, 900, d)
    first = run(*x, d ** -0.5, True)
    for _ in range(3):
        assert all(np.array_equal(a, b) for a, b in zip(first, run(*x, d ** -0.5, True)))
