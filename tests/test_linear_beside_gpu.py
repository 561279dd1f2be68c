"""Both gradients and the bias gradient of one call run side by side on the GPU: the bits of three calls, call after call, with results that
lie over one another's operands kept in order, and with what follows on the stream waiting for all of them."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import bf16_round, seeded
from ember_b200 import _lib

pytestmark = pytest.mark.gpu

BF16 = 1


def bwd(x, w, g, dx, dw, db, m, n, k, heads=(0, 0, 0, 0)):
    at = lambda t: t.ptr if t is not None else None  # noqa: E731
    _lib.check(_lib.lib().ember_linear_bwd(at(x), at(w), at(g), at(dx), at(dw), at(db), m, n, k, BF16, *heads, None))


# rows x inputs x outputs: one tile, several per pair, more pairs than tiles, both last rounds ragged, odd rows of results; then
# (x_heads, y_heads, sequence, head dimension) as a block's projections have them, sequences of whole tiles and of others
@pytest.mark.parametrize("m,k,n,heads", [
    *((m, k, n, (0, 0, 0, 0)) for m, k, n in [(256, 256, 256), (300, 264, 520), (8192, 256, 768), (2048, 2048, 2048), (4104, 1544, 4616), (1000, 512, 1536), (2048, 128, 8192)]),
    (1024, 512, 1536, (0, 4, 256, 128)), (1542, 2048, 6144, (0, 16, 1542, 128)), (2208, 1024, 3072, (0, 16, 69, 64)), (6000, 1024, 3072, (0, 16, 375, 64)),
    (1024, 512, 512, (4, 0, 512, 128)), (264, 1024, 1024, (8, 0, 24, 128)), (2208, 1024, 1024, (8, 0, 69, 128)), (4224, 512, 512, (8, 0, 1408, 64))])
def test_side_by_side_is_one_after_the_other(m, k, n, heads):
    x, w, g = (em.Tensor(bf16_round(seeded(s, i)), "bfloat16") for i, s in enumerate([(m, k), (k, n), (m, n)]))
    new = lambda: [em.Tensor.empty(s, "bfloat16") for s in [(m, k), (k, n), (n,)]]  # noqa: E731
    dx, dw, db = new()
    bwd(x, w, g, dx, None, None, m, n, k, heads)
    bwd(x, w, g, None, dw, None, m, n, k, heads)
    bwd(x, w, g, None, None, db, m, n, k, heads)
    want = [t.to_np() for t in (dx, dw, db)]
    for asked in ((1, 1, 1), (1, 1, 0), (0, 1, 1)) * 2:
        outs = [t if a else None for t, a in zip(new(), asked)]
        bwd(x, w, g, *outs, m, n, k, heads)
        for a, b in zip(outs, want):
            assert a is None or np.array_equal(a.to_np(), b)
    # a chain in which every call reads what the one before it wrote, nothing waited for in between
    ys = [x]
    for _ in range(4):
        outs = new()
        bwd(ys[-1], w, g, *outs, m, n, k, heads)
        ys.append(outs[0])
        last = outs
    assert np.array_equal(last[0].to_np(), want[0]) and np.array_equal(last[2].to_np(), want[2])
    ref = new()
    bwd(dx, w, g, None, ref[1], None, m, n, k, heads)
    assert np.array_equal(last[1].to_np(), ref[1].to_np())


@pytest.mark.parametrize("m,k,n", [(4104, 1544, 4616), (1000, 512, 1536), (1024, 512, 32768), (777, 264, 1008)])
def test_grad_y_rewritten_just_before(m, k, n):
    """grad_y comes into the same buffer from a product launched right before each call, other values every time."""
    L = _lib.lib()
    x, w = em.Tensor(bf16_round(seeded((m, k), 1)), "bfloat16"), em.Tensor(bf16_round(seeded((k, n), 2)), "bfloat16")
    a = [em.Tensor(bf16_round(seeded((m, 64), 10 + i)), "bfloat16") for i in range(6)]
    b = em.Tensor(bf16_round(seeded((64, n), 3)), "bfloat16")
    g = em.Tensor.empty((m, n), "bfloat16")
    new = lambda: [em.Tensor.empty(s, "bfloat16") for s in [(m, k), (k, n), (n,)]]  # noqa: E731
    fill = lambda t: _lib.check(L.ember_linear_fwd(t.ptr, b.ptr, None, g.ptr, m, n, 64, BF16, 0, 0, 0, 0, None))  # noqa: E731
    got = [new() for _ in a]
    for t, outs in zip(a, got):
        fill(t)
        bwd(x, w, g, *outs, m, n, k)
    got = [[t.to_np() for t in outs] for outs in got]
    for t, outs in zip(a, got):
        fill(t)
        em._core._sync()
        ref = new()
        for i in range(3):
            bwd(x, w, g, *(r if i == j else None for j, r in enumerate(ref)), m, n, k)
        for r, o in zip(ref, outs):
            assert np.array_equal(r.to_np(), o)


def test_results_over_operands():
    m, k, n = 1024, 512, 768
    x, w, g = (bf16_round(seeded(s, i)) for i, s in enumerate([(m, k), (k, n), (m, n)]))
    T = lambda a: em.Tensor(a, "bfloat16")  # noqa: E731
    dx, dw, db = (em.Tensor.empty(s, "bfloat16") for s in [(m, k), (k, n), (n,)])
    bwd(T(x), T(w), T(g), dx, dw, db, m, n, k)
    over, dw2, db2 = T(x), em.Tensor.empty((k, n), "bfloat16"), em.Tensor.empty((n,), "bfloat16")
    bwd(over, T(w), T(g), over, dw2, db2, m, n, k)  # grad_x in the place of x, which grad_w still reads
    for a, b in ((over, dx), (dw2, dw), (db2, db)):
        assert np.array_equal(a.to_np(), b.to_np())


@pytest.mark.parametrize("over", ["dx x", "dw w", "db x", "db w", "db dy", "db dw", "db dx", "dw dx"])
def test_results_over_operands_and_one_another(over):
    """A result that starts where an operand or another result does, where the products one after the other make that well defined: what
    three calls in the order weight, bias, input gradient leave behind."""
    result, place = over.split()
    sizes = {"x": (1024, 512), "w": (512, 768), "dy": (1024, 768), "dx": (1024, 512), "dw": (512, 768), "db": (768,)}
    (m, k), n = sizes["x"], 768
    values = {name: bf16_round(seeded(sizes[name], i)) for i, name in enumerate(("x", "w", "dy"))}
    got = []
    for together in (True, False):
        T = {name: em.Tensor(values[name], "bfloat16") if name in values else em.Tensor.empty(shape, "bfloat16") for name, shape in sizes.items()}
        T[result] = T[place].view(0, sizes[result])
        for wanted in [("dx", "dw", "db")] if together else [("dw",), ("db",), ("dx",)]:
            bwd(T["x"], T["w"], T["dy"], *(T[r] if r in wanted else None for r in ("dx", "dw", "db")), m, n, k)
        got.append({name: t.to_np() for name, t in T.items()})
    for name in sizes:
        assert np.array_equal(got[0][name], got[1][name]), name


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("m", [300, 8192])
def test_grad_x_in_the_place_of_grad_y(m, bias):
    """One tile of columns: a tile's rows of grad_y are all read before its grad_x is stored, so that the input gradient alone may take their
    place; the weight and bias gradients, which read grad_y too, then have to be done before it."""
    n = k = 128
    x, w, g = (em.Tensor(bf16_round(seeded(s, i)), "bfloat16") for i, s in enumerate([(m, k), (k, n), (m, n)]))
    new = lambda: [em.Tensor.empty(s, "bfloat16") for s in [(m, k), (k, n), (n,)]]  # noqa: E731
    dx, dw, db = new()
    bwd(x, w, g, dx, None, None, m, n, k)
    bwd(x, w, g, None, dw, db, m, n, k)
    want = [t.to_np() for t in (dx, dw, db)][:3 if bias else 2]
    for _ in range(5):
        over, dw2, db2 = em.Tensor(g.to_np(), "bfloat16"), *new()[1:]
        bwd(x, w, over, over, dw2, db2 if bias else None, m, n, k)
        for a, b in zip((over, dw2, db2), want):
            assert np.array_equal(a.to_np(), b)


@pytest.mark.parametrize("m,k,n", [(4104, 1544, 4616), (1000, 512, 1536), (1024, 512, 32768)])
def test_captured_and_on_another_stream(m, k, n):
    """In a graph, whose first and last kernels write what is read and read what is written: each replay sees its own inputs through."""
    import ctypes

    torch = pytest.importorskip("torch")
    L, dev = _lib.lib(), torch.device("cuda", 0)
    x, w, g = (torch.empty(s, device=dev, dtype=torch.bfloat16) for s in ((m, k), (k, n), (m, n)))
    src = torch.empty((m, n), device=dev)
    outs = [torch.empty(s, device=dev, dtype=torch.bfloat16) for s in ((m, k), (k, n), (n,))]
    seen = [torch.empty_like(t) for t in outs]
    s = torch.cuda.Stream(device=dev)

    def calls():
        g.copy_(src)
        _lib.check(L.ember_linear_bwd(*(t.data_ptr() for t in (x, w, g, *outs)), m, n, k, BF16, 0, 0, 0, 0, ctypes.c_void_p(s.cuda_stream)))
        for a, b in zip(seen, outs):
            a.copy_(b)
        g.zero_()

    def fill(seed):
        gen = torch.Generator(device=dev).manual_seed(seed)
        for t in (x, w, src):
            t.normal_(generator=gen)
        torch.cuda.synchronize()

    def want():
        g.copy_(src)
        torch.cuda.synchronize()
        ref = [torch.empty_like(t) for t in outs]
        for i in range(3):
            at = [r.data_ptr() if i == j else None for j, r in enumerate(ref)]
            _lib.check(L.ember_linear_bwd(*(t.data_ptr() for t in (x, w, g)), *at, m, n, k, BF16, 0, 0, 0, 0, None))
        torch.cuda.synchronize()
        _lib.check(L.ember_check_device_status(None, None))
        return ref

    fill(1)
    with torch.cuda.stream(s):
        calls()
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        calls()
    for seed in (2, 3, 4):
        fill(seed)
        ref = want()
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(seen, ref):
            assert torch.equal(a, b)
