"""MultiHeadAttention.decode_step over a KVCache makes its four calls natively: the bits of the calls made one by one, and the cache's rows and length."""
import numpy as np
import pytest

import ember_b200 as em
from conftest import seeded

pytestmark = pytest.mark.gpu


class PlainCache(em.KVCache):
    """A cache of another type takes the calls one by one."""


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("batch,heads,dim,fill", [(1, 1, 8, 1), (3, 4, 64, 129), (17, 2, 128, 600), (130, 2, 40, 3)])
def test_native_step_is_the_four_calls(batch, heads, dim, fill, dtype):
    layer = em.nn.MultiHeadAttention(heads * dim, heads, causal=True, dtype=dtype, seed=1)
    rows = [em.Tensor(seeded((batch, heads, fill, dim), s, 0.5), dtype) for s in (2, 3)]
    got = []
    for kind in (em.KVCache, PlainCache):
        cache = kind(batch, heads, fill + 2, dim, dtype)
        cache.append(*rows)
        steps = [layer.decode_step(em.Tensor(seeded((batch, 1, heads * dim), 4 + t), dtype), cache) for t in range(2)]
        assert cache.length == fill + 2 and all(y.shape == (batch, 1, heads * dim) and y.dtype == dtype for y in steps)
        got.append([t.to_np() for t in (*steps, cache.k, cache.v)])
        with pytest.raises(ValueError):  # full
            layer.decode_step(em.Tensor(seeded((batch, 1, heads * dim), 9), dtype), cache)
        assert cache.length == fill + 2
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    with pytest.raises((TypeError, ValueError)):
        layer.decode_step(em.Tensor(seeded((batch, 1, heads * dim), 9), "float32" if dtype == "bfloat16" else "bfloat16"), em.KVCache(batch, heads, 4, dim, dtype))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_other_weights_than_the_layer_made(dtype):
    """Set by the caller: no biases and an output of another width are taken, weights of the right size and a wrong shape are refused."""
    batch, heads, dim, fill = 3, 4, 64, 5
    e = heads * dim
    rows = [em.Tensor(seeded((batch, heads, fill, dim), s, 0.5), dtype) for s in (2, 3)]
    x = em.Tensor(seeded((batch, 1, e), 4), dtype)
    got = []
    for kind in (em.KVCache, PlainCache):
        layer = em.nn.MultiHeadAttention(e, heads, causal=True, dtype=dtype, seed=1)
        layer.b_qkv = layer.b_o = None
        layer.w_o = em.Tensor(seeded((e, 2 * e), 5, 0.1), dtype)
        cache = kind(batch, heads, fill + 1, dim, dtype)
        cache.append(*rows)
        y = layer.decode_step(x, cache)
        assert y.shape == (batch, 1, 2 * e) and cache.length == fill + 1
        got.append([t.to_np() for t in (y, cache.k, cache.v)])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    for name, shape in (("w_qkv", (3 * e, e)), ("w_o", (2 * e, e // 2))):
        layer, cache = em.nn.MultiHeadAttention(e, heads, causal=True, dtype=dtype, seed=1), em.KVCache(batch, heads, fill + 1, dim, dtype)
        cache.append(*rows)
        setattr(layer, name, em.Tensor(seeded(shape, 6, 0.1), dtype))
        with pytest.raises(ValueError):
            layer.decode_step(x, cache)
