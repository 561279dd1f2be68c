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
