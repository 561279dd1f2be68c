"""Performance cases of the library, through its Python entry points.

Each case is one piece of work that a program built on ``ember_b200`` repeats: an attention forward or
training step, one token of a decode loop, a self-attention block, a classifier head. ``listed()``
holds fixed cases, ``draw(rng)`` gives others of the same ranges. The families (``op``):

  numpy     NumPy arrays in, attention, NumPy array out: the way a caller without device data uses it
  attend    attention on device tensors; ``mode`` is "forward" (``attention``) or "train"
            (``nn.Attention`` forward and backward)
  decode    one step over a ``KVCache``: append one position, attend over everything stored
  generate  one token through ``nn.MultiHeadAttention.decode_step``: projections, cache and attention
  block     forward and backward of ``nn.MultiHeadAttention``
  head      ``nn.Linear`` and ``loss.CrossEntropyLoss``, forward and backward: a classifier's last layer
"""
import math

import numpy as np
import torch

import ember_b200 as em

F32, BF16 = "float32", "bfloat16"


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call, from host arrays and back: what a first program or a unit test does
        dict(name="numpy_f32_128", op="numpy", dtype=F32, batch=2, heads=4, lq=128, lk=128, dim=64, causal=False),
        # float32 training at an ordinary size: the storage type the library's callers start from
        dict(name="train_f32_1024", op="attend", mode="train", dtype=F32, batch=2, heads=8, lq=1024, lk=1024, dim=64, causal=True),
        # prompt processing of a batch
        dict(name="prefill_4096", op="attend", mode="forward", dtype=BF16, batch=4, heads=32, lq=4096, lk=4096, dim=128, causal=True),
        # cross-attention between sequences of uneven lengths, a head dimension between the native ones
        dict(name="train_ragged_d80", op="attend", mode="train", dtype=BF16, batch=3, heads=12, lq=777, lk=1301, dim=80, causal=False),
        # one GPU's share of a training step that is split over eight
        dict(name="train_2048_16_heads", op="attend", mode="train", dtype=BF16, batch=1, heads=16, lq=2048, lk=2048, dim=128, causal=True),
        # training on long sequences
        dict(name="train_8192", op="attend", mode="train", dtype=BF16, batch=2, heads=32, lq=8192, lk=8192, dim=128, causal=True),
        # decode for a full serving batch, long contexts, grouped query heads
        dict(name="decode_gqa_32768", op="decode", dtype=BF16, batch=64, kv_heads=8, group=4, fill=32767, dim=128),
        # decode for a few users with one key/value head per query head
        dict(name="decode_mha_4001", op="decode", dtype=BF16, batch=4, kv_heads=32, group=1, fill=4000, dim=128),
        # token-by-token generation through a whole block for a small batch
        dict(name="generate_b8_e2048", op="generate", dtype=BF16, batch=8, heads=16, dim=128, fill=1000),
        # training a block
        dict(name="block_2048_e2048", op="block", dtype=BF16, batch=4, length=2048, heads=16, dim=128),
        # a small float32 classifier: ten classes, a few hundred samples
        dict(name="head_f32_10", op="head", dtype=F32, rows=256, features=784, classes=10),
        # the vocabulary projection and loss of a training step
        dict(name="head_bf16_32768", op="head", dtype=BF16, rows=8192, features=2048, classes=32768),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_numpy(rng):
    n = _log(rng, 16, 512)
    return dict(op="numpy", dtype=rng.choice([F32, F32, BF16]), batch=rng.randint(1, 4), heads=rng.randint(1, 8),
                lq=n, lk=n, dim=rng.choice([16, 32, 64, 80, 128]), causal=rng.random() < 0.5)


def _draw_attend(rng):
    dtype = rng.choice([F32, BF16, BF16])
    lk = _log(rng, 64, 2048 if dtype == F32 else 8192)
    lq = lk if rng.random() < 0.6 else _log(rng, 32, lk)
    return dict(op="attend", mode=rng.choice(["forward", "train"]), dtype=dtype, batch=rng.randint(1, 4),
                heads=_log(rng, 1, 32), lq=lq, lk=lk, dim=rng.choice([64, 64, 128, 128, 40, 80, 96]), causal=rng.random() < 0.6)


def _draw_decode(rng):
    return dict(op="decode", dtype=rng.choice([F32, BF16, BF16, BF16]), batch=_log(rng, 1, 64), kv_heads=_log(rng, 1, 32),
                group=rng.choice([1, 2, 4, 8]), fill=_log(rng, 64, 32767), dim=rng.choice([64, 128]))


def _draw_generate(rng):
    return dict(op="generate", dtype=rng.choice([F32, BF16, BF16]), batch=_log(rng, 1, 32), heads=rng.choice([4, 8, 12, 16]),
                dim=rng.choice([64, 128]), fill=_log(rng, 32, 4000))


def _draw_block(rng):
    return dict(op="block", dtype=BF16, batch=rng.randint(1, 4), length=_log(rng, 64, 2048), heads=rng.choice([4, 8, 12, 16]),
                dim=rng.choice([64, 128]))


def _draw_head(rng):
    dtype = rng.choice([F32, BF16])
    return dict(op="head", dtype=dtype, rows=_log(rng, 32, 8192), features=8 * _log(rng, 8, 256),
                classes=_log(rng, 10, 32768) if rng.random() < 0.5 else 8 * _log(rng, 8, 4096))


def draw(rng):
    kind = rng.choice([_draw_numpy, _draw_attend, _draw_attend, _draw_decode, _draw_generate, _draw_block, _draw_head])
    while True:
        c = kind(rng)
        w = work(c)
        # no more than the largest listed cases; what has no matrix instructions (float32, rows that
        # are no multiple of 16 bytes) is used at smaller sizes
        slow = c["dtype"] == F32 or c.get("classes", 0) % 8 != 0
        if w["bytes"] <= 8.6e9 and w["flops"] <= (4e10 if slow else 3.8e12):
            return c


# ---------------------------------------------------------------- device tensors from and to torch
class _Memory:
    """What torch reads to look at a library tensor's memory in place (bfloat16 goes as 16-bit words)."""

    def __init__(self, t):
        self.owner = t
        self.__cuda_array_interface__ = {"shape": t.shape, "typestr": "<f4" if t.dtype == F32 else "<i2",
                                         "data": (t.ptr, False), "version": 2}


def _torch(t):
    x = torch.as_tensor(_Memory(t), device="cuda")
    return x if t.dtype == F32 else x.view(torch.bfloat16)


def _normal(gen, shape, dtype, std=1.0):
    t = em.Tensor.empty(shape, dtype)
    flat = _torch(t).view(-1)
    for at in range(0, flat.numel(), 1 << 28):
        part = flat[at:at + (1 << 28)]
        part.copy_(torch.randn(part.numel(), generator=gen, device="cuda", dtype=part.dtype).mul_(std))
    torch.cuda.synchronize()  # the library works on a stream of its own
    return t


def _one_hot(gen, rows, classes, dtype):
    t = em.Tensor.empty((rows, classes), dtype)
    y = torch.randint(classes, (rows, 1), generator=gen, device="cuda")
    _torch(t).zero_().scatter_(1, y, 1.0)
    torch.cuda.synchronize()
    return t


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    c, op = case, case["op"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if op == "numpy":
        rng = np.random.default_rng(seed)
        lens = (c["lq"], c["lk"], c["lk"])
        return dict(c, qkv=[rng.standard_normal((c["batch"], c["heads"], n, c["dim"]), dtype=np.float32) for n in lens])
    if op == "attend":
        shape = lambda n: (c["batch"], c["heads"], n, c["dim"])  # noqa: E731
        q, k, v = (_normal(gen, shape(n), c["dtype"], 0.5) for n in (c["lq"], c["lk"], c["lk"]))
        g = _normal(gen, shape(c["lq"]), c["dtype"]) if c["mode"] == "train" else None
        return dict(c, qkv=(q, k, v), g=g, layer=em.nn.Attention(causal=c["causal"]))
    if op == "decode":
        B, H, D = c["batch"], c["kv_heads"], c["dim"]
        cache = em.KVCache(B, H, c["fill"] + 1, D, c["dtype"])
        cache.append(*(_normal(gen, (B, H, c["fill"], D), c["dtype"], 0.5) for _ in range(2)))
        new = [_normal(gen, (B, H, 1, D), c["dtype"], 0.5) for _ in range(2)]
        return dict(c, cache=cache, kv=[_torch(cache.k), _torch(cache.v)], new=new, q=_normal(gen, (B, H * c["group"], D), c["dtype"], 0.5))
    if op == "generate":
        B, H, D = c["batch"], c["heads"], c["dim"]
        layer = em.nn.MultiHeadAttention(H * D, H, causal=True, dtype=c["dtype"], seed=seed)
        cache = em.KVCache(B, H, c["fill"] + 1, D, c["dtype"])
        cache.append(*(_normal(gen, (B, H, c["fill"], D), c["dtype"], 0.5) for _ in range(2)))
        return dict(c, layer=layer, cache=cache, kv=[_torch(cache.k), _torch(cache.v)], x=_normal(gen, (B, 1, H * D), c["dtype"]))
    if op == "block":
        E = c["heads"] * c["dim"]
        layer = em.nn.MultiHeadAttention(E, c["heads"], causal=True, dtype=c["dtype"], seed=seed)
        x, g = (_normal(gen, (c["batch"], c["length"], E), c["dtype"]) for _ in range(2))
        return dict(c, layer=layer, x=x, g=g)
    if op == "head":
        layer = em.nn.Linear(c["features"], c["classes"], dtype=c["dtype"], seed=seed)
        x = _normal(gen, (c["rows"], c["features"]), c["dtype"])
        return dict(c, layer=layer, loss=em.loss.CrossEntropyLoss(), x=x, target=_one_hot(gen, c["rows"], c["classes"], c["dtype"]))
    raise ValueError(f"unknown op {op!r}")


def run(state):
    s, op = state, state["op"]
    if op == "numpy":
        q, k, v = (em.Tensor(x, s["dtype"]) for x in s["qkv"])
        return em.attention(q, k, v, causal=s["causal"]).to_np()
    if op == "attend":
        if s["mode"] == "forward":
            return _torch(em.attention(*s["qkv"], causal=s["causal"]))
        y = s["layer"](s["qkv"])
        return [_torch(t) for t in (y, *s["layer"].backward(s["g"]))]
    if op == "decode":
        s["cache"].length = s["fill"]  # the step after the same prompt again
        s["cache"].append(*s["new"])
        return [_torch(t) for t in s["cache"].decode(s["q"])] + s["kv"]
    if op == "generate":
        s["cache"].length = s["fill"]
        return [_torch(s["layer"].decode_step(s["x"], s["cache"]))] + s["kv"]
    if op == "block":
        layer = s["layer"]
        y = layer(s["x"])
        dx = layer.backward(s["g"])
        return [_torch(t) for t in (y, dx, *layer.gradients())]
    layer, loss = s["layer"], s["loss"]
    logits = layer(s["x"])
    value = loss(logits, s["target"])
    dx = layer.backward(loss.backward())
    return [value] + [_torch(t) for t in (logits, loss.probs, dx, *layer.gradients())]


# ---------------------------------------------------------------- work and tolerance
def _attend_flops(units, lq, lk, dim, causal):
    """Forward: two products over the visible (query, key) pairs; bottom-right causal mask."""
    pairs = lq * lk - (lq * (lq - 1) // 2 if causal else 0)
    return 4.0 * units * pairs * dim


def work(case):
    c, op = case, case["op"]
    e = 4 if c["dtype"] == F32 else 2
    if op in ("numpy", "attend"):
        units = c["batch"] * c["heads"]
        q, k = units * c["lq"] * c["dim"], units * c["lk"] * c["dim"]
        f = _attend_flops(units, c["lq"], c["lk"], c["dim"], c["causal"])
        if op == "attend" and c["mode"] == "train":  # reads q, k, v, g; writes y, dq, dk, dv
            return {"bytes": 4.0 * e * (q + k), "flops": 3.5 * f}
        return {"bytes": 2.0 * (4 if op == "numpy" else e) * (q + k), "flops": f}
    if op == "decode":
        units, heads, n = c["batch"] * c["kv_heads"], c["batch"] * c["kv_heads"] * c["group"], c["fill"] + 1
        moved = 2 * units * n * c["dim"] * e + 2 * units * c["dim"] * e + heads * (2 * c["dim"] * e + 4)
        return {"bytes": float(moved), "flops": 4.0 * heads * n * c["dim"]}
    if op == "generate":
        B, E, n = c["batch"], c["heads"] * c["dim"], c["fill"] + 1
        moved = (4 * E * E + 4 * E + 2 * B * n * E + 2 * B * E + 2 * B * E) * e
        return {"bytes": float(moved), "flops": 8.0 * B * E * E + 4.0 * B * n * E}
    if op == "block":
        B, L, E = c["batch"], c["length"], c["heads"] * c["dim"]
        m = B * L  # x, g in and y, dx out; weights and biases in, their gradients out
        f = 3 * 8.0 * m * E * E + 3.5 * _attend_flops(B * c["heads"], L, L, c["dim"], True)
        return {"bytes": float((4 * m * E + 2 * (4 * E * E + 4 * E)) * e), "flops": f}
    m, k, n = c["rows"], c["features"], c["classes"]
    # x, target, w, b in; logits, probabilities, dx, dw, db out
    return {"bytes": float((2 * m * k + 3 * m * n + 2 * k * n + 2 * n) * e), "flops": 6.0 * m * k * n + 8.0 * m * n}


def tolerance(case):
    # float32: sums of up to a few thousand terms in another order; bfloat16: 8-bit significands in
    # the operands of each product (the probabilities and score gradients too) and in the results
    if case["dtype"] == F32:
        return {"rel": 1e-5, "max": 2e-4}
    return {"rel": 1e-2, "max": 1e-1}
