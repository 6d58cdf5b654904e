"""Kernels of the portable executor against the torch operators they stand for, and both against 64 bits:
the kernels may not be further off."""
import pytest
import torch

from shardtrain_b200.models.qwen2 import apply_rotary, causal_attention, rotary_tables, swiglu

pytestmark = pytest.mark.gpu
DEV = "cuda"
DTYPES = [torch.float32, torch.float16, torch.bfloat16]


def off(got, want):
    return ((got.double() - want).norm() / want.norm().clamp_min(1e-300)).item()


def no_worse(got, torch_way, exact, dtype):
    """1.25 for the luck of single roundings, and the last bit of what can be stored"""
    last = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    for g, t, e in zip(got, torch_way, exact):
        assert off(g, e) <= 1.25 * off(t, e) + 0.5 * last, (off(g, e), off(t, e))


def operators(q, k, v, cos, sin, mask, d, dtype):
    def heads(t):
        return t.reshape(*t.shape[:2], -1, d).transpose(1, 2)

    q, k = apply_rotary(heads(q), heads(k), cos, sin)
    out = causal_attention(q.to(dtype), k.to(dtype), heads(v).to(dtype), mask)
    return out.transpose(1, 2).reshape(*out.shape[:1], out.shape[2], -1)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("batch,seq,hq,hkv,d", [(1, 1, 1, 1, 64), (2, 127, 4, 2, 64), (3, 129, 6, 1, 32),
                                                (1, 300, 2, 2, 96)])
@pytest.mark.parametrize("mask", ["none", "left", "right", "holes"])
def test_attention(dtype, batch, seq, hq, hkv, d, mask):
    from shardtrain_b200.runtime import portable_kernels

    torch.manual_seed(seq)
    q, k, v = (torch.randn(batch, seq, n * d, device=DEV).to(dtype) for n in (hq, hkv, hkv))
    where = torch.arange(seq, device=DEV)[None].expand(batch, seq)
    m = {"none": None, "left": (where >= seq // 2).long(), "right": (where < (seq + 1) // 2).long(),
         "holes": (where % 3 > 0).float()}[mask]
    positions = where if mask == "left" else where[:1]
    inv = 1e4 ** (-torch.arange(0, d, 2, device=DEV) / d)
    cos, sin = rotary_tables(positions, inv, torch.float32)
    grad = torch.randn(batch, seq, hq * d, device=DEV).to(dtype)

    def both(way, *tensors):
        leaves = [t.clone().requires_grad_() for t in tensors]
        out = way(*leaves)
        out.backward(grad.to(out.dtype))
        return [out.detach(), *(t.grad for t in leaves)]

    def kernels(q, k, v):
        out = portable_kernels.attention(q, k, v, (cos, sin), m, d)
        assert out is not None and type(out.grad_fn).__name__ == "AttentionBackward"
        return out

    got = both(kernels, q, k, v)
    way = both(lambda *t: operators(*t, cos, sin, m, d, dtype), q, k, v)
    # (`causal_attention` forms its scores in fp32 whatever it is given: written out for 64 bits)
    def exact(q, k, v):
        def heads(t):
            return t.reshape(batch, seq, -1, d).transpose(1, 2)

        qr, kr = apply_rotary(heads(q), heads(k), cos.double(), sin.double())
        kr, vr = (t.repeat_interleave(hq // hkv, 1) for t in (kr, heads(v)))
        seen = torch.ones(seq, seq, dtype=torch.bool, device=DEV).tril()[None, None]
        if m is not None:
            seen = seen & m.bool()[:, None, None, :]
        s = (qr @ kr.transpose(-1, -2) / d ** 0.5).masked_fill(~seen, -1e300)
        p = torch.softmax(s, -1).masked_fill(~seen, 0)
        return (p @ vr).transpose(1, 2).reshape(batch, seq, -1)

    ref = both(exact, q.double(), k.double(), v.double())
    assert all(a.dtype == dtype and a.shape == b.shape for a, b in zip(got, way))
    no_worse(got, way, ref, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("where", [(0, 0, 0, 0), (0, 0, 5, 3), (0, 0, 5, 5), (0, 0, 5, 7)])
def test_softmax_of_values_that_are_not_finite(dtype, value, where):
    """Scores and gradients with one such value, at a visible and at an invisible key, and a dead row."""
    from shardtrain_b200 import ops as module

    ops = module.load()
    torch.manual_seed(1)
    seq, d = 9, 64
    mask = torch.ones(1, seq, device=DEV, dtype=torch.bool)
    mask[0, 0] = False
    base, grads = (torch.randn(1, 1, seq, seq, device=DEV).to(dtype) for _ in range(2))
    for spoil in (0, 1):
        scores, grad = base.clone(), grads.clone()
        (scores, grad)[spoil][where] = value
        leaf = scores.clone().requires_grad_()
        seen = torch.ones(seq, seq, dtype=torch.bool, device=DEV).tril() & mask
        s = (leaf.float() / d ** 0.5).masked_fill(~seen, float("-inf"))
        dead = ~seen.any(-1, keepdim=True)
        p = torch.softmax(s.masked_fill(dead, 0.0), -1).masked_fill(dead, 0.0)
        p.to(dtype).backward(grad)
        probs, stats = ops.portable_softmax(scores, mask, d)
        back = ops.portable_softmax_bwd(scores, mask, stats, grad, d)
        torch.testing.assert_close(probs, p.to(dtype), equal_nan=True)
        torch.testing.assert_close(back, leaf.grad, equal_nan=True)


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 127), (130, 512), (700, 1000), (2, 8192)])
def test_norm(rows, cols):
    from shardtrain_b200 import ops as module

    ops = module.load()
    torch.manual_seed(cols)
    x, g = torch.randn(rows, cols, device=DEV), torch.randn(rows, cols, device=DEV)
    w = torch.rand(cols, device=DEV) + 0.5

    def chain(x, w, g):
        inv = torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6)
        scaled = g * w
        dx = inv * (scaled - x * inv.square() * (scaled * x).mean(-1, keepdim=True))
        return x * inv * w, dx, (g * (x * inv)).sum(0)

    out, inv = ops.portable_norm_fwd(x, w, 1e-6)
    dx, dw = ops.portable_norm_bwd(g, x, inv, w)
    no_worse((out, dx, dw), chain(x, w, g), chain(x.double(), w.double(), g.double()), torch.float32)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", [1, 255, 257, 100003])
def test_swiglu_and_sum(dtype, n):
    from shardtrain_b200 import ops as module
    from shardtrain_b200.runtime import portable_kernels

    torch.manual_seed(n)
    gate, up, grad = (4 * torch.randn(n, device=DEV)).to(dtype), *(torch.randn(2, n, device=DEV).to(dtype))

    def both(way):
        a, b = gate.clone().requires_grad_(), up.clone().requires_grad_()
        out = way(a, b)
        out.backward(grad)
        return out.detach(), a.grad, b.grad

    # the same roundings in the same order; only the last bit of fp32 may differ before them
    last = {torch.float32: 2.0 ** -22, torch.float16: 2.0 ** -10, torch.bfloat16: 2.0 ** -7}[dtype]
    for got, want in zip(both(portable_kernels.swiglu), both(swiglu)):
        torch.testing.assert_close(got, want, rtol=2 * last, atol=1e-6)
    ops = module.load()
    assert torch.equal(ops.portable_sum(gate, None, None), gate.float())
    assert torch.equal(ops.portable_sum(gate, up, grad), gate.float() + up.float() + grad.float())


@pytest.mark.parametrize("lengths", [[1], [300, 8, 1000003], [7, 5, 256, 257]])
def test_commit(lengths):
    from shardtrain_b200 import ops as module

    ops = module.load()
    starts = [sum(lengths[:i]) for i in range(len(lengths))]
    offs = [8 + sum(-(-n // 8) * 8 for n in lengths[:i]) for i in range(len(lengths))]
    table = torch.tensor([[s, n, o] for s, n, o in zip(starts, lengths, offs)], device=DEV)
    packed, arena = torch.randn(sum(lengths), device=DEV), torch.randn(offs[-1] + lengths[-1] + 5, device=DEV)
    for accumulate in (False, True):
        want = arena.clone()
        for s, n, o in zip(starts, lengths, offs):
            want[o:o + n] = packed[s:s + n] + (want[o:o + n] if accumulate else 0)
        ops.portable_commit(packed, table, max(lengths), arena, accumulate)
        assert torch.equal(arena, want)
