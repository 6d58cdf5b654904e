"""Attention kernels at the edges of their 128-row blocks, against an fp64 oracle."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, D = "cuda:0", 128


@pytest.fixture(scope="module")
def ops():
    from shardtrain_b200 import ops as ops_module

    return ops_module.load()


def oracle(qkv, dout, B, S, hq, hkv, keep):
    x = qkv.double().view(B, S, hq + 2 * hkv, D).clone().requires_grad_(True)
    q = x[:, :, :hq].transpose(1, 2)
    k = x[:, :, hq:hq + hkv].transpose(1, 2).repeat_interleave(hq // hkv, 1)
    v = x[:, :, hq + hkv:].transpose(1, 2).repeat_interleave(hq // hkv, 1)
    allow = torch.ones(S, S, dtype=torch.bool, device=DEV).tril()[None, None] & keep[:, None, None, :]
    scores = (q @ k.transpose(-1, -2) / math.sqrt(D)).masked_fill(~allow, float("-inf"))
    dead = ~allow.any(-1, keepdim=True)
    probs = torch.softmax(scores.masked_fill(dead, 0), -1).masked_fill(dead, 0)
    out = (probs @ v).transpose(1, 2).reshape(B * S, hq * D)
    out.backward(dout.double())
    return out.detach(), x.grad.view(B * S, -1)


@pytest.mark.parametrize("S", [1, 31, 127, 128, 129, 255, 257, 640])
@pytest.mark.parametrize("mask", ["none", "holes"])
@pytest.mark.parametrize("hq,hkv,split", [(2, 2, False), (6, 2, False), (6, 2, True)])
def test_block_edges(ops, S, mask, hq, hkv, split):
    B = 2
    torch.manual_seed(S)
    W = (hq + 2 * hkv) * D
    qkv, dout = torch.randn(B * S, W, device=DEV).bfloat16(), torch.randn(B * S, hq * D, device=DEV).bfloat16()
    keep = torch.ones(B, S, dtype=torch.bool, device=DEV)
    bits = None
    if mask == "holes":
        keep = torch.rand(B, S, device=DEV) > 0.4
        bits = torch.empty(B, 4 * ((S + 127) // 128), device=DEV, dtype=torch.int32)
        ops.pack_key_mask(keep.to(torch.uint8), bits)
    guard = torch.full((B * S + 1, hq * D), 7.0, device=DEV, dtype=torch.bfloat16)
    out = guard[:-1]
    lse, delta = torch.zeros(B, hq, S, device=DEV), torch.zeros(B, hq, S, device=DEV)
    d_guard = torch.full((B * S + 1, W), 7.0, device=DEV, dtype=torch.bfloat16)
    scratch = torch.empty((hq // hkv) * B * S * 2 * hkv * D if split else 1, device=DEV)
    scale = 1 / math.sqrt(D)
    ops.attention_fwd(qkv, out, lse, bits, B, S, hq, hkv, scale)
    ops.attention_bwd(qkv, out, dout, lse, delta, d_guard[:-1], scratch, bits, B, S, hq, hkv, scale)
    want, d_want = oracle(qkv, dout, B, S, hq, hkv, keep)
    # P and dS are rounded to bf16 (2^-9 each) before products that sum values of size ~1 with
    # weights that add up to 1, and the results once more
    def near(got, ref, size):
        assert torch.all((got.double() - ref).abs() <= 2.0 ** -7 * (size + ref.abs()))

    near(out, want, 1.0)
    near(d_guard[:-1], d_want, max(4.0, d_want.abs().max().item() / 2))
    assert torch.all(guard[-1] == 7.0) and torch.all(d_guard[-1] == 7.0)
    # ... and block by block: late rows are averages over many keys, a tenth of the size of early ones.
    # The same roundings (P and dS, out inside delta, results) done in torch on fp64 values put up to
    # 0.0037 of a block's norm and, on single elements, 0.044 of its rms between the two.
    got = torch.cat([out, d_guard[:-1]], 1).double().view(B, S, -1, D)
    ref = torch.cat([want, d_want], 1).view(B, S, -1, D)
    for first in range(0, S, 128):
        diff, size = (got - ref)[:, first:first + 128], ref[:, first:first + 128]
        norm = lambda t: t.square().sum((1, 3)).sqrt()                      # noqa: E731
        rows = diff.shape[1]
        assert torch.all(norm(diff) <= 0.006 * norm(size) + 1e-5 * (rows * D) ** 0.5)
        rms = (norm(size) / (rows * D) ** 0.5)[:, None, :, None]
        assert torch.all(diff.abs() <= 2.0 ** -7 * size.abs() + 0.1 * rms + 1e-5)
    if mask == "holes":
        dead = (keep.cumsum(1) == 0).reshape(-1)
        assert not out[dead].any() and not d_guard[:-1][dead][:, :hq * D].any()
        assert not d_guard[:-1][~keep.reshape(-1)][:, hq * D:].any()


def test_values_that_are_not_finite_stay_where_they_belong(ops):
    """A NaN value row and an infinite query row: rows that see them are not finite, other heads, other
    samples and earlier blocks keep their bits, forward and backward."""
    B, S, hq, hkv = 2, 256, 2, 2
    torch.manual_seed(1)
    W = (hq + 2 * hkv) * D
    dout = torch.randn(B * S, hq * D, device=DEV).bfloat16()
    clean = torch.randn(B * S, W, device=DEV).bfloat16()
    bad = clean.clone()
    bad.view(B, S, -1, D)[0, 140, hq + hkv] = float("nan")        # value of head 0, sample 0
    bad.view(B, S, -1, D)[1, 200, 1] = float("inf")               # query of head 1, sample 1
    outs, grads = [], []
    for qkv in (clean, bad):
        out, d_qkv = torch.empty(B * S, hq * D, device=DEV, dtype=torch.bfloat16), torch.empty_like(clean)
        lse, delta = torch.empty(B, hq, S, device=DEV), torch.empty(B, hq, S, device=DEV)
        ops.attention_fwd(qkv, out, lse, None, B, S, hq, hkv, 1 / math.sqrt(D))
        ops.attention_bwd(qkv, out, dout, lse, delta, d_qkv, torch.empty(1, device=DEV), None, B, S, hq, hkv,
                          1 / math.sqrt(D))
        outs.append(out.view(B, S, hq, D))
        grads.append(d_qkv.view(B, S, hq + 2 * hkv, D))
    out, ref = outs[1], outs[0]
    assert out[0, 140:, 0].isnan().all() and out[1, 200, 1].isnan().all()
    assert torch.equal(out[0, :128, 0], ref[0, :128, 0]) and torch.equal(out[0, :, 1], ref[0, :, 1])
    assert torch.equal(out[1, :, 0], ref[1, :, 0])
    assert torch.equal(out[1, :200, 1], ref[1, :200, 1]) and torch.equal(out[1, 201:, 1], ref[1, 201:, 1])
    d, ref = grads[1], grads[0]
    assert not d[0, 140:, 0].isfinite().any() and not d[1, 200, 1].isfinite().any()
    assert torch.equal(d[0, :128, 0], ref[0, :128, 0])                      # dQ of the block before
    assert torch.equal(d[1, :200, 1], ref[1, :200, 1]) and torch.equal(d[1, 201:, 1], ref[1, 201:, 1])
    for head, sample in ((1, 0), (0, 1)):
        for plane in (head, hq + head, hq + hkv + head):                    # dQ, dK, dV
            assert torch.equal(d[sample, :, plane], ref[sample, :, plane])
