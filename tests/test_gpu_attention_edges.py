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
    if mask == "holes":
        dead = (keep.cumsum(1) == 0).reshape(-1)
        assert not out[dead].any() and not d_guard[:-1][dead][:, :hq * D].any()
        assert not d_guard[:-1][~keep.reshape(-1)][:, hq * D:].any()
