"""Kernels behind a recorded failure: nothing is written, nothing is kept, and the next launch is whole."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
HYPER = (1e-3, 0.9, 0.999, 1e-8, 0.01, 0.1, 0.001, 1.0)      # lr, betas, eps, decay, bias corrections, scale


@pytest.fixture
def ops():
    from shardtrain_b200 import ops as module

    ops = module.load()
    yield ops
    torch.cuda.synchronize()
    ops.status_reset()


def untouched_then_whole(ops, launch, written):
    """`launch()` with a failure on record leaves `written` alone; without one it changes all of them."""
    before = [t.clone() for t in written]
    ops.status_tensor()[:1].fill_(7)
    launch()
    torch.cuda.synchronize()
    assert ops.status_read() == 7
    for got, was in zip(written, before):
        assert torch.equal(got, was)
    ops.status_reset()
    launch()
    torch.cuda.synchronize()
    assert ops.status_read() == 0
    for got, was in zip(written, before):
        assert not torch.equal(got, was)


# whole tiles of 4096, tails of whole and of odd vectors, segments below one tile
@pytest.mark.parametrize("numels", [[8192], [4096, 4100], [1536, 3], [2 * 4096 + 2]])
@pytest.mark.parametrize("members", [1, 2, 3])
@pytest.mark.parametrize("adamw", [True, False])
def test_reduction(ops, numels, members, adamw):
    torch.manual_seed(4)
    segs, shard_off, full_off = [], 0, 0
    for n in numels:
        q = -(-n // members)
        segs.append([shard_off, q, n, full_off, 0])
        shard_off += -(-q // 4) * 4
        full_off += -(-n // 4) * 4
    table = torch.tensor(segs, dtype=torch.int64)
    slots = [torch.randn(full_off, device=DEV) for _ in range(members)]
    slots[0][1] = float("inf")                        # the check has something to say
    held, p, m, v = (torch.rand(shard_off, device=DEV) for _ in range(4))
    shadow = torch.zeros(shard_off, device=DEV, dtype=torch.bfloat16)
    flags = torch.zeros(2, device=DEV, dtype=torch.int32)
    pointers = [t.data_ptr() for t in slots]

    def launch():
        if adamw:
            ops.reduce_scatter_adamw(pointers, 0, table, held, p, m, v, 1.0 / members, False, *HYPER, flags, 1, 0,
                                     1.0, shadow)
        else:
            ops.reduce_scatter(pointers, 0, table, held, 1.0 / members, False, flags)

    untouched_then_whole(ops, launch, [held, flags, *([p, m, v, shadow] if adamw else [])])


# one block, more CTAs than fit at once, and dK/dV cut into parts
@pytest.mark.parametrize("batch,seq,hq,hkv", [(1, 100, 1, 1), (4, 700, 12, 2), (1, 2048, 4, 1)])
def test_attention(ops, batch, seq, hq, hkv):
    torch.manual_seed(seq)
    qkv = torch.randn(batch * seq, (hq + 2 * hkv) * 128, device=DEV).bfloat16()
    out = torch.zeros(batch * seq, hq * 128, device=DEV, dtype=torch.bfloat16)
    lse = torch.zeros(batch, hq, seq, device=DEV)
    scale = 128 ** -0.5
    untouched_then_whole(ops, lambda: ops.attention_fwd(qkv, out, lse, None, batch, seq, hq, hkv, scale), [out, lse])

    q, k, v = (t.view(batch, seq, -1, 128).transpose(1, 2).double().requires_grad_()
               for t in qkv.split([hq * 128, hkv * 128, hkv * 128], dim=1))
    want = torch.nn.functional.scaled_dot_product_attention(
        q, k.repeat_interleave(hq // hkv, 1), v.repeat_interleave(hq // hkv, 1), is_causal=True)
    # probabilities and outputs are rounded to 8 bits: 2^-8 of the largest value covers both
    exact = want.transpose(1, 2).reshape(batch * seq, -1)
    torch.testing.assert_close(out.double(), exact, rtol=0, atol=2.0 ** -7 * exact.abs().max().item())

    grad = torch.randn_like(out)
    dqkv = torch.full_like(qkv, 3.0)
    delta = torch.zeros_like(lse)
    parts = torch.zeros(16 * batch * seq * 2 * hkv * 128, device=DEV)
    # (dK and dV that were cut into parts are added up whatever the status says, from parts nobody wrote: like
    # delta they are scratch, which the GEMMs behind a failure do not read)
    untouched_then_whole(
        ops, lambda: ops.attention_bwd(qkv, out, grad, lse, delta, dqkv, parts, None, batch, seq, hq, hkv, scale),
        [dqkv[:, :hq * 128] if hq > hkv else dqkv])
    exact = torch.autograd.grad(want, (q, k, v), grad.view(batch, seq, hq, 128).transpose(1, 2).double())
    for got, ref in zip(dqkv.split([hq * 128, hkv * 128, hkv * 128], dim=1), exact):
        ref = ref.transpose(1, 2).reshape(batch * seq, -1)
        error = (got.double() - ref).norm() / ref.norm()
        assert error < 2.0 ** -6, error        # 8-bit roundings of P, dS and the result
