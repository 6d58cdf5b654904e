"""Gradient reduction + AdamW around the edges of its 4096-element tiles: one tile, the last element of a
tile, the first of the next, several segments of different lengths, lengths that are not whole 16 bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
HYPER = (1e-3, 0.9, 0.999, 1e-8, 0.01, 0.1, 0.001, 1.0)      # lr, betas, eps, decay, bias corrections, scale


def oracle(p, g, m, v):
    """AdamW in 64 bits with the kernel's 32-bit hyperparameters."""
    lr, b1, b2, eps, wd, bc1, bc2 = (float(torch.tensor(x)) for x in HYPER[:7])
    p, g, m, v = (t.double() for t in (p, g, m, v))
    m = b1 * m + (1 - b1) * g
    v = b2 * v + (1 - b2) * g * g
    return p * (1 - lr * wd) - lr / bc1 * m / ((v / bc2).sqrt() + eps), m, v


@pytest.mark.parametrize("members", [1, 2])
@pytest.mark.parametrize("numels", [[1], [4095], [4096], [4097], [8192, 4, 4100, 1], [3, 2 * 4096 + 2, 12288]])
@pytest.mark.parametrize("accumulate", [False, True])
def test_tiles(numels, members, accumulate):
    from shardtrain_b200 import ops as module

    ops = module.load()
    torch.manual_seed(3)
    segs, shard_off, full_off = [], 0, 0
    for n in numels:
        q = -(-n // members)
        segs.append([shard_off, q, n, full_off, 0])
        shard_off += -(-q // 4) * 4
        full_off += -(-n // 4) * 4
    table = torch.tensor(segs, dtype=torch.int64)
    slots = [torch.randn(full_off, device=DEV) for _ in range(members)]
    for rank in range(members):
        held, p, m = (torch.randn(shard_off, device=DEV) for _ in range(3))
        v = torch.rand(shard_off, device=DEV)
        for at, q, n, _, _ in segs:                          # a shard's padding holds zeros
            held[at + max(0, min(q, n - rank * q)):at + q] = 0
        was = [t.clone() for t in (held, p, m, v)]
        shadow = torch.zeros(shard_off, device=DEV, dtype=torch.bfloat16)
        flags = torch.zeros(2, device=DEV, dtype=torch.int32)
        only = held.clone()
        ptrs = [t.data_ptr() for t in slots]
        ops.reduce_scatter_adamw(ptrs, rank, table, held, p, m, v, 1.0 / members, accumulate, *HYPER, flags,
                                 1, 0, 1.0, shadow)
        ops.reduce_scatter(ptrs, rank, table, only, 1.0 / members, accumulate, flags)
        assert flags.tolist() == [0, 0]
        covered = torch.zeros(shard_off, dtype=torch.bool, device=DEV)
        for at, q, n, full, _ in segs:
            keep = max(0, min(q, n - rank * q))
            covered[at:at + q] = True
            mine = slice(at, at + keep)
            want = sum(s[full + rank * q:full + rank * q + keep].double() for s in slots) / members
            if accumulate:
                want = want + was[0][mine]
            # one rounding per addition: at most three of 2^-24 of what is added
            size = sum(s.abs().max().item() for s in slots) + was[0].abs().max().item()
            torch.testing.assert_close(held[mine].double(), want, rtol=0, atol=3 * 2.0 ** -24 * size)
            for got, ref in zip((p, m, v), oracle(was[1][mine], held[mine], was[2][mine], was[3][mine])):
                # approximate reciprocal and square root (2^-22 each), a handful of roundings
                torch.testing.assert_close(got[mine].double(), ref, rtol=2e-6, atol=2e-6)
            assert torch.equal(shadow[at:at + q], p[at:at + q].bfloat16())
        for got, before in zip((held, p, m, v), was):       # between the segments nothing is written
            assert torch.equal(got[~covered], before[~covered])
        assert torch.equal(only, held)


@pytest.mark.parametrize("at", [0, 4095, 4096, 9000])
def test_not_finite_and_status(at):
    from shardtrain_b200 import ops as module

    ops = module.load()
    n = 9001
    table = torch.tensor([[0, n, n, 0, 0]], dtype=torch.int64)
    grad = torch.randn(n + 3, device=DEV)
    flags = torch.zeros(2, device=DEV, dtype=torch.int32)
    ops.reduce_scatter([grad.data_ptr()], 0, table, grad, 1.0, False, flags)
    assert flags.tolist() == [0, 0]
    grad[at] = float("nan")
    ops.reduce_scatter([grad.data_ptr()], 0, table, grad, 1.0, False, flags)
    assert flags.tolist() == [1, 0]
