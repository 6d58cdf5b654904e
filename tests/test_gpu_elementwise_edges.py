"""Elementwise kernels of a layer's backward at the edges of their vector widths and register tiles."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from shardtrain_b200 import ops as ops_module

    return ops_module.load()


# 1024 columns per register tile, up to four; wider rows take the general kernel
@pytest.mark.parametrize("cols", [4, 1020, 1024, 1028, 2048, 3072, 3584, 4096, 4100, 5120])
@pytest.mark.parametrize("rows", [1, 593, 1300])       # 592 CTAs: none, one and several rows each
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_backward(ops, rows, cols, residual):
    torch.manual_seed(cols)
    dy, x = torch.randn(rows, cols, device=DEV), torch.randn(rows, cols, device=DEV)
    w, res = torch.randn(cols, device=DEV), torch.randn(rows, cols, device=DEV) if residual else None
    inv = torch.rsqrt(x.square().mean(-1) + 1e-6)
    guard = torch.full((rows + 1, cols), 7.0, device=DEV)
    copy = torch.full((rows + 1, cols), 7.0, device=DEV, dtype=torch.bfloat16)
    partial, dw = torch.empty(592, cols, device=DEV), torch.empty(cols, device=DEV)
    ops.rmsnorm_bwd(dy, x, w, inv, res, guard[:rows], partial, copy[:rows])
    ops.colsum_f32(partial, dw, False)
    g, xd, iv = dy.double() * w.double(), x.double(), inv.double()[:, None]
    want = iv * (g - xd * iv * iv * (g * xd).mean(-1, keepdim=True)) + (res.double() if residual else 0)
    # fp32 sums of `cols` terms (2^-24 sqrt(cols) each side of their size), a handful of products
    scale = iv * (g.abs() + xd.abs() * iv * iv * (g * xd).abs().mean(-1, keepdim=True)) + 1
    assert torch.all((guard[:rows].double() - want).abs() <= 2.0 ** -21 * scale * max(1, cols ** 0.5 / 8))
    assert torch.equal(copy[:rows], guard[:rows].bfloat16())
    assert torch.all(guard[rows] == 7.0) and torch.all(copy[rows] == 7.0)
    terms = dy.double() * xd * iv
    assert torch.all((dw.double() - terms.sum(0)).abs() <= 2.0 ** -22 * (terms.abs().sum(0) + 1))


@pytest.mark.parametrize("d", [4, 8, 12, 16, 64, 128])      # 16-byte pieces from 16 on
@pytest.mark.parametrize("shift", [0, 2])                   # elements off a 16-byte boundary
@pytest.mark.parametrize("inverse", [False, True])
def test_rope(ops, d, shift, inverse):
    rows, seq, hq, hkv = 37, 13, 3, 1
    torch.manual_seed(d)
    width = (hq + 2 * hkv) * d
    flat = torch.randn(rows * width + shift, device=DEV).bfloat16()
    qkv = flat[shift:].view(rows, width)
    before = qkv.double().view(rows, -1, d)
    cos, sin = torch.randn(rows, d // 2, device=DEV), torch.randn(rows, d // 2, device=DEV)
    pos = torch.randint(0, rows, (rows,), device=DEV, dtype=torch.int32)
    ops.rope(qkv, cos, sin, pos, seq, hq, hkv, d, inverse)
    c, s = cos.double()[pos.long()][:, None], sin.double()[pos.long()][:, None] * (-1 if inverse else 1)
    lo, hi = before[:, :hq + hkv, : d // 2], before[:, :hq + hkv, d // 2:]
    want = torch.cat([lo * c - hi * s, hi * c + lo * s], -1)
    got = qkv.double().view(rows, -1, d)
    assert torch.all((got[:, :hq + hkv] - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5)   # one bf16 rounding
    assert torch.equal(got[:, hq + hkv:], before[:, hq + hkv:])                            # v is left alone


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 100003])
@pytest.mark.parametrize("shift", [0, 1])
def test_sgd(ops, n, shift):
    p, g = torch.randn(n + shift + 1, device=DEV), torch.randn(n + shift + 1, device=DEV)
    before = p.clone()
    ops.sgd(p[shift:shift + n], g[shift:shift + n], 0.3)
    want = before.double()[shift:shift + n] - 0.3 * g.double()[shift:shift + n]
    assert torch.all((p[shift:shift + n].double() - want).abs() <= 2.0 ** -23 * (want.abs() + 1))
    assert torch.equal(p[shift + n:], before[shift + n:]) and torch.equal(p[:shift], before[:shift])


@pytest.mark.parametrize("rows", [1, 7, 64, 65, 1025, 2500])
def test_column_sums(ops, rows):
    cols = 264
    x = torch.randn(rows, cols, device=DEV)
    out, base = torch.empty(cols, device=DEV), torch.randn(cols, device=DEV)
    ops.colsum_f32(x, out, False)
    bound = 2.0 ** -22 * (x.abs().double().sum(0) + 1)
    assert torch.all((out.double() - x.double().sum(0)).abs() <= bound)
    xb, scratch = x.bfloat16(), torch.empty(64, cols, device=DEV)
    total = base.clone()
    ops.colsum_bf16(xb, total, True, scratch)
    assert torch.all((total.double() - base.double() - xb.double().sum(0)).abs() <= bound + 2.0 ** -22 * base.abs())


@pytest.mark.parametrize("cols", [260, 1536, 4096])
@pytest.mark.parametrize("shift", [1, 2, 3])             # floats off a 16-byte boundary
def test_rmsnorm_backward_takes_partial_sums_at_any_address(ops, cols, shift):
    rows, parts = 37, 8
    torch.manual_seed(cols)
    dy, x, w = torch.randn(rows, cols, device=DEV), torch.randn(rows, cols, device=DEV), torch.randn(cols, device=DEV)
    inv = torch.rsqrt(x.square().mean(-1) + 1e-6)
    flat = torch.full((parts * cols + 8,), 7.0, device=DEV)
    partial, aligned = flat[shift:shift + parts * cols].view(parts, cols), torch.empty(parts, cols, device=DEV)
    dx, want = torch.empty_like(x), torch.empty_like(x)
    ops.rmsnorm_bwd(dy, x, w, inv, None, dx, partial)
    ops.rmsnorm_bwd(dy, x, w, inv, None, want, aligned)
    assert torch.equal(dx, want) and torch.equal(partial, aligned)       # both kernels sum in the same order
    assert torch.all(flat[:shift] == 7.0) and torch.all(flat[shift + parts * cols:] == 7.0)


def test_rmsnorm_backward_refuses_a_copy_off_an_8_byte_boundary(ops):
    x, w = torch.randn(4, 64, device=DEV), torch.randn(64, device=DEV)
    copy = torch.empty(4 * 64 + 2, device=DEV, dtype=torch.bfloat16)[2:].view(4, 64)
    with pytest.raises(RuntimeError, match="rmsnorm_bwd"):
        ops.rmsnorm_bwd(x, x, w, torch.ones(4, device=DEV), None, torch.empty_like(x), torch.empty(2, 64, device=DEV),
                        copy)
