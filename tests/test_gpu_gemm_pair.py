"""GEMM with pairs of CTAs on 256-row tiles: edges of tiles, every operand order, K splits."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from shardtrain_b200 import ops as ops_module

    return ops_module.load()


CASES = [
    # M, N, K, a_mn, b_mn, out_fp32, bias, residual, tile width, split
    (8, 8, 8, False, False, True, False, False, 256, 1),         # one corner of one tile
    (128, 256, 64, False, False, False, True, False, 256, 1),    # the second CTA's rows are all past M
    (257, 264, 72, False, False, True, True, True, 256, 1),      # one row / one column group over a tile
    (256, 192, 512, False, False, False, False, True, 192, 1),
    (520, 200, 136, False, True, True, False, False, 192, 1),    # MN-major B: 96 columns in two chunks
    (520, 392, 136, True, True, True, False, False, 192, 1),
    (264, 136, 200, True, True, True, False, False, 128, 1),
    (384, 128, 328, False, True, False, False, False, 128, 1),
    (264, 520, 64, True, False, True, False, False, 256, 1),
    (2048, 2560, 192, False, False, True, False, True, 256, 1),  # 80 tiles: several per pair
    (512, 1536, 1096, False, True, True, False, False, 256, 4),  # tail tiles cut along K
    (300, 584, 1104, False, False, False, True, True, 128, 3),
    (640, 520, 1104, True, True, True, False, False, 192, 2),
]


@pytest.mark.parametrize("case", CASES, ids=["x".join(map(str, c[:3])) + f"_{int(c[3])}{int(c[4])}_{c[8]}s{c[9]}"
                                             for c in CASES])
def test_pair_gemm_matches_reference_and_stays_inside_the_output(ops, case):
    M, N, K, a_mn, b_mn, out_fp32, bias, residual, bn, split = case
    torch.manual_seed(2)
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device=DEV).bfloat16()
    dtype = torch.float32 if out_fp32 else torch.bfloat16
    bias_t = torch.randn(N, device=DEV) if bias else None
    res = torch.randn(M, N + 8, device=DEV).to(dtype)[:, :N] if residual else None
    plane = torch.full((M + 3, N + 8), 7.0, device=DEV, dtype=dtype)
    out = plane[:M, :N]
    ops.gemm(a, b, out, a_mn, b_mn, bias_t, res, False, 1.0, bn, split, True, True)
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    want = want + (bias_t if bias else 0) + (res.double() if residual else 0)
    # products of bf16 values are exact in fp32; K roundings of 2^-24 on partial sums of size up to
    # a few sqrt(K), and one output rounding
    bound = 2.0 ** -24 * math.sqrt(K) * K * 0.5 + 1e-6
    if not out_fp32:
        bound = bound + want.abs() * 2.0 ** -8
    assert torch.all((out.double() - want).abs() <= bound)
    assert torch.all(plane[M:] == 7.0) and torch.all(plane[:, N:] == 7.0)
    again = torch.empty_like(plane)
    ops.gemm(a, b, again[:M, :N], a_mn, b_mn, bias_t, res, False, 1.0, bn, split, True, True)
    assert torch.equal(again[:M, :N], out)      # split sums run in index order


@pytest.mark.parametrize("shape", [(512, 1536, 8960, False, False), (1024, 1536, 4096, False, True),
                                   (1536, 1536, 4096, True, True), (777, 1536, 8960, False, False),
                                   (4096, 1536, 512, False, True), (1554, 2048, 1536, False, False),
                                   (16, 264, 72, False, False), (2048, 1536, 4096, True, True),
                                   (4096, 1536, 8960, False, True), (4096, 17920, 1536, False, False)],
                         ids=lambda s: "x".join(map(str, s[:3])) + f"_{int(s[3])}{int(s[4])}")
def test_automatic_choice_has_the_bits_of_single_ctas(ops, shape):
    """Whatever kernel runs, it sums the elements in the K ranges that single CTAs on 128-row tiles of
    the chosen width would cut."""
    M, N, K, a_mn, b_mn = shape
    bn, _, split = ops.gemm_tile(M, N, K)
    torch.manual_seed(4)
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device=DEV).bfloat16()
    got, want = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.gemm(a, b, got, a_mn, b_mn, None, None, False, 1.0, 0)
    ops.gemm(a, b, want, a_mn, b_mn, None, None, False, 1.0, bn, split, True, False)
    assert torch.equal(got, want)


def test_the_rule_takes_every_kind_of_kernel(ops):
    """{single CTAs, pairs} x {whole, cut along K}, at sizes the tests above compare."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are picked for 148 SMs")
    kinds = {(pair, split > 1) for _, pair, split in
             (ops.gemm_tile(*s) for s in [(4096, 1536, 512), (512, 1536, 8960), (2048, 1536, 4096), (4096, 1536, 8960)])}
    assert kinds == {(0, False), (0, True), (1, False), (1, True)}


ACCUMULATE = [
    # M, N, K, tile width, split (0, 0: the rule)
    (8, 8, 8, 256, 1),                # boxes that overhang both edges of the output
    (264, 264, 72, 256, 1),
    (776, 392, 328, 192, 1),
    (264, 1544, 200, 128, 1),
    (512, 1536, 1096, 256, 4),        # tail tiles cut along K
    (296, 584, 1104, 128, 3),
    (1544, 1536, 4100, 0, 0),         # dW of 4100 tokens
]


@pytest.mark.parametrize("case", ACCUMULATE, ids=["x".join(map(str, c[:3])) + f"_{c[3]}s{c[4]}" for c in ACCUMULATE])
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("residual", [False, True])
def test_accumulating_gemm_adds_to_what_the_output_holds(ops, case, pair, residual):
    """dW of a later micro-step: the boxes of the staged store are added in L2, the row stores read and
    write; either is one fp32 addition to the old value, so the bits agree."""
    M, N, K, bn, split = case
    torch.manual_seed(8)
    a, b = torch.randn(K, M, device=DEV).bfloat16(), torch.randn(K, N, device=DEV).bfloat16()
    old = torch.randn(M + 3, N + 8, device=DEV) * 30
    res = torch.randn(M, N + 8, device=DEV)[:, :N] if residual else None
    planes = []
    for staged in (True, False):
        plane = old.clone()
        ops.gemm(a, b, plane[:M, :N], True, True, None, res, True, 1.0, bn, split, staged, pair)
        planes.append(plane)
    assert torch.equal(planes[0], planes[1])
    want = a.double().t() @ b.double() + old[:M, :N].double() + (res.double() if residual else 0)
    # as above, and one rounding of the sum
    bound = 2.0 ** -24 * (math.sqrt(K) * K * 0.5 + 2 * want.abs()) + 1e-6
    assert torch.all((planes[0][:M, :N].double() - want).abs() <= bound)
    assert torch.equal(planes[0][M:], old[M:]) and torch.equal(planes[0][:, N:], old[:, N:])


def test_pairs_with_the_swiglu_epilogue(ops):
    """Gate and up halves of a tile come from the two CTAs' operands; ragged rows and columns."""
    M, inter, K = 2040, 4728, 1032
    assert ops.gemm_tile(M, 2 * inter, K, inter)[1] == 1
    torch.manual_seed(9)
    x = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(2 * inter, K, device=DEV) / math.sqrt(K)).bfloat16()
    planes = [torch.full((M + 1, c), 7.0, device=DEV, dtype=torch.bfloat16) for c in (2 * inter, inter)]
    gu, h = planes[0][:M], planes[1][:M]
    ops.gemm_swiglu(x, w, gu, h)
    gu2, h2 = torch.empty_like(gu), torch.empty_like(h)
    ops.gemm(x, w, gu2, False, False, None, None, False, 1.0, 256, 1)        # single CTAs, then the kernel
    ops.swiglu_fwd(gu2, h2)
    assert torch.equal(gu, gu2) and torch.equal(h, h2)
    want = x.double() @ w.double().t()
    assert torch.all((gu.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -24 * K)
    assert torch.all(planes[0][M] == 7.0) and torch.all(planes[1][M] == 7.0)


@pytest.mark.parametrize("pair", [True, False])
def test_a_failure_on_record_ends_a_running_gemm(ops, pair):
    """Another kernel records a failure while a long GEMM runs.  Its roles give up one after the other, in
    whatever state their pipelines are; the kernel waits for the copies and MMAs it has in flight and
    returns, and the next launch finds barriers, TMEM and tile counters in order."""
    torch.manual_seed(6)
    side, code = torch.cuda.Stream(), torch.full((1,), 7, dtype=torch.int32).pin_memory()
    x, w = torch.randn(512, 4096, device=DEV).bfloat16(), torch.randn(1536, 4096, device=DEV).bfloat16()
    want = torch.empty(512, 1536, device=DEV)
    ops.gemm(x, w, want, False, False, None, None, False, 1.0, 256, 4, True, pair)
    a = torch.randn(2048, 1 << 17, device=DEV).bfloat16()
    out = torch.empty(2048, 2048, device=DEV)
    torch.cuda.synchronize()
    assert ops.status_read() == 0
    for _ in range(3):
        ops.gemm(a, a, out, False, False, None, None, False, 1.0, 128, 1, True, pair)     # about 1 ms each
    with torch.cuda.stream(side):
        ops.status_tensor()[:1].copy_(code, non_blocking=True)
    torch.cuda.synchronize()
    assert ops.status_read() == 7
    ops.status_reset()
    got = torch.empty_like(want)
    ops.gemm(x, w, got, False, False, None, None, False, 1.0, 256, 4, True, pair)
    assert ops.status_read() == 0
    assert torch.equal(got, want)


def test_forced_pairs_run_as_pairs_whatever_the_width(ops):
    """`force_pair` without a width used to run whatever the rule picked."""
    M, N, K = 300, 520, 200
    assert ops.gemm_tile(M, N, K)[1] == 0                       # the rule takes single CTAs here
    bn, pair, split = ops.gemm_tile(M, N, K, 0, True)
    assert pair == 1 and bn in (128, 192, 256) and split == 1
    torch.manual_seed(3)
    a, b = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16()
    outs = []
    for width in (0, bn):
        out = torch.empty(M, N, device=DEV)
        ops.gemm(a, b, out, False, False, None, None, False, 1.0, width, 0, True, True)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    _, pair, split = ops.gemm_tile(512, 1536, 8960, 0, True)    # too few tiles for 74 pairs: cut along K
    assert pair == 1 and split > 1
