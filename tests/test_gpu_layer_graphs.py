"""A decoder layer whose launches are chained and branch inside a captured graph, against the same layer launched
kernel by kernel, at the shapes real steps are made of: GEMMs in pairs of CTAs, split K, several waves of dK/dV
next to dQ, key masks.  Every sum has a fixed order, so all bits are the same."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def layer(hq, hkv, inter):
    """Weights (bf16, norms and bias fp32) in the order of the executor's arguments."""
    hidden, width = hq * 128, (hq + 2 * hkv) * 128

    def w(*shape):
        return (torch.randn(*shape, device=DEV) * shape[-1] ** -0.5).bfloat16()

    return dict(w_qkv=w(width, hidden), b_qkv=torch.randn(width, device=DEV), w_o=w(hidden, hidden),
                w_gu=w(2 * inter, hidden), w_down=w(hidden, inter), ln1=torch.rand(hidden, device=DEV) + 0.5,
                ln2=torch.rand(hidden, device=DEV) + 0.5)


# rows of one wave and of many, ragged rows, K of 512 to 18944, one to four parts of dK/dV
@pytest.mark.parametrize("batch,seq,hq,hkv,inter", [(1, 512, 12, 2, 8960), (8, 512, 12, 2, 8960),
                                                    (2, 777, 12, 2, 8960), (1, 1024, 28, 4, 18944),
                                                    (3, 130, 4, 4, 512)])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("accumulate", [False, True])
def test_captured_layers_have_the_bits_of_single_launches(batch, seq, hq, hkv, inter, masked, accumulate):
    from shardtrain_b200 import ops as module

    ops = module.load()
    torch.manual_seed(seq + hq)
    rows, hidden, width = batch * seq, hq * 128, (hq + 2 * hkv) * 128
    w = layer(hq, hkv, inter)
    x, grad = torch.randn(rows, hidden, device=DEV), torch.randn(rows, hidden, device=DEV)
    angle = torch.rand(seq, 64, device=DEV) * 6
    cos, sin = angle.cos(), angle.sin()
    mask = None
    if masked:
        keep = torch.randint(1, seq + 1, (batch, 1), device=DEV)
        as_bytes = (torch.arange(seq, device=DEV)[None] < keep).to(torch.uint8).contiguous()
        mask = torch.empty(batch, 4 * ((seq + 127) // 128), device=DEV, dtype=torch.int32)
        ops.pack_key_mask(as_bytes, mask)
    status = ops.status_tensor()
    shapes = [(hidden, inter), (2 * inter, hidden), (hidden,), (hidden, hidden), (width,), (width, hidden), (hidden,)]
    start = [torch.randn(*s, device=DEV) for s in shapes]     # earlier micro-steps' sums
    slots = [torch.empty_like(g) for g in start]

    def run(replay):
        saved = ops.layer_forward(x, *w.values(), cos, sin, None, mask, status, batch, seq, hq, hkv, 1e-6, [], False,
                                  None, None, None, replay)
        h1, inv1, qkv, attn, lse, x_mid, h2, inv2, gu, out, hm = saved
        for slot, value in zip(slots, start):
            slot.copy_(value)
        dx = ops.layer_backward(grad, x, inv1, h1, qkv, attn, lse, x_mid, inv2, h2, gu, hm, w["w_qkv"], w["w_o"],
                                w["w_gu"], w["w_down"], w["ln1"], w["ln2"], *slots, cos, sin, None, mask, status,
                                batch, seq, hq, hkv, replay, accumulate)
        return [t.clone() for t in (*saved, dx, *slots)]

    ops.replay_clear()
    with torch.cuda.stream(torch.cuda.Stream()):
        want = run(False)
        for turn in range(4):                                 # launched, captured, replayed twice
            for k, (got, ref) in enumerate(zip(run(True), want)):
                assert torch.equal(got, ref), (turn, k, (got.float() - ref.float()).abs().max().item())
    torch.cuda.synchronize()
    assert ops.replay_graphs() == 2 and ops.status_read() == 0
    ops.replay_clear()
