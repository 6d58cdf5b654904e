"""fp32 -> bf16 around the edges of its 4096-element tiles: the same bits as torch's rounding, nothing beyond."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 1025, 4095, 4096, 4097, 3 * 4096 + 7, 1554 * 1536, 2368 * 4096 + 2])
def test_cast(n):
    from shardtrain_b200 import ops as module

    torch.manual_seed(n)
    x = torch.randn(n, device="cuda") * 10 ** torch.randint(-20, 20, (n,), device="cuda").float()
    x[torch.randint(0, n, (3,), device="cuda")] = torch.tensor([float("inf"), float("-inf"), -0.0], device="cuda")
    out = torch.full((n + 8,), 7.0, device="cuda", dtype=torch.bfloat16)
    module.load().cast_bf16(x, out[:n])
    assert torch.equal(out[:n].view(torch.int16), x.bfloat16().view(torch.int16))
    assert (out[n:] == 7).all()
