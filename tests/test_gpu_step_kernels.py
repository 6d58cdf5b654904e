"""The bookkeeping kernels of a step against the operators they stand for: the same bits."""
import pytest
import torch
from torch.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from shardtrain_b200 import ops as module

    return module.load()


@pytest.mark.parametrize("batch,seq", [(1, 1), (1, 2), (3, 255), (2, 257), (7, 1000), (160, 8192)])
@pytest.mark.parametrize("layout", ["rows", "slice", "transposed", "all ignored"])
def test_targets_and_their_count(ops, batch, seq, layout):
    torch.manual_seed(batch + seq)
    labels = torch.randint(-2, 5, (batch + 2, seq + 3), device=DEV)
    labels[labels < 0] = -100
    labels = {"rows": labels[:batch, :seq].contiguous(), "slice": labels[1:1 + batch, 2:2 + seq],
              "transposed": labels[:batch, :seq].t().contiguous().t(),
              "all ignored": torch.full((batch, seq), -100, device=DEV)}[layout]
    want = F.pad(labels[:, 1:], (0, 1), value=-100)
    assert torch.equal(ops.shift_targets(labels), want)
    assert torch.equal(ops.count_targets(labels), want.ne(-100).sum())


def test_labels_it_cannot_read_are_refused(ops):
    for bad in (torch.zeros(2, 3, dtype=torch.int64), torch.zeros(2, 3, device=DEV, dtype=torch.int32),
                torch.zeros(6, device=DEV, dtype=torch.int64)):
        with pytest.raises(RuntimeError):
            ops.shift_targets(bad)
        with pytest.raises(RuntimeError):
            ops.count_targets(bad)


@pytest.mark.parametrize("total", [0.0, 1.0, 93210.7, 3e38, float("inf"), float("nan")])
@pytest.mark.parametrize("labels", [1, 3, 8176, 2 ** 24 + 1])
@pytest.mark.parametrize("degree", [1, 3])
def test_loss_and_metrics(ops, total, labels, degree):
    t, n = torch.full((1,), total, device=DEV), torch.tensor(labels, device=DEV)
    loss, factor = ops.loss_of(t, n, float(degree))
    torch.testing.assert_close(loss, t[0] * degree / n, rtol=0, atol=0, equal_nan=True)
    torch.testing.assert_close(factor[0], degree / n, rtol=0, atol=0)
    status = torch.tensor([5, 1, 2, 3], device=DEV, dtype=torch.int32)
    for seen in ([0, 0], [1, 0], [0, 1]):
        flags = torch.tensor(seen, device=DEV, dtype=torch.int32)
        got = ops.step_metrics(flags, t, n, n + 7, status)
        reported = t[0] / n
        finite = float(seen[0] == 0 and bool(torch.isfinite(reported)))
        want = torch.tensor([finite, reported.item(), labels + 7, seen[1], 5], dtype=torch.float64, device=DEV)
        torch.testing.assert_close(got, want, rtol=0, atol=0, equal_nan=True)
        assert flags.tolist() == [0, 0]
