"""The native depth hint (one kernel) against the same formula on the CPU."""
import pytest
import torch

from ever_b200 import scheduler as SCH

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 255, 257, 100_003])
def test_depth_from_prediction(n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator().manual_seed(n)
    pred, o, d = (torch.randn((n, k), generator=g) for k in (2, 3, 3))
    want = SCH.depth_from_prediction(pred.double(), o.double(), d.double(), (0.1, -0.2, 0.3), 1.7)
    got = SCH.depth_from_prediction(pred.cuda(), o.cuda(), d.cuda(), (0.1, -0.2, 0.3), 1.7)
    out = torch.empty(n, device="cuda")
    assert SCH.depth_from_prediction(pred.cuda(), o.cuda(), d.cuda(), (0.1, -0.2, 0.3), 1.7, out=out) is out
    assert torch.equal(out, got)
    # about ten float32 roundings of the terms' magnitudes, divided by |d| twice
    m = d.norm(dim=1).double().clamp_min(1e-30)
    size = (pred[:, 1].abs() * 1.7 + (o.abs().sum(1) + 0.6)).double() / m + 1.0
    assert bool(((got.cpu().double() - want).abs() <= 16 * 2.0 ** -24 * size / m).all())
