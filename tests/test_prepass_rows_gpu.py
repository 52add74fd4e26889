"""Staged feature rows of the colour pre-pass: block edges, every row width, bases that are not
16-byte aligned. Tolerances as in test_prepass_gpu.py."""
import numpy as np
import pytest
import torch

from ever_b200 import eval_sh as E
from oracle import prepass_np as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 129, 1000])
@pytest.mark.parametrize("deg,K", [(0, 1), (0, 5), (1, 4), (1, 7), (2, 9), (2, 16), (3, 16)])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows(n, deg, K, shift):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n + K)
    means = rng.uniform(-2, 2, (n, 3)).astype(np.float32)
    feats = (rng.normal(size=(n, K, 3)) * 0.4).astype(np.float32)
    cam = np.array([0.5, -4.0, 1.5], np.float32)
    g = rng.normal(size=(n, 3)).astype(np.float32)
    g[::5] = 0.0
    buf = torch.zeros(n * K * 3 + 4, device="cuda")
    ft = buf[shift:shift + n * K * 3].view(n, K, 3)  # shift 1: a base 4 bytes off
    ft.copy_(torch.tensor(feats))
    ft.requires_grad_(True)
    t = lambda a: torch.tensor(a, device="cuda")
    f64 = torch.tensor(feats, dtype=torch.float64, requires_grad=True)
    m64, c64 = torch.tensor(means, dtype=torch.float64), torch.tensor(cam, dtype=torch.float64)
    for mine, oracle in ((E.eval_sh, P.eval_sh), (E.sh_features, P.sh_features)):
        out, want = mine(t(means), ft, t(cam), deg).reshape(n, 3), oracle(m64, f64, c64, deg).reshape(n, 3)
        np.testing.assert_allclose(out.detach().cpu().numpy(), want.detach().numpy(), rtol=1e-5, atol=1e-5)
        got = torch.autograd.grad(out, ft, t(g))[0].cpu().numpy()
        ref = torch.autograd.grad(want, f64, torch.tensor(g, dtype=torch.float64))[0].numpy()
        assert got.shape == ref.shape and np.abs(got - ref).max() <= 1e-5 * max(np.abs(ref).max(), 1e-30)
        assert not got[::5].any() and not got[:, (deg + 1) ** 2:].any()
