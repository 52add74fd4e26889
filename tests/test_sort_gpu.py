"""The radix sort behind the orders: stable and sorted at the sizes where its path changes (one
block up to 8,192 keys; tiles of 2,048 that sum their histograms themselves up to 16 tiles;
scanned rows beyond), on one 8-bit pass and on four, and few or many distinct keys."""
import numpy as np
import pytest
import torch

from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu
SIZES = [1, 31, 1025, 8191, 8192, 8193, 2048 * 16, 2048 * 16 + 1, 2048 * 300 + 7]


def _hilbert_key(d):
    """The ray order's direction key in the kernel's float32 operations."""
    f = np.float32
    dx, dy, dz = (d[:, i].astype(f) for i in range(3))
    l1 = (np.abs(dx) + np.abs(dy)).astype(f) + np.abs(dz)
    u, v = dx / l1, dy / l1
    neg = dz < 0
    uu = (f(1) - np.abs(v)) * np.where(u >= 0, f(1), f(-1))
    vv = (f(1) - np.abs(u)) * np.where(v >= 0, f(1), f(-1))
    u, v = np.where(neg, uu, u), np.where(neg, vv, v)
    q = [np.minimum((np.maximum(a * f(0.5) + f(0.5), f(0)) * f(4096)).astype(np.uint32), 4095).astype(np.int64)
         for a in (u, v)]
    x, y = q
    key = np.zeros(len(d), np.int64)
    s = 1 << 11
    while s:
        rx, ry = (x & s) > 0, (y & s) > 0
        key += s * s * ((3 * rx.astype(np.int64)) ^ ry.astype(np.int64))
        flip = ~ry & rx
        x, y = np.where(flip, x ^ (s - 1), x), np.where(flip, y ^ (s - 1), y)
        x, y = np.where(~ry, y, x), np.where(~ry, x, y)
        s >>= 1
    return key


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("distinct", [3, 10_000_000])
def test_ray_order_is_the_stable_sort(n, distinct):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n)
    d = rng.standard_normal((min(n, distinct), 3)).astype(np.float32)
    d = d[rng.integers(0, len(d), n)]
    o = np.zeros((n, 3), np.float32)
    order = T.ray_order(torch.tensor(o, device="cuda"), torch.tensor(d, device="cuda")).cpu().numpy()
    assert np.array_equal(order, np.argsort(_hilbert_key(d), kind="stable"))


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("most", [1, 300])
def test_slot_order_is_the_stable_sort(n, most):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    it = torch.randint(0, most, (n,), generator=torch.Generator().manual_seed(n)).to(torch.int32)
    fwd = T.ForwardResult(*[None] * 3, it.cuda(), *[None] * 4)
    order = T.backward_order(fwd, None, 0).cpu()
    want = torch.sort(255 - it.clamp(max=255), stable=True).indices
    assert torch.equal(order.long(), want)
