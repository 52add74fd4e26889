"""Leaf lists of the frustum phase that are cut among nearly equal entry bounds: discs faced by a
narrow packet, a few ulps of t apart, so that what is listed and what is left for the next
stage lie within the margins of the bounds. No event is lost or out of order: the result
equals the gather rounds' (traversal 2) bit for bit, and the event counts the oracle's."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu


def _discs(dist, thick, n, ulps, seed):
    r = np.random.default_rng(seed)
    z = np.round(r.uniform(0, ulps, n)) * float(np.spacing(np.float32(dist)))
    mean = np.stack([r.uniform(-0.2, 0.2, n), r.uniform(-0.2, 0.2, n), -z], 1)
    scale = np.stack([np.ones(n), np.ones(n), np.full(n, thick * dist)], 1)
    arrays = (mean, scale, np.tile([1.0, 0, 0, 0], (n, 1)), np.full(n, 0.01 / (thick * dist) / n),
              r.standard_normal((n, 1, 3)))
    i = np.arange(256)
    d = np.stack([(i // 16) * 1e-6, (i % 16) * 1e-6, -np.ones(256)], 1)
    o = np.broadcast_to([0.0, 0.0, dist], d.shape)
    return [[np.ascontiguousarray(v, dtype=np.float32) for v in x] for x in (arrays, (o, d))]


# n: just over the first stage's 128 leaves, well over, over a later stage's 256, far over both.
# thick: the boxes' padding (0.2 % of the half thickness) is more than an ulp of t, below which
# the rounds' own slab test misses events tied with the last of a round.
@pytest.mark.parametrize("n", [140, 150, 200, 300, 420])
@pytest.mark.parametrize("thick", [1e-3, 1e-4])
@pytest.mark.parametrize("dist", [10.0, 30.0, 100.0, 300.0])
def test_cut_among_equal_bounds(dist, thick, n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    t = lambda a: torch.tensor(a, device="cuda:0")
    for ulps in (20, 50, 70, 100, 150):
        for seed in range(6):
            arrays, (o, d) = _discs(dist, thick, n, ulps, seed)
            scene = T.Scene(*[t(a) for a in arrays])
            f = [T.forward(scene, t(o), t(d), 0.0, 1000.0, 300, touch_count=True, tune=T.Tune(16, 128, m))
                 for m in (0, 2)]
            for k in ("iters", "out", "states", "last_dirac", "touch_count"):
                assert torch.equal(getattr(f[0], k), getattr(f[1], k)), (k, ulps, seed)
            assert torch.equal(*[T.reference_tri_collection(scene, x, 300) for x in f]), (ulps, seed)


def test_event_counts_equal_the_oracle():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    arrays, (o, d) = _discs(300.0, 1e-4, 150, 70, 1)
    t = lambda a: torch.tensor(a, device="cuda:0")
    f = T.forward(T.Scene(*[t(a) for a in arrays]), t(o), t(d), 0.0, 1000.0, 300)
    ref = O.trace(O.Scene(*arrays), o, d, 0.0, 1000.0, 300)
    assert np.array_equal(f.iters.cpu().numpy(), ref.iters)
