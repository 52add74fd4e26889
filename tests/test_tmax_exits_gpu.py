"""Rays that tmax ends inside many ellipsoids: each of their exits beyond tmax counts if the
reference's round of 16 events that took the entry takes the exit too, however many of our own
rounds, passes and stages that round spans. Event sequences against the oracle."""
import numpy as np
import pytest
import torch

from ever_b200 import synthetic as S
from ever_b200 import tracer as T
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ITERS = 200


def _scene():
    sc = S.uniform_scene(3000, 0, seed=12)
    sc.density *= 0.02
    sc.scale[:150] *= 4
    return sc


@pytest.fixture(scope="module")
def cases():
    sc = _scene()
    out = {}
    for tmax in (2.6, 3.1, 3.5):
        o, d = S.look_at_rays(S.Camera(S.sphere_point(3.0, 5), 61, 37, 45.0))
        out[tmax] = sc, o, d, O.trace(O.Scene(sc.mean, sc.scale, sc.quat, sc.density.reshape(-1), sc.features), o, d, 0.0,
                                      tmax, ITERS)
    return out


@pytest.mark.parametrize("tmax", [2.6, 3.1, 3.5])
@pytest.mark.parametrize("traversal,packed", [(0, True), (1, False), (2, False), (2, True)])
@pytest.mark.parametrize("kbuf", [8, 16, 32])
def test_events_equal_the_oracle(cases, kbuf, traversal, packed, tmax):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc, o, d, ref = cases[tmax]
    t = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda:0")
    scene = T.Scene(t(sc.mean), t(sc.scale), t(sc.quat), t(sc.density.reshape(-1)), t(sc.features))
    f = T.forward(scene, t(o), t(d), 0.0, tmax, ITERS, tune=T.Tune(kbuf, 128, traversal, 1), regrouped=packed)
    tri = T.reference_tri_collection(scene, f, ITERS).cpu().numpy().reshape(ITERS, -1)
    it = f.iters.cpu().numpy()
    assert np.array_equal(it, ref.iters)
    mask = np.arange(ITERS)[:, None] < it[None, :]
    assert np.array_equal(np.where(mask, tri, -1), np.where(mask, ref.events, -1))
