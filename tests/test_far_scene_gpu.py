"""Scenes in world coordinates: coordinates large against the distances and radii, rays that
start off the camera. The rounding of a ray's start is then a good part of a small radius, and
the frustum phase (traversal 0) still takes exactly the events of the gather rounds
(traversal 2), bit for bit."""
import numpy as np
import pytest
import torch

from ever_b200 import synthetic as S
from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu


def _same(arrays, o, d, tmin, order=None):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    t = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda:0")
    scene = T.Scene(*[t(a) for a in arrays])
    ro, rd = t(o), t(d)
    order = T.ray_order(ro, rd) if order else None
    f = [T.forward(scene, ro, rd, tmin, 1000.0, 300, touch_count=True, ray_order=order, tune=T.Tune(16, 128, m))
         for m in (0, 2)]
    for k in ("iters", "touch_count", "out", "states", "last_dirac", "status"):
        assert torch.equal(getattr(f[0], k), getattr(f[1], k)), k
    assert torch.equal(*[T.reference_tri_collection(scene, x, 300, order) for x in f])
    return f[0]


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def _grazing(packets, coord, dist, radius, over, thin=1.0, half=2e-5, seed=1):
    """One packet of 32 rays (a narrow 8 x 4 tile, each packet with its own apex) and one
    ellipsoid for each: past the tile's corner ray, whose closest approach is 1 to 1 + over
    radii, so that roundings decide. thin: the third radius over the others."""
    r = np.random.default_rng(seed)
    apex = r.uniform(-coord, coord, (packets, 3)).astype(np.float32)
    fwd = _unit(r.standard_normal((packets, 3)))
    a = _unit(np.cross(fwd, r.standard_normal((packets, 3))))
    b = np.cross(fwd, a)
    i = np.arange(32)
    d = _unit(fwd[:, None] + ((i % 8 - 3.5) / 3.5 * half)[:, None] * a[:, None]
              + ((i // 8 - 1.5) / 1.5 * half / 2)[:, None] * b[:, None])
    corner, out = d[:, -1], a + b
    out = _unit(out - (out * corner).sum(1, keepdims=True) * corner)
    # the thin axis along `out`: the ellipsoid is seen edge-on (rotation by the conjugate quaternion)
    axis = np.cross(out, [0.0, 0.0, 1.0])
    quat = _unit(np.concatenate([1 + out[:, 2:], -axis], 1))
    centre = apex + dist * corner + radius * thin * (1 + r.uniform(0, over, (packets, 1))) * out
    scale = np.broadcast_to([radius, radius, radius * thin], centre.shape)
    arrays = (centre, scale, quat, np.full(packets, 1.0), r.standard_normal((packets, 1, 3)))
    return arrays, np.repeat(apex, 32, 0), d.reshape(-1, 3)


# the coordinates, the distance and the radii of scenes in metres seen from close by
@pytest.mark.parametrize("tmin", [0.0, 0.05, 0.2])
@pytest.mark.parametrize("coord,dist,radius,over,thin", [
    (4.0, 3.0, 0.002, 0.02, 1.0), (200.0, 0.5, 0.001, 0.02, 1.0), (1000.0, 1.0, 0.002, 0.02, 1.0),
    (1000.0, 1.0, 0.005, 0.02, 1.0), (5000.0, 20.0, 0.02, 0.1, 1.0), (4.0, 3.0, 0.2, 0.02, 1e-4),
    (1000.0, 1.0, 0.1, 0.1, 1e-2)])
def test_grazed_ellipsoids(coord, dist, radius, over, thin, tmin):
    f = _same(*_grazing(16384, coord, dist, radius, over, thin), tmin)
    assert 0 < int((f.iters > 0).sum()) < f.iters.numel()  # some tiles just hit, others just miss


@pytest.mark.parametrize("order", [False, True])
@pytest.mark.parametrize("tmin", [0.05, 0.2])
@pytest.mark.parametrize("shift,size", [(200.0, 0.5), (1000.0, 1.0), (5000.0, 5.0)])
def test_moved_scene(shift, size, tmin, order):
    # ellipsoids of 0.1 % to 1 % of the distance to the camera
    sc = S.uniform_scene(20_000, 0, seed=21)
    r = np.random.default_rng(4)
    at = shift * np.array([1.0, -0.7, 0.4])
    o, d = S.look_at_rays(S.Camera(S.sphere_point(2.0, 21), 150, 100, 35.0))
    scale = size * 2.0 * np.exp(r.uniform(np.log(1e-3), np.log(1e-2), sc.scale.shape))
    f = _same((at + 0.5 * size * sc.mean, scale, sc.quat, sc.density.reshape(-1) / size, sc.features),
              at + size * o, d, tmin, order)
    assert int(f.iters.sum()) > 10_000
