"""The packed gather rounds (k_trace_fwd_pass: the rays that need more rounds packed into full
warps for a second and third pass) under traversal 2, the one that runs them: the outputs equal
those of the single launch and of the frustum phase (traversal 0), bit for bit."""
import numpy as np
import pytest
import torch

from ever_b200 import camera as CAM
from ever_b200 import synthetic as S
from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu

KEYS = ("out", "states", "last_dirac", "iters", "touch_count", "ray_stats", "status")


def _scene(n, deg, seed):
    # a faint uniform cloud: rays consume about 150 events, so all three passes carry rays
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = S.uniform_scene(n, deg, seed)
    t = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda:0")
    return T.Scene(t(sc.mean), t(sc.scale), t(sc.quat), t(0.02 * sc.density), t(sc.features))


def _equal(fs, tris):
    for f, tri in zip(fs[1:], tris[1:]):
        for k in KEYS:
            assert torch.equal(getattr(fs[0], k), getattr(f, k)), k
        assert torch.equal(tris[0], tri), "event sequences differ"
    return fs[0]


def _all(scene, ro, rd, max_iters=500, tmin=0.0, tmax=1000.0, order=None, kbuf=16, block=128, split=1):
    kw = dict(touch_count=True, ray_stats=True, ray_order=order)
    fs = [T.forward(scene, ro, rd, tmin, tmax, max_iters, regrouped=packed,
                    tune=T.Tune(kbuf, block, traversal, regroup_min=split), **kw)
          for traversal, packed in ((2, True), (2, False), (0, True))]
    return _equal(fs, [T.reference_tri_collection(scene, f, max_iters, order) for f in fs])


def _view(w, h, seed, fov=40.0):
    return S.look_at_rays_device(S.Camera(S.sphere_point(3.0, seed), w, h, fov), torch.device("cuda:0"))


@pytest.mark.parametrize("kbuf,block", [(16, 128), (8, 64), (16, 256), (8, 128), (16, 64)])
@pytest.mark.parametrize("ordered", [False, True])
def test_passes(kbuf, block, ordered):
    scene = _scene(20_000, 2, 51)
    ro, rd = _view(45, 37, 51)  # 1,665 rays: a ragged last warp
    f = _all(scene, ro, rd, order=T.ray_order(ro, rd) if ordered else None, kbuf=kbuf, block=block)
    assert int(f.iters.max()) > 2 * kbuf and int((f.iters < kbuf).sum()) > 0


@pytest.mark.parametrize("max_iters", [1, 16, 17, 33])
def test_truncated(max_iters):
    scene = _scene(10_000, 3, 52)
    ro, rd = _view(33, 29, 52)
    _all(scene, ro, rd, max_iters=max_iters, order=T.ray_order(ro, rd))


@pytest.mark.parametrize("tmin,tmax", [(0.05, 1000.0), (0.0, 0.7), (0.2, 1.1)])
def test_t_range_and_rays_starting_inside(tmin, tmax):
    scene = _scene(3000, 1, 53)
    ro, rd = S.look_at_rays_device(S.Camera(np.array([0.1, -0.2, 0.3]), 31, 19, 70.0), torch.device("cuda:0"))
    _all(scene, ro, rd, tmin=tmin, tmax=tmax)


@pytest.mark.parametrize("split", [0, 1, 300_000])
def test_many_rays(split):
    # 388,800 rays, more than four times the resident lanes: 0 splits by the default rule; 300,000
    # splits after the first round only
    scene = _scene(5000, 0, 55)
    ro, rd = _view(720, 540, 55, 45.0)
    f = _all(scene, ro, rd, order=T.ray_order(ro, rd), split=split)
    assert int((f.iters > 32).sum()) > 10_000


@pytest.mark.parametrize("kbuf,block", [(16, 128), (8, 64)])
def test_camera(kbuf, block):
    scene = _scene(20_000, 2, 61)
    cam = CAM.Camera(70, 45, 60.0, 60.0, np.array([[1.0, 0, 0, 0], [0, 1, 0, 0], [0, 0, 1, -2.5]]))
    fs = [CAM.forward(scene, cam, None, 0.0, 1000.0, 500, touch_count=True, ray_stats=True, regrouped=packed,
                      tune=T.Tune(kbuf, block, traversal, regroup_min=1))
          for traversal, packed in ((2, True), (2, False), (0, True))]
    f = _equal(fs, [CAM.tri_collection(scene, cam, x, 500) for x in fs])
    assert int(f.iters.max()) > 2 * kbuf
