"""The packet frustum phase where its rules change: packets of 4 to 32 rays, lists cut into
stages, full event buffers, packets split at a gap, rays in no order, rays off their apex. The
event sequence, the outputs and the states equal the gather rounds' (traversal 2) bit for bit;
on small scenes the events equal the oracle's."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from ever_b200 import synthetic as S
from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu


def _dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def _view(w, h, seed=3, radius=4.0, fov=50.0):
    return S.look_at_rays(S.Camera(S.sphere_point(radius, seed), w, h, fov))


def _rays(kind):
    rng = np.random.default_rng(7)
    if kind == "random":  # no order at all: the rounds
        o = rng.standard_normal((777, 3)).astype(np.float32)
        d = rng.standard_normal((777, 3)).astype(np.float32)
        return o, d / np.linalg.norm(d, axis=1, keepdims=True)
    if kind == "shuffled":  # one apex, directions in no order
        o, d = _view(64, 40)
        p = rng.permutation(o.shape[0])
        return o[p], d[p]
    if kind == "patches":  # packets made of short runs from distant patches of the view
        o, d = _view(256, 200)
        at = (rng.integers(0, o.shape[0] - 7, 1500)[:, None] + np.arange(7)[None]).reshape(-1)
        return o[at], d[at]
    if kind == "inside":
        o, d = _view(50, 30)
        return (o * np.float32(0.05)), d
    if kind == "parallel":  # one direction, origins on a grid
        x, y = np.meshgrid(np.linspace(-1, 1, 40), np.linspace(-1, 1, 30))
        o = np.stack([x, y, np.full_like(x, 4.0)], -1).reshape(-1, 3).astype(np.float32)
        return o, np.broadcast_to(np.array([0.0, 0.0, -1.0], np.float32), o.shape).copy()
    w, h = kind
    return _view(w, h)


def _scene(kind):
    if kind == "shells":  # 60 nested ellipsoids: every ray holds far more events than the buffer
        n = 60
        r = np.linspace(0.2, 1.4, n, dtype=np.float32)
        rng = np.random.default_rng(5)
        q = rng.standard_normal((n, 4)).astype(np.float32)
        return S.SceneArrays(mean=(0.02 * rng.standard_normal((n, 3))).astype(np.float32),
                             scale=np.stack([r, 1.1 * r, 0.9 * r], 1), quat=q / np.linalg.norm(q, axis=1, keepdims=True),
                             density=np.full((n, 1), 0.05, np.float32),
                             features=rng.standard_normal((n, 1, 3)).astype(np.float32))
    if kind == "dense":  # hundreds of leaves per packet: lists cut into stages
        return S.uniform_scene(20_000, 0, seed=8)
    if kind == "sheets":
        return S.clustered_scene(60_000, 0, seed=9, n_clusters=120)
    return S.uniform_scene(kind, 0, seed=11)


def _trace(sc, o, d, traversal, kbuf=16, tmin=0.0, tmax=1000.0, order=None, hint=None):
    dev = _dev()
    t = lambda a: torch.tensor(np.ascontiguousarray(a), device=dev)
    scene = T.Scene(t(sc.mean), t(sc.scale), t(sc.quat), t(sc.density.reshape(-1)), t(sc.features))
    ro, rd = t(o), t(d)
    order = T.ray_order(ro, rd) if order == "sorted" else None
    f = T.forward(scene, ro, rd, tmin, tmax, 300, touch_count=True, ray_order=order, tune=T.Tune(kbuf, 128, traversal),
                  depth_hint=None if hint is None else t(hint))
    tri = T.reference_tri_collection(scene, f, 300, order)
    return f, tri


# 1, 37: a lone ragged packet; 592, 4,736, 9,472, 18,944, 37,888 rays: the last that packets of
# 4 (twice), 4, 8 and 16 take on 148 SMs, one ray more on the next width
CASES = [(s, r, k, tmin) for s, r, k, tmin in (
    (1, (5, 3), 16, 0.0), (2, (37, 1), 16, 0.0), (300, (37, 16), 8, 0.0), (1000, (128, 74), 16, 0.1),
    (1000, (9473, 1), 16, 0.0), (1000, (256, 74), 32, 0.0), (1000, (18945, 1), 16, 0.0), (1000, (37889, 1), 16, 0.0),
    ("shells", (40, 30), 16, 0.0), ("shells", (40, 30), 8, 0.3), ("shells", "inside", 32, 0.0),
    ("dense", (48, 40), 16, 0.0), ("dense", "inside", 16, 0.05), ("dense", "parallel", 16, 0.0),
    ("dense", "random", 16, 0.0), ("sheets", (210, 200), 16, 0.0), ("sheets", (17, 13), 16, 0.0),
    ("sheets", "shuffled", 16, 0.0), ("sheets", "patches", 16, 0.0))]


@pytest.mark.parametrize("order", ["given", "sorted"])
@pytest.mark.parametrize("scene,rays,kbuf,tmin", CASES, ids=lambda v: str(v).replace(" ", ""))
def test_equals_the_rounds(scene, rays, kbuf, tmin, order):
    sc = _scene(scene)
    o, d = _rays(rays)
    a, ta = _trace(sc, o, d, 0, kbuf, tmin, order=order)
    b, tb = _trace(sc, o, d, 2, kbuf, tmin, order=order)
    assert int(a.status.item()) == int(b.status.item())
    for k in ("out", "iters", "states", "last_dirac", "touch_count"):
        assert torch.equal(getattr(a, k), getattr(b, k)), k
    assert torch.equal(ta, tb)


@pytest.mark.parametrize("scene,rays,tmin,tmax", [(300, (37, 16), 0.0, 1000.0), ("shells", (23, 9), 0.2, 4.1),
                                                  (300, "inside", 0.0, 0.9), (2, (37, 1), 0.0, 1000.0)],
                         ids=lambda v: str(v).replace(" ", ""))
def test_events_equal_the_oracle(scene, rays, tmin, tmax):
    sc = _scene(scene)
    o, d = _rays(rays)
    f, tri = _trace(sc, o, d, 0, 16, tmin, tmax)
    ref = O.trace(O.Scene(sc.mean, sc.scale, sc.quat, sc.density.reshape(-1), sc.features), o, d, tmin, tmax, 300)
    it = f.iters.cpu().numpy()
    assert np.array_equal(it, ref.iters)
    mask = np.arange(300)[:, None] < it[None, :]
    tri = tri.cpu().numpy().reshape(300, -1)
    assert np.array_equal(np.where(mask, tri, -1), np.where(mask, ref.events, -1))


@pytest.mark.parametrize("guess", [0.01, 2.5, 3.6, 1e4])
def test_depth_hint_changes_nothing(guess):
    sc = _scene("sheets")
    o, d = _rays((210, 200))
    a, ta = _trace(sc, o, d, 0, order="sorted")
    b, tb = _trace(sc, o, d, 0, order="sorted", hint=np.full(o.shape[0], guess, np.float32))
    assert torch.equal(a.out, b.out) and torch.equal(a.iters, b.iters) and torch.equal(a.states, b.states)
    assert torch.equal(ta, tb)
