"""Scenes whose rays are inside many ellipsoids at once. Their leaf lists do not fit or take many
passes, so stages end early, and packets hand their rays to the gather rounds: the first ones after
two rounds of their own, the others at once. The outputs are the same bits whichever way a ray
goes, and such a launch costs about what the rounds cost."""
import numpy as np
import pytest
import torch

from ever_b200 import camera as CAM
from ever_b200 import synthetic as S
from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu


def _scene(kind, n, deg=0):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = S.uniform_scene(n, deg, seed=3)
    if kind == "large":  # one in fifty is huge and faint: hundreds of leaves over every t
        sc.scale[: n // 50] *= 20
        sc.density[: n // 50] *= 0.01
    elif kind == "threefold":  # every ellipsoid three times: events in threes, many passes over a list
        k = n // 3
        for a in (sc.mean, sc.scale, sc.quat):
            a[k:2 * k] = a[:k]
            a[2 * k:3 * k] = a[:k]
        sc.density *= 0.1
    elif kind == "faint":
        sc.density *= 0.02
    t = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda:0")
    return T.Scene(t(sc.mean), t(sc.scale), t(sc.quat), t(sc.density), t(sc.features))


def _rays(kind, w, h):
    if kind == "parallel":
        x, y = np.meshgrid(np.linspace(-1, 1, w), np.linspace(-1, 1, h))
        o = np.stack([x, y, np.full_like(x, -4)], -1).reshape(-1, 3)
        d = np.broadcast_to(np.array([0.3, -0.2, 0.93]), o.shape)
    elif kind == "around":
        a, b = np.meshgrid(np.linspace(0, 2 * np.pi, w), np.linspace(0.01, np.pi - 0.01, h))
        d = np.stack([np.cos(a) * np.sin(b), np.sin(a) * np.sin(b), np.cos(b)], -1).reshape(-1, 3)
        o = np.full_like(d, 0.1)
    else:
        o, d = S.look_at_rays(S.Camera(S.sphere_point(3.0, 4), w, h, 45.0))
    t = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda:0")
    return t(o), t(d)


def _equal(fs, tris):
    for f, tri in zip(fs[1:], tris[1:]):
        for k in ("out", "states", "last_dirac", "iters", "touch_count", "ray_stats", "status"):
            assert torch.equal(getattr(fs[0], k), getattr(f, k)), k
        assert torch.equal(tris[0], tri)


# 64 x 37 rays: narrow packets, which run all rounds themselves; 193 x 197: the smallest full
# packets; 512 x 300: 4,800 packets, more than the 2,368 that run rounds of their own
@pytest.mark.parametrize("kind,n,rays,w,h,kbuf,tmin,deg", [
    ("large", 20_000, "view", 64, 37, 16, 0.0, 0), ("large", 20_000, "view", 193, 197, 16, 0.05, 0),
    ("large", 20_000, "view", 512, 300, 16, 0.0, 0), ("large", 20_000, "around", 512, 300, 8, 0.0, 0),
    ("large", 20_000, "parallel", 512, 300, 16, 0.0, 2), ("threefold", 30_000, "view", 64, 37, 8, 0.0, 0),
    ("threefold", 30_000, "view", 512, 300, 16, 0.0, 1), ("threefold", 30_000, "parallel", 512, 300, 16, 0.0, 0),
    ("faint", 60_000, "around", 512, 300, 16, 0.2, 0), ("faint", 60_000, "parallel", 193, 197, 32, 0.0, 0)])
@pytest.mark.parametrize("ordered", [True, False])
def test_same_bits(kind, n, rays, w, h, kbuf, tmin, deg, ordered):
    scene = _scene(kind, n, deg)
    ro, rd = _rays(rays, w, h)
    order = T.ray_order(ro, rd) if ordered else None
    fs = [T.forward(scene, ro, rd, tmin, 1000.0, 200, sh_degree=deg or None, touch_count=True, ray_stats=True,
                    ray_order=order, tune=T.Tune(kbuf, 128, m), regrouped=packed)
          for m, packed in ((0, True), (0, False), (2, True))]
    _equal(fs, [T.reference_tri_collection(scene, f, 200, order) for f in fs])
    assert float(fs[0].iters.float().mean()) > 20


def _camera(w, h):
    eye = S.sphere_point(3.0, 4)
    f = -eye / np.linalg.norm(eye)
    x = np.cross(f, [0, 0, 1.0])
    x /= np.linalg.norm(x)
    c2w = np.eye(4)
    c2w[:3, 0], c2w[:3, 1], c2w[:3, 2], c2w[:3, 3] = x, np.cross(f, x), f, eye
    return CAM.Camera(w, h, 1.2 * w, 1.2 * w, c2w)


@pytest.mark.parametrize("kind,w,h", [("large", 509, 301), ("large", 61, 37), ("threefold", 509, 301)])
def test_camera_same_bits(kind, w, h):
    scene = _scene(kind, 20_000)
    cam = _camera(w, h)
    fs = [CAM.forward(scene, cam, None, max_iters=200, touch_count=True, ray_stats=True, tune=T.Tune(16, 128, m),
                      regrouped=packed) for m, packed in ((0, True), (0, False), (2, False))]
    _equal(fs, [CAM.tri_collection(scene, cam, f, 200) for f in fs])


@pytest.mark.parametrize("rays", ["view", "camera"])
def test_many_leaves_over_one_t_cost_what_the_rounds_cost(rays):
    # lists that never fit, halved down to single rays, took five times as long
    scene = _scene("large", 50_000)
    ro, rd = _rays("view", 512, 512)
    order, cam = T.ray_order(ro, rd), _camera(512, 512)
    best = {0: 1e9, 2: 1e9}
    for _ in range(4):
        for m in best:
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            if rays == "view":
                T.forward(scene, ro, rd, log_events=False, ray_order=order, tune=T.Tune(16, 128, m))
            else:
                CAM.forward(scene, cam, None, log_events=False, tune=T.Tune(16, 128, m))
            b.record()
            torch.cuda.synchronize()
            best[m] = min(best[m], a.elapsed_time(b))
    print(f"{rays}: default {best[0]:.2f} ms, rounds {best[2]:.2f} ms")
    assert best[0] < 2.0 * best[2], best


@pytest.mark.parametrize("max_iters,kernels", [(0, 1), (1, 3)])
def test_no_iterations_need_no_second_kernel(max_iters, kernels):
    # the start density alone (sp.Forward's initial_drgb): neither vote nor rounds
    scene = _scene("large", 20_000)
    ro, rd = _rays("view", 256, 256)
    T.forward(scene, ro, rd, 0.0, 1000.0, max_iters)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        T.forward(scene, ro, rd, 0.0, 1000.0, max_iters)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "k_order_vote" in e.name or "k_trace_fwd" in e.name]
    assert len(names) == kernels, names
