"""Launches whose rays come in no order: from the size on at which packets are full, the default
trace samples its packets and hands such a launch to the gather rounds in their own kernel. The
outputs are the same bits whichever way a launch goes, and it costs no more than the rounds."""
import numpy as np
import pytest
import torch

from ever_b200 import synthetic as S
from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu

FULL = 37_889  # the smallest launch of full packets on 148 SMs


def _scene(n, deg):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = S.uniform_scene(n, deg, seed=31)
    t = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda:0")
    return T.Scene(t(sc.mean), t(sc.scale), t(sc.quat), t(sc.density), t(sc.features))


def _rays(n, unordered, seed=5):
    """n rays: pixels of a view in scanline order, the packets of the share `unordered` random rays."""
    g = torch.Generator(device="cuda:0").manual_seed(seed)
    ro, rd = S.look_at_rays_device(S.Camera(S.sphere_point(3.0, 8), 256, n // 256 + 1, 45.0), torch.device("cuda:0"))
    ro, rd = ro[:n].clone(), rd[:n].clone()
    o = torch.randn((n, 3), device="cuda:0", generator=g)
    d = 0.5 * torch.randn((n, 3), device="cuda:0", generator=g) - 3 * o / o.norm(dim=1, keepdim=True)
    o, d = 3 * o / o.norm(dim=1, keepdim=True), d / d.norm(dim=1, keepdim=True)
    packet = torch.arange(n, device="cuda:0") // 32
    pick = (packet * unordered).floor() != ((packet + 1) * unordered).floor()  # evenly spaced packets
    ro[pick], rd[pick] = o[pick], d[pick]
    return ro.contiguous(), rd.contiguous()


# just below and above full packets; a ragged last packet; shares around one half
@pytest.mark.parametrize("n,unordered,deg,order", [
    (FULL - 1, 1.0, 0, False), (FULL, 1.0, 0, False), (FULL + 38, 1.0, 0, True), (40_007, 1.0, 2, False),
    (40_007, 0.0, 2, False), (65_536, 0.4, 0, False), (65_536, 0.6, 0, False), (262_151, 0.5, 0, False)])
def test_same_bits(n, unordered, deg, order):
    scene = _scene(3000, deg)
    ro, rd = _rays(n, unordered)
    order = T.ray_order(ro, rd) if order else None
    fs = [T.forward(scene, ro, rd, 0.05, 1000.0, 120, sh_degree=deg or None, touch_count=True, ray_stats=True,
                    ray_order=order, tune=T.Tune(16, 128, m), regrouped=packed)
          for m, packed in ((0, True), (0, False), (2, True))]
    tris = [T.reference_tri_collection(scene, f, 120, order) for f in fs]
    for f, tri in zip(fs[1:], tris[1:]):
        for k in ("out", "states", "last_dirac", "iters", "touch_count", "ray_stats", "status"):
            assert torch.equal(getattr(fs[0], k), getattr(f, k)), k
        assert torch.equal(tris[0], tri)
    assert int(fs[0].iters.sum()) > n


def test_random_rays_cost_what_the_rounds_cost():
    # called inside the frustum kernel the rounds take half as long again
    scene = _scene(20_000, 0)
    ro, rd = _rays(262_144, 1.0)
    best = {0: 1e9, 2: 1e9}
    for _ in range(6):
        for m in best:
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            T.forward(scene, ro, rd, log_events=False, tune=T.Tune(16, 128, m))
            b.record()
            torch.cuda.synchronize()
            best[m] = min(best[m], a.elapsed_time(b))
    print(f"random rays: default {best[0]:.2f} ms, rounds {best[2]:.2f} ms")
    assert best[0] < 1.25 * best[2], best
