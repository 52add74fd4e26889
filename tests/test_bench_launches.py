"""bench.py's count of the library's kernels per step, at sizes on either side of each rule that it
depends on, against the kernels that a profiler sees."""
import pytest
import torch

import bench
from ever_b200 import synthetic as S
from ever_b200.fast_ellipsoid_splinetracer import trace_rays


def test_default_step():
    assert bench.step_launches(1_000_000, 1920 * 1080) == 41


@pytest.mark.gpu
@pytest.mark.parametrize("prims,w,h", [(1000, 64, 64), (8193, 91, 91), (32_768, 256, 128), (32_769, 256, 148),
                                       (40_000, 300, 127)])
def test_counts_what_runs(prims, w, h):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = S.uniform_scene(prims, 1, seed=2)
    t = [torch.tensor(a, device="cuda:0").requires_grad_(True)
         for a in (sc.mean, sc.scale, sc.quat, sc.density, sc.features)]
    ro, rd = S.look_at_rays_device(S.Camera(S.sphere_point(3.0, 2), w, h, 40.0), torch.device("cuda:0"))

    def step():
        trace_rays(*t, ro, rd, max_iters=64).sum().backward()

    step()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        step()
        torch.cuda.synchronize()
    seen = [e.name for e in prof.events() if "ever::" in e.name]
    assert len(seen) == bench.step_launches(prims, ro.shape[0]), sorted(seen)
