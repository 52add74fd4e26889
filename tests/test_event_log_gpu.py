"""tri_collection from the event log: rows of whole and of broken 16-byte groups, one thread per
slot (blocks of 128), entries past a ray's events zero, camera slots as rays."""
import numpy as np
import pytest
import torch

from ever_b200 import camera as CAM
from ever_b200 import synthetic as S
from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (127, 1), (43, 3), (40, 33)])
@pytest.mark.parametrize("max_iters", [1, 4, 7, 30, 256])
def test_rows_and_zeros(w, h, max_iters):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = S.uniform_scene(400, 0, seed=4)
    t = lambda a: torch.tensor(np.ascontiguousarray(a, np.float32), device="cuda")
    scene = T.Scene(t(sc.mean), t(sc.scale), t(sc.quat), t(sc.density.reshape(-1)), t(sc.features))
    cam = S.Camera(S.sphere_point(3.0, 2), w, h, 50.0)
    wc, hc, f, c2w = S.pinhole(cam)
    camera = CAM.Camera(wc, hc, f, f, c2w)
    ro, rd = CAM.camera_rays(wc, hc, f, f, c2w)
    order = T.ray_order(ro, rd)
    full = T.forward(scene, ro, rd, 0.0, 1000.0, 256, tune=T.Tune(traversal=1))  # per-ray traversal
    ref = T.reference_tri_collection(scene, full, 256).view(256, -1)[:max_iters]
    for o in (None, order):
        fwd = T.forward(scene, ro, rd, 0.0, 1000.0, max_iters, ray_order=o)
        tri = T.reference_tri_collection(scene, fwd, max_iters, o).view(max_iters, -1)
        live = torch.arange(max_iters, device="cuda")[:, None] < fwd.iters[None]
        assert torch.equal(tri, torch.where(live, ref, torch.zeros_like(ref)))
    cf = CAM.forward(scene, camera, max_iters=max_iters)
    assert torch.equal(CAM.tri_collection(scene, camera, cf, max_iters).view(max_iters, -1), tri)
