"""A camera's default forward allocates its outputs and nothing else: the workspace of the packed
gather rounds belongs to the traversal that packs them."""
import numpy as np
import pytest
import torch

from ever_b200 import camera as CAM
from ever_b200 import synthetic as S
from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu


def test_camera_forward_allocates_its_outputs_only():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = S.uniform_scene(500, 0, seed=3)
    t = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda:0")
    scene = T.Scene(t(sc.mean), t(sc.scale), t(sc.quat), t(sc.density), t(sc.features))
    cam = CAM.Camera(640, 480, 500.0, 500.0, np.array([[1.0, 0, 0, 0], [0, 1, 0, 0], [0, 0, 1, -3.0]]))
    CAM.forward(scene, cam, None, log_events=False)
    torch.cuda.synchronize()
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    CAM.forward(scene, cam, None, log_events=False)
    # out, states, last_dirac, iters, status
    assert torch.cuda.memory_stats()["allocation.all.allocated"] - before == 5
