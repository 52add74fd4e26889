"""The colour quotients of an event and their derivatives are IEEE divisions: with one opaque
ellipsoid per ray (weight exactly 1) the image, the feature gradients and the density gradients
equal the same float32 operations in numpy, bit for bit."""
import numpy as np
import pytest
import torch

from ever_b200 import tracer as T

pytestmark = pytest.mark.gpu

C0 = np.float32(0.28209479177387814)
N = 4096


def _scene():
    r = np.random.default_rng(3)
    mean = np.stack([10.0 * np.arange(N), np.zeros(N), np.zeros(N)], 1)
    density = np.exp(r.uniform(np.log(100), np.log(3000), N)).astype(np.float32)
    features = (np.round(256 * r.standard_normal((N, 1, 3))) / 256).astype(np.float32)
    colour = (np.float64(C0) * features[:, 0] + 0.5).astype(np.float32)  # the fma: exact in 64 bits, then rounded
    arrays = (mean, np.ones((N, 3)), np.tile([1.0, 0, 0, 0], (N, 1)), density, features)
    return arrays, mean + [0, 0, 3.0], np.tile([0.0, 0, -1.0], (N, 1)), density[:, None], colour


def _traced(traversal):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    t = lambda a: torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda:0")
    arrays, o, d, sigma, colour = _scene()
    scene, ro, rd = T.Scene(*[t(a) for a in arrays]), t(o), t(d)
    fwd = T.forward(scene, ro, rd, tune=T.Tune(16, 128, traversal))
    assert bool((fwd.iters == 2).all())
    return fwd, scene, ro, rd, t, sigma, sigma * colour, colour


@pytest.mark.parametrize("traversal", [0, 1, 2])
def test_colours_are_the_quotients(traversal):
    fwd, _, _, _, _, sigma, sc, _ = _traced(traversal)
    assert np.array_equal(fwd.out[:, :3].cpu().numpy(), sc / sigma)


def test_gradients_are_the_quotients():
    fwd, scene, ro, rd, t, sigma, sc, colour = _traced(0)
    g = np.random.default_rng(4).standard_normal((N, 3)).astype(np.float32)
    grad = np.concatenate([g, np.zeros((N, 2))], 1)
    got = T.backward(scene, ro, rd, fwd, t(grad))
    gd = g / sigma  # d loss / d (density * colour) before the exit
    assert np.array_equal(got.features[:, 0].cpu().numpy(), np.clip(C0 * (sigma * gd), -1e3, 1e3))
    gx = ((-sc) / (sigma * sigma)) * g
    gx = (gx[:, 0] + gx[:, 1]) + gx[:, 2]
    want = ((gx + gd[:, 0] * colour[:, 0]) + gd[:, 1] * colour[:, 1]) + gd[:, 2] * colour[:, 2]
    assert np.array_equal(got.density.cpu().numpy(), np.clip(want, -50, 50))
