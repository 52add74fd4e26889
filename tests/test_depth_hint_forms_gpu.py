"""depth_from_prediction takes every form of its arguments that its torch expression takes, also
those that its kernel does not: the results are the CPU's."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from ever_b200 import scheduler as SCH

pytestmark = pytest.mark.gpu


def _inputs(dev="cuda"):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator().manual_seed(5)
    return [torch.randn((301, k), generator=g).to(dev) for k in (2, 3, 3)]


def _close(got, want):
    # a dozen float32 roundings of terms of a few tens at most (|d| >= 0.17 here), as on the CPU
    assert torch.allclose(got.cpu(), want, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("centre", [0.5, (0.5,), [[0.1, -0.2, 0.3]], torch.tensor([0.1, -0.2, 0.3])],
                         ids=["number", "one", "row", "tensor"])
def test_centre_forms(centre):
    _close(SCH.depth_from_prediction(*_inputs(), centre, 1.7), SCH.depth_from_prediction(*_inputs("cpu"), centre, 1.7))


def test_scale_keeps_its_gradient():
    scale = torch.tensor(1.7, device="cuda", requires_grad=True)
    d = SCH.depth_from_prediction(*_inputs(), (0.1, -0.2, 0.3), scale)
    d.sum().backward()
    p, _, r = _inputs("cpu")
    _close(scale.grad.reshape(1), (p[:, 1] / r.norm(dim=1)).sum().reshape(1))


def test_forward_mode():
    def tangent(dev):
        p, o, d = _inputs(dev)
        with fwAD.dual_level():
            out = SCH.depth_from_prediction(p, fwAD.make_dual(o, torch.ones_like(o)), d, (0.1, -0.2, 0.3), 1.7)
            return fwAD.unpack_dual(out).tangent
    _close(tangent("cuda"), tangent("cpu"))


def test_vmap():
    def mapped(dev):
        p, o, d = _inputs(dev)
        return torch.vmap(lambda x: SCH.depth_from_prediction(x, o, d, (0.1, -0.2, 0.3), 1.7))(torch.stack([p, 2 * p]))
    _close(mapped("cuda"), mapped("cpu"))


def test_lazily_negated_view():
    p, o, d = _inputs()
    _close(SCH.depth_from_prediction(torch._neg_view(p), o, d), SCH.depth_from_prediction(-p.cpu(), o.cpu(), d.cpu()))


def test_out_over_an_input():
    want = SCH.depth_from_prediction(*_inputs("cpu"), (0.1, -0.2, 0.3), 1.7)
    p, o, d = _inputs()
    out = o.view(-1)[:p.shape[0]]
    assert SCH.depth_from_prediction(p, o, d, (0.1, -0.2, 0.3), 1.7, out=out) is out
    _close(out, want)
