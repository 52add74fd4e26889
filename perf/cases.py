"""The work this library is measured on: calls through its public entry points, with the
inputs a program has in hand before each call.

The cases are traces of synthetic scenes (forward only, and forward + backward through
autograd) from a 64x64 view of 1,000 ellipsoids to full-HD views of one and two million,
through trace_rays, trace_camera, the sp object API and the batched tracer, plus the
trainer's colour pre-pass and the ray-cost model. Scenes follow the distributions of
ever_b200.synthetic (uniform ellipsoids in a cube; ellipsoids clustered on thin sheets),
drawn on the GPU from the seed.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

import ever_b200.batched as batched
import ever_b200.camera as camera
import ever_b200.eval_sh as eval_sh
import ever_b200.scheduler as scheduler
import ever_b200.sp as sp
from ever_b200.fast_ellipsoid_splinetracer import trace_rays

C0 = 0.28209479177387814


# ------------------------------------------------------------------------------- cases
def listed():
    return [
        # a thumbnail render of a small scene: nothing but latency and launches
        _rays("render_small", "uniform", 1_000, 1, 64, 64, grad=False),
        # one training step on a thumbnail, called as the trainer calls it: extras, the
        # screen-space mean gradient through one camera matrix, 400 iterations at most
        _rays("train_small", "clustered", 20_011, 1, 123, 77, extras=True, wct=True, max_iters=400),
        # one training step on a mid-size scene with degree-3 features, DC colour
        _rays("train_mid", "uniform", 100_000, 16, 800, 800),
        # the headline: one training step, 1M ellipsoids, one full-HD view
        _rays("train_scene", "clustered", 1_000_000, 16, 1920, 1080),
        # the trainer's call on a downscaled photograph of odd size, rays starting off the camera
        _rays("train_trainer", "clustered", 300_007, 1, 979, 546, extras=True, wct=True, max_iters=400, tmin=0.2),
        # view-dependent colour evaluated along the rays in both passes
        _rays("train_sh3", "clustered", 200_000, 16, 640, 480, sh=3),
        # one training step with the rays made from the camera in the kernels
        dict(name="train_camera", kind="camera", scene="clustered", n=500_009, k=16, w=1237, h=822, grad=True),
        # a viewer's full-HD frame of a large scene, no gradients
        dict(name="render_camera", kind="camera", scene="clustered", n=2_000_000, k=1, w=1920, h=1080, grad=False),
        # a renderer that keeps its BVH: refit to moved ellipsoids, then one frame
        dict(name="frame_refit", kind="frame", scene="clustered", n=400_000, k=1, w=1280, h=720),
        # several views over several scenes in one persistent launch, replayed from a graph
        dict(name="batch_graph", kind="batch", n=400_000, k=16, views=8, w=960, h=540),
        # the trainer's colour pre-pass, forward and backward
        dict(name="prepass", kind="prepass", n=1_000_000, k=16, sh=3),
        # the ray-cost model's inference over one full-HD view
        dict(name="cost_predict", kind="cost", w=1920, h=1080),
    ]


def _rays(name, scene, n, k, w, h, grad=True, extras=False, wct=False, max_iters=500, tmin=0.0, sh=0):
    return dict(name=name, kind="rays", scene=scene, n=n, k=k, w=w, h=h, grad=grad, extras=extras, wct=wct,
                max_iters=max_iters, tmin=tmin, sh=sh)


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["rays"] * 6 + ["camera"] * 2 + ["frame", "batch", "prepass", "cost"])
    w = log_int(48, 1900)
    h = max(16, min(1080, int(w * rng.uniform(0.5, 1.0))))
    if kind == "rays":
        scene = rng.choice(["uniform", "clustered", "clustered"])
        n = log_int(300, 150_000 if scene == "uniform" else 1_000_000)
        trainer = rng.random() < 0.3
        k = 1 if trainer else rng.choice([1, 4, 9, 16])
        sh = rng.choice([0, 0, 0, 1, 2, 3])
        sh = sh if (sh + 1) ** 2 <= k else 0
        c = _rays("", scene, n, k, min(w, 979) if trainer else w, min(h, 546) if trainer else h,
                  grad=trainer or rng.random() < 0.75, extras=trainer, wct=trainer, max_iters=400 if trainer else 500,
                  tmin=rng.choice([0.0, 0.0, 0.05, 0.2]), sh=sh)
        del c["name"]
        return c
    if kind == "camera":
        return dict(kind="camera", scene=rng.choice(["uniform", "clustered"]), n=log_int(300, 150_000),
                    k=rng.choice([1, 16]), w=w, h=h, grad=rng.random() < 0.6)
    if kind == "frame":
        return dict(kind="frame", scene="clustered", n=log_int(300, 400_000), k=rng.choice([1, 16]), w=min(w, 1280),
                    h=min(h, 720))
    if kind == "batch":
        return dict(kind="batch", n=log_int(1_000, 400_000), k=rng.choice([1, 16]), views=rng.randint(2, 8),
                    w=min(w, 960), h=min(h, 540))
    if kind == "prepass":
        sh = rng.choice([0, 1, 2, 3])
        return dict(kind="prepass", n=log_int(1_000, 1_500_000), k=rng.choice([v for v in (1, 4, 9, 16)
                                                                              if v >= (sh + 1) ** 2]), sh=sh)
    return dict(kind="cost", w=w, h=h)


# ------------------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda")


def _gen(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed) * 1_000_003 + 17)


def _scene(g, scene, n, k):
    """(mean, scale, quat, density (n,1), features (n,k,3)), float32."""
    dev = _device()

    def uniform(lo, hi, shape):
        return lo + (hi - lo) * torch.rand(shape, generator=g, device=dev)

    def log_uniform(lo, hi, shape):
        return torch.exp(uniform(math.log(lo), math.log(hi), shape))

    def normal(shape):
        return torch.randn(shape, generator=g, device=dev)

    quat = normal((n, 4))
    quat = quat / quat.norm(dim=1, keepdim=True)
    if scene == "uniform":
        mean, scale = uniform(-1, 1, (n, 3)), log_uniform(0.02, 0.2, (n, 3))
        density, sd = log_uniform(0.1, 50.0, (n, 1)), 0.5 if k == 1 else 0.3
    else:  # thin sheets of about 500 ellipsoids each
        sheets = max(1, n // 500)
        centre = uniform(-2, 2, (sheets, 3))
        # random orthonormal frames by Gram-Schmidt
        a, b = normal((sheets, 3)), normal((sheets, 3))
        a = a / a.norm(dim=1, keepdim=True)
        b = b - (a * b).sum(1, keepdim=True) * a
        b = b / b.norm(dim=1, keepdim=True)
        frame = torch.stack([a, b, torch.linalg.cross(a, b)], 1)
        which = torch.randint(0, sheets, (n,), generator=g, device=dev)
        local = normal((n, 3)) * torch.tensor([0.3, 0.3, 0.01], device=dev)
        mean = centre[which] + (frame[which] * local[:, :, None]).sum(1)
        scale, density, sd = log_uniform(0.002, 0.05, (n, 3)), log_uniform(1.0, 200.0, (n, 1)), 0.3
    return mean.contiguous(), scale, quat, density, normal((n, k, 3)) * sd


def _camera(g, scene, w, h):
    """A pinhole looking at the origin from a random point: (focal length in pixels, 3x4
    camera-to-world matrix, float64, on the host)."""
    radius, fov = (3.0, 60.0) if scene == "uniform" else (4.0, 50.0)
    v = torch.randn(3, generator=g, device=_device(), dtype=torch.float64).cpu()
    eye = radius * v / v.norm()
    fwd = -eye / eye.norm()
    up = torch.tensor([0.0, 0.0, 1.0] if abs(float(fwd[2])) < 0.99 else [0.0, 1.0, 0.0], dtype=torch.float64)
    right = torch.linalg.cross(fwd, up)
    right = right / right.norm()
    down = torch.linalg.cross(fwd, right)
    return 0.5 * h / math.tan(math.radians(fov) / 2), torch.stack([right, down, fwd, eye], 1)


def _view_rays(f, c2w, w, h):
    m = c2w.to(_device())
    y, x = torch.meshgrid(torch.arange(h, dtype=torch.float64, device=_device()) + 0.5,
                          torch.arange(w, dtype=torch.float64, device=_device()) + 0.5, indexing="ij")
    d = torch.stack([(x - 0.5 * w) / f, (y - 0.5 * h) / f, torch.ones_like(x)], -1).reshape(-1, 3) @ m[:, :3].T
    d = d / d.norm(dim=1, keepdim=True)
    return m[:, 3].expand_as(d).float().contiguous(), d.float().contiguous()


def _grad_out(g, rays):
    # the gradient of a loss averaged over the view's pixels
    return torch.randn((rays, 5), generator=g, device=_device()) / rays


def _trace_inputs(case, seed):
    g = _gen(seed)
    scene = _scene(g, case["scene"], case["n"], case["k"])
    f, c2w = _camera(g, case["scene"], case["w"], case["h"])
    return scene, f, c2w, _grad_out(g, case["w"] * case["h"])


def prepare(case, seed):
    s = SimpleNamespace(case=case)
    kind = case["kind"]
    if kind == "prepass":
        g = _gen(seed)
        s.mean, _, _, _, s.features = _scene(g, "clustered", case["n"], case["k"])
        s.features.requires_grad_(True)
        s.cam = 4.0 * torch.nn.functional.normalize(torch.randn(3, generator=g, device=_device()), dim=0)
        s.grad = torch.randn((case["n"], 1, 3), generator=g, device=_device()) * 1e-3
        return s
    if kind == "cost":
        s.model = scheduler.CostModel((0.1, -0.05, 0.0), 2.0, device=_device(), params=_cost_params(seed))
        s.rayo, s.rayd = _cost_rays(case, seed)
        return s
    if kind == "batch":
        g = _gen(seed)
        sizes = [max(64, case["n"] // 8), max(64, case["n"] // 2), case["n"]]
        scenes = [_scene(g, "clustered", n, case["k"]) for n in sizes]
        scenes = [(m, sc, q, d.reshape(-1), f) for m, sc, q, d, f in scenes]
        views = []
        for v in range(case["views"]):
            w, h = (case["w"], case["h"]) if v % 2 == 0 else (max(8, case["w"] // 3), max(8, case["h"] // 3))
            views.append((v % 3, *_view_rays(*_camera(g, "clustered", w, h), w, h)))
        s.tracer = batched.BatchedTracer(scenes, views, graph=True)
        s.grad = _grad_out(g, s.tracer.R)
        return s
    scene, f, c2w, s.grad = _trace_inputs(case, seed)
    if kind == "frame":
        s.prims = sp.Primitives(_device())
        s.prims.add_primitives(scene[0], scene[1], scene[2], None, scene[3], scene[4])
        ctx = sp.OptixContext(_device())
        s.gas = sp.GAS(ctx, _device(), s.prims)
        s.forward = sp.Forward(ctx, _device(), s.prims)
        s.rayo, s.rayd = _view_rays(f, c2w, case["w"], case["h"])
        # the ellipsoids move a little after the build
        move = torch.randn(scene[0].shape, generator=_gen(seed + 1), device=_device()) * 1e-3
        s.prims.tensors[0].add_(move)
        return s
    if kind == "camera":
        s.params = [t.requires_grad_(case["grad"]) for t in scene]
        s.camera = camera.Camera(case["w"], case["h"], f, f, c2w)
        return s
    s.rayo, s.rayd = _view_rays(f, c2w, case["w"], case["h"])
    s.params = [t.requires_grad_(case["grad"]) for t in (*scene, s.rayo, s.rayd)]
    s.kwargs = dict(tmin=case["tmin"], max_iters=case["max_iters"], return_extras=case["extras"])
    if case["sh"]:
        s.kwargs["sh_degree"] = case["sh"]
    if case["wct"]:
        s.means2d = torch.zeros((case["n"], 2), device=_device(), requires_grad=True)
        s.kwargs.update(dL_dmeans2D=s.means2d, wcts=_wct(f, c2w, case["w"], case["h"]).reshape(1, 4, 4).float())
        s.params.append(s.means2d)
    return s


def _wct(f, c2w, w, h):
    """World-to-clip matrix of the camera in the trainer's row-vector convention."""
    view = torch.eye(4, dtype=torch.float64)
    view[:3] = c2w
    near, far = 0.01, 100.0
    proj = torch.zeros(4, 4, dtype=torch.float64)
    proj[0, 0], proj[1, 1], proj[2, 2] = 2 * f / w, 2 * f / h, far / (far - near)
    proj[2, 3], proj[3, 2] = -far * near / (far - near), 1.0
    return (proj @ torch.linalg.inv(view)).T.contiguous().to(_device())


def _cost_params(seed):
    return scheduler.init_params(int(seed) % 100_000)


def _cost_rays(case, seed):
    g = _gen(seed)
    f, c2w = _camera(g, "clustered", case["w"], case["h"])
    return _view_rays(f, c2w, case["w"], case["h"])


# --------------------------------------------------------------------------------- run
def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "prepass":
        out = eval_sh.sh_features(state.mean, state.features, state.cam, case["sh"])
        return dict(out=out, grad=torch.autograd.grad(out, state.features, state.grad)[0])
    if kind == "cost":
        return dict(pred=state.model.predict(state.rayo, state.rayd)[0])
    if kind == "batch":
        t = state.tracer
        t.step(state.grad)
        return dict(out=t.out, iters=t.iters, rayo=t.drayo, rayd=t.drayd,
                    scenes=[[g.mean, g.scale, g.quat, g.density, g.features] for g in t.grads])
    if kind == "frame":
        state.gas.refit(state.prims)
        r = state.forward.trace_rays(state.gas, state.rayo, state.rayd, 0.0, 1000.0, 256)
        return dict(color=r["color"], tri=r["tri_collection"], drgb=r["initial_drgb"], iters=r["saved"].iters,
                    touch=r["saved"].touch_count)
    if kind == "camera":
        out = camera.trace_camera(*state.params, state.camera)
        if not case["grad"]:
            return dict(out=out)
        return dict(out=out, grads=list(torch.autograd.grad(out, state.params, state.grad)))
    got = {}
    out = trace_rays(*state.params[:7], **state.kwargs)
    if case["extras"]:
        out, ex = out
        got.update(tri=ex["tri_collection"], iters=ex["iters"], touch=ex["touch_count"])
    got["out"] = out
    if case["grad"]:
        got["grads"] = list(torch.autograd.grad(out, state.params, state.grad))
    return got


def work(case):
    kind = case["kind"]
    if kind == "prepass":
        n, k, nb = case["n"], case["k"], (case["sh"] + 1) ** 2
        # means and the features of the degree in, colours out; again with the colour
        # gradients in and the feature gradients out
        return dict(bytes=n * 4 * (3 + 3 * nb + 3) + n * 4 * (3 + 3 * nb + 3 + 3 * k), flops=n * (12 * nb + 60))
    if kind == "cost":
        rays = case["w"] * case["h"]
        return dict(bytes=rays * 32, flops=rays * 2 * (39 * 64 + 64 * 64 + 64 * 2))
    if kind == "batch":
        sizes = [max(64, case["n"] // 8), max(64, case["n"] // 2), case["n"]]
        big, small = case["w"] * case["h"], max(8, case["w"] // 3) * max(8, case["h"] // 3)
        rays = (case["views"] + 1) // 2 * big + case["views"] // 2 * small
        prims = sum(sizes)
        # ellipsoids in and their gradients out; rays in, images out, image gradients in, ray
        # gradients and iteration counts out
        return dict(bytes=2 * prims * 4 * (11 + 3 * case["k"]) + rays * (24 + 20 + 20 + 24 + 4), flops=0)
    n, k, rays = case["n"], case["k"], case["w"] * case["h"]
    prim, ray = 4 * (11 + 3 * k), 24 if kind != "camera" else 0
    colour = 4 * (11 + 3 * max(1, (case.get("sh", 0) + 1) ** 2))  # what the colour in use reads
    b = n * colour + rays * (ray + 20)
    if kind == "frame":
        return dict(bytes=n * (colour + 4) + rays * (ray + 16 + 16 + 4) + 4 * 256 * rays, flops=0)
    if case["grad"]:
        b += n * prim + rays * (20 + ray)
    if case.get("extras"):
        b += rays * (4 + 4 * case["max_iters"]) + 4 * n
    if case.get("wct"):
        b += 8 * n
    return dict(bytes=b, flops=0)


# ------------------------------------------------------------------- results in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind == "prepass":
        return _exact_prepass(case, seed)
    if kind == "cost":
        return _exact_cost(case, seed)
    if kind in ("batch", "frame") or case["n"] * case["w"] * case["h"] > 250_000_000 or case.get("sh"):
        return None
    return _exact_trace(case, seed)


def _sh_basis(d, deg):
    x, y, z = d.unbind(-1)
    b = [torch.full_like(x, C0)]
    if deg > 0:
        b += [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if deg > 1:
        c = (1.0925484305920792, -1.0925484305920792, 0.31539156525252005, -1.0925484305920792, 0.5462742152960396)
        b += [c[0] * x * y, c[1] * y * z, c[2] * (2 * z * z - x * x - y * y), c[3] * x * z, c[4] * (x * x - y * y)]
    if deg > 2:
        c = (-0.5900435899266435, 2.890611442640554, -0.4570457994644658, 0.3731763325901154, -0.4570457994644658,
             1.445305721320277, -0.5900435899266435)
        b += [c[0] * y * (3 * x * x - y * y), c[1] * x * y * z, c[2] * y * (4 * z * z - x * x - y * y),
              c[3] * z * (2 * z * z - 3 * x * x - 3 * y * y), c[4] * x * (4 * z * z - x * x - y * y),
              c[5] * z * (x * x - y * y), c[6] * x * (x * x - 3 * y * y)]
    return torch.stack(b, -1)


def _exact_prepass(case, seed):
    s = prepare(case, seed)
    f = s.features.detach().double().requires_grad_(True)
    basis = _sh_basis(torch.nn.functional.normalize(s.mean.double() - s.cam.double(), dim=1), case["sh"])
    c = (basis[:, :, None] * f[:, :basis.shape[1]]).sum(1) + 0.5
    out = ((torch.nn.functional.softplus(c, beta=10) - 0.5) / C0).reshape(-1, 1, 3)
    return dict(out=out.detach(), grad=torch.autograd.grad(out, f, s.grad.double())[0])


def _exact_cost(case, seed):
    p = torch.tensor(_cost_params(seed), dtype=torch.float64, device=_device())
    rayo, rayd = (t.double() for t in _cost_rays(case, seed))
    o = rayo - torch.tensor([0.1, -0.05, 0.0], dtype=torch.float64, device=_device())
    d = rayd / rayd.norm(dim=1, keepdim=True)
    x = (o - (o * d).sum(1, keepdim=True) * d) / 2.0
    cols = [x]
    for q in range(6):
        cols += [torch.sin(math.pi * 2 ** q * x), torch.cos(math.pi * 2 ** q * x)]
    a = torch.cat(cols, 1)
    w1, w2, w3 = p[:4096].reshape(64, 64)[:, :39], p[4096:8192].reshape(64, 64), p[8192:9216].reshape(16, 64)
    a = torch.relu(a @ w1.T + p[9216:9280])
    a = torch.relu(a @ w2.T + p[9280:9344])
    return dict(pred=(a @ w3.T + p[9344:9360])[:, :2].contiguous())


def _local_frame(quat, scale):
    """W (n,3,3) with W (x - mean) the unit-sphere coordinates: rotation by the conjugate of
    the quaternion as given (not normalised), then division by the radii."""
    w, u = quat[:, :1], -quat[:, 1:]
    cols = []
    for e in torch.eye(3, dtype=quat.dtype, device=quat.device):
        t = 2 * torch.linalg.cross(u, e.expand_as(u))
        cols.append((e + w * t + torch.linalg.cross(u, t)) / scale)
    return torch.stack(cols, 2)


def _roots(frame, mean, o, d):
    """(discriminant, near t, far t) of |frame (o + t d - mean)| = 1."""
    oc, rd = (frame * (o - mean)[..., None, :]).sum(-1), (frame * d[..., None, :]).sum(-1)
    a, b = (rd * rd).sum(-1), (oc * rd).sum(-1)
    near = oc - (b / a)[..., None] * rd
    h = a * (1 - (near * near).sum(-1))
    r = torch.sqrt(h.clamp_min(1e-300)) / a
    return h, -b / a - r, -b / a + r


def _exact_trace(case, seed):
    """Brute force: every ray against every ellipsoid, events sorted per ray, the density
    between events integrated; gradients by autograd through the same expressions."""
    scene, f, c2w, grad = _trace_inputs(case, seed)
    rayo, rayd = _view_rays(f, c2w, case["w"], case["h"])
    rays, n, tmin, max_iters = rayo.shape[0], case["n"], case.get("tmin", 0.0), case.get("max_iters", 500)
    mean, scale, quat, density, feat, rayo, rayd = leaves = [t.double().requires_grad_(True)
                                                             for t in (*scene, rayo, rayd)]
    with torch.no_grad():
        o, d = rayo + tmin * rayd, torch.nn.functional.normalize(rayd, dim=1)
        frame, found = _local_frame(quat, scale), []
        step = max(1, 10_000_000 // n)
        for r in range(0, rays, step):
            oc = torch.einsum("nij,rnj->rni", frame, o[r:r + step, None] - mean[None])
            rd = torch.einsum("nij,rj->rni", frame, d[r:r + step])
            a, b = (rd * rd).sum(-1), (oc * rd).sum(-1)
            near = oc - (b / a)[..., None] * rd
            h = a * (1 - (near * near).sum(-1))
            hit = (h >= 0) & (-b / a + torch.sqrt(h.clamp_min(0)) / a > 0)
            hr, hj = torch.nonzero(hit, as_tuple=True)
            found.append(torch.stack([hr + r, hj]))
        ray, prim = torch.cat(found, 1)
        count = torch.bincount(ray, minlength=rays)
        most = max(1, int(count.max()))
        place = torch.arange(ray.numel(), device=ray.device) - (torch.cumsum(count, 0) - count)[ray]

    def padded(v, fill):
        t = torch.full((rays, most) + v.shape[1:], fill, dtype=v.dtype, device=v.device)
        return t.index_put((ray, place), v)

    o, d = rayo + tmin * rayd, rayd / rayd.norm(dim=1, keepdim=True)
    _, t0, t1 = _roots(_local_frame(quat, scale)[prim], mean[prim], o[ray], d[ray])
    sigma, colour = density[:, 0], C0 * feat[:, 0] + 0.5
    drgb = torch.cat([sigma[:, None], sigma[:, None] * colour], 1)[prim]
    inside = t0 <= 0
    start = torch.zeros((rays, 4), dtype=torch.float64, device=o.device).index_add(
        0, ray, torch.where(inside[:, None], drgb, torch.zeros_like(drgb)))
    inf = float("inf")
    t = torch.cat([padded(torch.where(inside, torch.full_like(t0, inf), t0), inf), padded(t1, inf)], 1)
    step = torch.cat([padded(drgb, 0.0), padded(-drgb, 0.0)], 1)
    at = torch.argsort(t.detach(), 1)
    t, step = torch.gather(t, 1, at), torch.gather(step, 1, at[..., None].expand_as(step))
    real = torch.isfinite(t.detach()) & (t.detach() <= 1000.0)
    t = torch.where(real, t, torch.zeros_like(t))
    before = start[:, None] + torch.cumsum(step, 1) - step
    last = torch.cat([torch.zeros_like(t[:, :1]), t[:, :-1]], 1)
    with torch.no_grad():  # an event counts while the ray is not opaque before it
        area = torch.where(real, (before[..., 0] * (t - last)).clamp_min(0), torch.zeros_like(t))
        opaque = torch.cumsum(area, 1) - area >= 5.54
        used = real & ~opaque & (torch.arange(t.shape[1], device=t.device) < max_iters)
        iters = used.sum(1)
    zero = torch.zeros_like(t)
    filled = used & (before[..., 0].detach() > 1e-7)  # a gap has no colour of its own
    area = torch.where(filled, before[..., 0] * (t - last), zero)
    log_t = torch.cumsum(area, 1)
    w = -torch.expm1(-area) * torch.exp(-(log_t - area))
    rgb = before[..., 1:] / torch.where(filled, before[..., 0], torch.ones_like(t))[..., None]
    image = (w[..., None] * torch.where(filled[..., None], rgb, torch.zeros_like(rgb))).sum(1)
    x = torch.where(used, (t + last) * 500.0, torch.ones_like(t))
    m = torch.where(used, (1.1 / -0.1) * ((x / 1.1 + 1) ** -0.1 - 1), zero)
    w = torch.where(used, w, zero)
    before_w, before_wm = torch.cumsum(w, 1) - w, torch.cumsum(w * m, 1) - w * m
    dist = (2 * w * (m * before_w - before_wm)).sum(1)
    out = torch.cat([image, (1 - torch.exp(-log_t[:, -1:])), dist[:, None]], 1)
    got = dict(out=out.detach())
    if case.get("extras"):
        got.update(tri=None, iters=None, touch=None)
    if not case["grad"]:
        return got
    ended = (iters >= max_iters - 1) | (iters <= 0)
    wanted = leaves if case["kind"] == "rays" else leaves[:5]
    g = list(torch.autograd.grad(out, wanted, torch.where(ended[:, None], 0.0, grad.double())))
    gm = g[0]
    got["grads"] = [v.clamp(-50, 50) if i == 3 else v.clamp(-1e3, 1e3) for i, v in enumerate(g)]
    if case.get("wct"):
        wct = _wct(f, c2w, case["w"], case["h"]).float().double()
        inv = torch.linalg.inv(wct)
        z = (torch.cat([mean.detach(), torch.ones_like(mean[:, :1])], 1) * wct[:, 2]).sum(1, keepdim=True)
        got["grads"].append(z * (gm @ inv[:2, :3].T))
    return got
