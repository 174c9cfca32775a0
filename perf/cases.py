"""The work that users of this framework have it do, as measurable cases.

A case names a path through the public entry points (``kind``), a grid resolution ``R`` and
the sizes and options of that path:

* ``train``      one step of the training loop up to the optimizer: gradients zeroed, the ray
                 order, then the fused forward + MSE + backward over a batch of random rays;
* ``train_list`` the same step at the proposal network's samples: 64 coarse MLP points and the
                 sampler place 32 fine samples per ray, which the fused kernel trains at;
* ``autograd``   the model as an ``nn.Module`` in a plain PyTorch step: forward, MSE, backward();
* ``separable``  the reference's own parametrisation (three layers, an offset, the appearance
                 grid) through its fused training step;
* ``ops``        the reference's per-op chain: the sample lists of one camera's view, then
                 RenderGrid forward and backward;
* ``frame``      a whole view: ray generation, rendering by the uniform march, image assembly;
* ``frame_proposal``  the same view at the proposal network's samples;
* ``adam``       the optimizer step over the grids;
* ``mlp_train``  the proposal network's loss gradient over a set of training points.

Grids, cameras and ray batches are made here from the seed with plain torch: quadric cells
fitted to a union of four spheres with N(0, noise) on each cell's distance (a grid in
training; frames use a nearly converged one), appearance rows distributed as a trained grid's
(SH DC around 0.5, small higher orders, colours in [0, 1]), pinhole cameras on the upper
hemisphere at radius 4.03 that look at the origin with 1111.1 px of focal length per 800.

``exact`` restates every path in float64 torch.  Sample positions and cells are part of the
definition of the path (the reference's float32 ray marching), so they are evaluated with its
float32 roundings; everything computed from them is float64.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from qsdvr_b200 import fused
from qsdvr_b200.camera import Camera
from qsdvr_b200.optim import FusedGridAdam
from qsdvr_b200.proposal import ProposalNet
from qsdvr_b200.qsdvr import CameraArgs
from qsdvr_b200.render import RenderGrid

K = 5.0  # logistic coefficient, the model's default
NEAR, FAR, RADIUS = 2.0, 6.0, 4.03
F64 = torch.float64


def listed():
    return [
        # a small CPU-sized problem: one 100 x 100 view's rays on a 64^3 grid, 64 samples a ray
        dict(name="train_64", kind="train", R=64, rays=10000, per_ray=64, sh=2, storage="f32", mode="compat"),
        # the headline training batch: 65536 random rays, 256 samples a ray, fp32, reference mode
        dict(name="train_256", kind="train", R=256, rays=65536, per_ray=256, sh=2, storage="f32", mode="compat"),
        # the precision form of that batch with the larger appearance model
        dict(name="train_256_bf16_sh3", kind="train", R=256, rays=65536, per_ray=256, sh=3, storage="bf16",
             mode="fixed"),
        # the smallest call: a short batch through autograd, where launches and host work count
        dict(name="autograd_64", kind="autograd", R=64, rays=1024, per_ray=64, sh=2, storage="f32", mode="fixed"),
        # an ordinary batch of the degree-3 model through autograd
        dict(name="autograd_128_sh3", kind="autograd", R=128, rays=8192, per_ray=256, sh=3, storage="f32",
             mode="fixed"),
        # the reference's own model trained through the fused kernels
        dict(name="separable_256", kind="separable", R=256, rays=65536, per_ray=256),
        # the reference's training step as its users write it: default grid and march interval
        dict(name="ops_128", kind="ops", R=128, size=200, interval=0.03),
        # training at the proposal network's samples
        dict(name="train_list_256", kind="train_list", R=256, rays=65536, per_ray=256, sh=2, storage="f32"),
        # the online update of the proposal network, at the trainer's default number of points
        dict(name="mlp_train", kind="mlp_train", R=128, points=65536),
        # a held-out view of the largest model: 384^3, bf16, degree 3, 800 x 800, 512 samples a ray
        dict(name="frame_384", kind="frame", R=384, size=800, per_ray=512, sh=3, storage="bf16"),
        # the same view at the proposal network's samples
        dict(name="frame_proposal_384", kind="frame_proposal", R=384, size=800, per_ray=512, sh=3, storage="bf16"),
        # the optimizer step of the headline model: 671 M parameters
        dict(name="adam_256", kind="adam", R=256, storage="f32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "train_list", "autograd", "separable", "ops", "frame",
                       "frame_proposal", "adam", "mlp_train"])
    R = _log_int(rng, 48, 256)
    case = dict(kind=kind, R=R)
    if kind == "mlp_train":
        return dict(case, points=_log_int(rng, 2000, 262144))
    if kind == "ops":
        return dict(case, R=_log_int(rng, 48, 160), size=rng.randint(64, 240), interval=rng.choice([0.03, 0.02, 1 / 64]))
    if kind == "adam":
        return dict(case, storage=rng.choice(["f32", "bf16"]))
    if kind == "separable":
        return dict(case, rays=_log_int(rng, 512, 65536), per_ray=rng.randint(64, 256))
    sh = rng.choice([2, 3])
    case.update(sh=sh, storage=rng.choice(["f32", "bf16"]))
    if kind in ("frame", "frame_proposal"):
        return dict(case, size=rng.randint(100, 640), per_ray=rng.randint(128, 512))
    case.update(rays=_log_int(rng, 512, 65536), per_ray=rng.randint(64, 256))
    if kind != "train_list":
        case["mode"] = "fixed" if sh == 3 else rng.choice(["compat", "fixed"])
    return case


# ----------------------------------------------------------------------------- inputs

def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _generator(seed, stream=0):
    return torch.Generator(device=_device()).manual_seed(1000003 * stream + int(seed))


def _channels(case):
    return 32 if case.get("sh", 2) == 2 else 64


def _spheres(seed):
    r = np.random.default_rng(seed)
    return [(r.uniform(-0.4, 0.4, 3), float(r.uniform(0.25, 0.4))) for _ in range(4)]


def _distance(p, seed):
    """Signed distance of the scene (a union of spheres) at p [..., 3], and its unit gradient
    and centre distance, from the nearest sphere."""
    best = None
    for c, r in _spheres(seed):
        v = p - torch.tensor(c, dtype=p.dtype, device=p.device)
        rho = torch.linalg.norm(v, dim=-1)
        d = rho - r
        n = v / rho.clamp_min(1e-4).unsqueeze(-1)
        if best is None:
            best = (d, n, rho)
        else:
            near = d < best[0]
            best = (torch.where(near, d, best[0]), torch.where(near.unsqueeze(-1), n, best[1]),
                    torch.where(near, rho, best[2]))
    return best


def _cells(R, seed, noise):
    """[R^3, 8] fp32 quadric cells of the scene: a3..a5 the unit gradient over R, a0..a2 half
    the curvature over R^2, a6 the distance at the cell centre plus N(0, noise); slot 7 is 0."""
    dev, gen = _device(), _generator(seed, 1)
    k = (2 * torch.arange(R, device=dev, dtype=torch.float32) + 1 - R) / R
    out = torch.zeros((R ** 3, 8), dtype=torch.float32, device=dev)
    for z0 in range(0, R, 32):
        z = k[z0:z0 + 32]
        p = torch.stack(torch.meshgrid(z, k, k, indexing="ij")[::-1], -1).reshape(-1, 3)
        d, n, rho = _distance(p, seed)
        o = out[z0 * R * R:z0 * R * R + p.shape[0]]
        o[:, 0:3] = 0.5 * (1 - n * n) / rho.clamp_min(2.0 / R).unsqueeze(-1) / R ** 2
        o[:, 3:6] = n / R
        o[:, 6] = d + noise * torch.randn(d.shape, generator=gen, device=dev)
    return out


def _cells_bf16(cells):
    """The bf16 storage form of the cells: a0..a5 rounded to nearest, a6 rescaled by the change
    of |a3..a5| and kept as the sum of two bf16 in slots 6 and 7."""
    out = cells.to(torch.bfloat16)
    for s in range(0, cells.shape[0], 1 << 24):
        a, b = cells[s:s + (1 << 24)], out[s:s + (1 << 24)]
        a6 = a[:, 6] * (torch.linalg.norm(b[:, 3:6].float(), dim=1) / torch.linalg.norm(a[:, 3:6], dim=1))
        b[:, 6] = a6.to(torch.bfloat16)
        b[:, 7] = (a6 - b[:, 6].float()).to(torch.bfloat16)
    return out


def _appearance(R, C, seed, dtype):
    """[(R+1)^3, C] vertex rows (SH coefficients packed as RGB triples, diffuse colour, metallic,
    ambient occlusion; the degree-3 rows end in zero padding)."""
    dev, gen = _device(), _generator(seed, 2)
    nsh = 27 if C == 32 else 48
    V = (R + 1) ** 3
    out = torch.zeros((V, C), dtype=dtype, device=dev)
    for s in range(0, V, 1 << 22):
        o = out[s:s + (1 << 22)]
        n = o.shape[0]
        sh = 0.1 * torch.randn((n, nsh), generator=gen, device=dev)
        sh[:, :3] = 0.5 + 0.5 * sh[:, :3]
        u = torch.rand((n, 5), generator=gen, device=dev)
        u[:, 4] = 0.5 + 0.5 * u[:, 4]
        o[:, :nsh] = sh
        o[:, nsh:nsh + 5] = u
    return out


def _grids(case, seed, noise):
    cells = _cells(case["R"], seed, noise)
    bf16 = case["storage"] == "bf16"
    data = _appearance(case["R"], _channels(case), seed, torch.bfloat16 if bf16 else torch.float32)
    return (_cells_bf16(cells) if bf16 else cells), data


def _look_at(position):
    """Columns: right, down and forward of a camera at ``position`` that looks at the origin."""
    f = -position / np.linalg.norm(position)
    right = np.cross(f, (0.0, 0.0, 1.0))
    right /= np.linalg.norm(right)
    return np.stack([right, np.cross(f, right), f], 1)


def _position(r):
    z, phi = r.uniform(0.05, 0.95), r.uniform(0.0, 2 * math.pi)
    s = math.sqrt(1 - z * z)
    return RADIUS * np.array([s * math.cos(phi), s * math.sin(phi), z])


def _interval(case):
    return case["interval"] if "interval" in case else (FAR - NEAR) / case["per_ray"]


def _batch(case, seed):
    """Random pixels of 100 views as ray tables: RayInfo records, the first in-box march point
    and the direction of each ray (rays that miss the volume have no samples)."""
    dev, gen, n, interval = _device(), _generator(seed, 3), case["rays"], _interval(case)
    r = np.random.default_rng(seed)
    pos = [_position(r) for _ in range(100)]
    rot = torch.tensor(np.stack([_look_at(p) for p in pos]), device=dev)
    pos = torch.tensor(np.stack(pos), device=dev)
    view = torch.randint(0, 100, (n,), generator=gen, device=dev)
    pixel = torch.randint(0, 800, (n, 2), generator=gen, device=dev)
    c = torch.cat([(pixel.to(F64) + 0.5 - 400.0) / 1111.1, torch.ones((n, 1), dtype=F64, device=dev)], 1)
    ray = (rot[view] @ c.unsqueeze(-1)).squeeze(-1)
    near, d = pos[view] + NEAR * ray, ray / torch.linalg.norm(ray, dim=1, keepdim=True)
    a, b = (-0.9995 - near) / d, (0.9995 - near) / d  # a margin to the volume's faces: every sample is inside
    t0, t1 = torch.minimum(a, b).amax(1).clamp_min(0.0), torch.maximum(a, b).amin(1)
    j0, j1 = torch.ceil(t0 / interval), torch.floor(t1 / interval)
    count = (j1 - j0 + 1).clamp_min(0).to(torch.int64)
    count = torch.where(count < 2, torch.zeros_like(count), count)
    render = (count - 1).clamp_min(0)
    rays = torch.stack([count, count.cumsum(0) - count, render, render.cumsum(0) - render], 1).to(torch.int32)
    origin = torch.where(count.unsqueeze(1) > 0, near + d * (j0 * interval).unsqueeze(1), torch.zeros_like(near))
    target = torch.rand((n, 3), generator=gen, device=dev)
    return rays.contiguous(), origin.float().contiguous(), d.float().contiguous(), target


def _camera_args(case, seed):
    p = _position(np.random.default_rng(seed + 1))
    a = CameraArgs()
    a.width, a.height = case["size"], case["size"]
    a.rotation, a.translation = _look_at(p).reshape(-1), p
    a.fx = a.fy = 1111.1 * case["size"] / 800
    a.cx = a.cy = -case["size"] / 2.0
    a.near, a.far = NEAR, FAR
    return a


def _layers(R, seed):
    """Layers and offset of a separable quadric grid: the paraboloid z = 0.2 - x^2 - y^2 with
    noise on every layer entry, as a grid in training has."""
    gen = torch.Generator().manual_seed(int(seed))
    x = 1 + 0.05 * torch.randn(R, generator=gen)
    y = 1 + 0.05 * torch.randn(R, generator=gen)
    z = 0.05 * torch.randn(R, generator=gen)
    k0 = 1.0 - R
    return x, y, z, torch.tensor([2 * k0, 2 * k0, float(R), 2 * k0 * k0 + R * k0 - 0.2 * R * R])


def _encode(p):
    """The proposal network's input features: p, sin and cos of pi 2^l p for l = 0..3, 1."""
    f = [p]
    for level in range(4):
        a = math.pi * 2 ** level * p
        f.append(torch.stack([torch.sin(a), torch.cos(a)], -1).flatten(-2))
    return torch.cat(f + [torch.ones_like(p[..., :1])], -1)


def _hidden(w, p):
    h1 = torch.relu(_encode(p) @ w[:2048].view(64, 32)[:, :28].T)
    return torch.relu(h1 @ w[2048:6144].view(64, 64).T + w[6144:6208])


def _network(seed):
    """Parameters of a proposal network that knows the scene: random hidden layers and an
    output layer fitted to the scene's density by ridge regression."""
    gen = torch.Generator().manual_seed(int(seed))
    w = torch.zeros(6280, dtype=F64)
    w[:2048].view(64, 32)[:, :28] = (torch.rand((64, 28), generator=gen, dtype=F64) * 2 - 1) * 0.6
    w[2048:6208] = (torch.rand(4160, generator=gen, dtype=F64) * 2 - 1) * 0.25
    p = torch.rand((8192, 3), generator=gen, dtype=F64) * 2 - 1
    h = torch.cat([_hidden(w, p), torch.ones((8192, 1), dtype=F64)], 1)
    y = 24.0 * torch.sigmoid(-_distance(p, seed)[0] / 0.05) - 1.0
    s = torch.linalg.solve(h.T @ h + 1e-2 * torch.eye(65, dtype=F64), h.T @ y)
    w[6208:6273] = s
    return w.float()


def _proposal(seed):
    net = ProposalNet(_device(), seed=0)
    net.params.copy_(_network(seed))
    net.params_bf16.copy_(net.params)
    return net


def _points(case, seed):
    """(x, y, z, density) training points of the proposal network."""
    gen = _generator(seed, 4)
    p = torch.rand((case["points"], 3), generator=gen, device=_device()) * 2 - 1
    d = _distance(p, seed)[0]
    return torch.cat([p, (20.0 * torch.sigmoid(-d / 0.05)).unsqueeze(1)], 1).contiguous()


def _moments(shape, seed):
    """Gradient, first and second moment of a grid some steps into training: about half of the
    rows are touched by a step."""
    gen = _generator(seed, 5)
    g, m, v = (torch.empty(shape, dtype=torch.float32, device=_device()) for _ in range(3))
    for s in range(0, shape[0], 1 << 22):
        o = g[s:s + (1 << 22)]
        hit = torch.rand((o.shape[0], 1), generator=gen, device=o.device) < 0.55
        o.copy_(1e-5 * torch.randn(o.shape, generator=gen, device=o.device) * hit)
        m[s:s + (1 << 22)] = 3e-6 * torch.randn(o.shape, generator=gen, device=o.device)
        v[s:s + (1 << 22)] = 1e-11 * (0.5 + torch.rand(o.shape, generator=gen, device=o.device))
    return g, m, v


def _adam_grids(case, seed):
    return {"sdf": _cells(case["R"], seed, 0.01), "data": _appearance(case["R"], 32, seed, torch.float32)}


def prepare(case, seed):
    kind, R = case["kind"], case["R"]
    dev = _device()
    s = dict(case=dict(case), interval=_interval(case) if kind not in ("adam", "mlp_train") else None)
    if kind in ("train", "train_list", "autograd"):
        s["sdf"], s["data"] = _grids(case, seed, 0.01)
        s["batch"] = _batch(case, seed)
        s["transmittance"] = "log" if case["storage"] == "bf16" else "product"
        if kind == "autograd":
            # the module holds fp32 masters and refreshes the bf16 copies itself
            cells, data = s.pop("sdf"), s.pop("data")
            if case["storage"] == "bf16":
                cells, data = _cells(R, seed, 0.01), data.float()
            s["model"] = fused.DenseRenderGrid(R, K, s["interval"], mode=case["mode"], storage=case["storage"],
                                               device=dev, sdf_grid=cells, data=data, sh_degree=case["sh"])
        else:
            s["sdf_grad"] = torch.zeros(s["sdf"].shape, dtype=torch.float32, device=dev)
            s["data_grad"] = torch.zeros(s["data"].shape, dtype=torch.float32, device=dev)
            s["loss"] = torch.zeros(1, dtype=torch.float32, device=dev)
        if kind == "train_list":
            s["net"] = _proposal(seed)
    elif kind == "separable":
        s["batch"] = _batch(case, seed)
        model = fused.SeparableRenderGrid(R, K, s["interval"], device=dev)
        with torch.no_grad():
            for p, v in zip((model.xLayer, model.yLayer, model.zLayer, model.offset), _layers(R, seed)):
                p.copy_(v)
            model.renderData.copy_(_appearance(R, 32, seed, torch.float32))
        s["model"] = model
    elif kind == "ops":
        model = RenderGrid(R, K, device=dev)
        q = model.quadricGrid
        with torch.no_grad():
            for p, v in zip((q.xLayer, q.yLayer, q.zLayer, q.offset), _layers(R, seed)):
                p.copy_(v)
            model.renderData.copy_(_appearance(R, 32, seed, torch.float32).view_as(model.renderData))
        s["model"] = model
        s["camera"] = Camera(_camera_args(case, seed), s["interval"], R, device=dev)
        s["camera"].GenerateRayPoints(torch.ones(case["size"] ** 2, dtype=torch.bool))
        s["target"] = torch.rand((case["size"] ** 2, 3), generator=_generator(seed, 6), device=dev)
    elif kind in ("frame", "frame_proposal"):
        s["sdf"], s["data"] = _grids(case, seed, 0.001)
        s["camera"] = Camera(_camera_args(case, seed), s["interval"], R, device=dev)
        s["mask"] = torch.ones(case["size"] ** 2, dtype=torch.bool)
        s["transmittance"] = "log" if case["storage"] == "bf16" else "product"
        if kind == "frame_proposal":
            s["net"] = _proposal(seed)
    elif kind == "adam":
        params = {k: torch.nn.Parameter(v) for k, v in _adam_grids(case, seed).items()}
        copies = None
        if case["storage"] == "bf16":
            copies = {p: torch.empty(p.shape, dtype=torch.bfloat16, device=dev) for p in params.values()}
        s["opt"] = FusedGridAdam(params.values(), lr=1e-2, bf16_copies=copies, sdf_cells=(params["sdf"],))
        for i, p in enumerate(params.values()):
            p.grad, m, v = _moments(p.shape, seed + i)
            s["opt"].state[p] = {"step": 20, "exp_avg": m, "exp_avg_sq": v}
        s["params"], s["copies"] = params, copies
    else:
        s["net"], s["points"] = _proposal(seed), _points(case, seed)
    return s


# ----------------------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    kind, R, interval = case["kind"], case["R"], s["interval"]
    if kind in ("train", "train_list"):
        rays, origin, direction, target = s["batch"]
        s["sdf_grad"].zero_()
        s["data_grad"].zero_()
        s["loss"].zero_()
        tlist, mode = None, case.get("mode", "fixed")
        if kind == "train_list":
            tlist = s["net"].sample(rays, origin, direction, interval, 0.25)
        order = fused.ray_order(rays, origin, direction, interval, tlist=tlist)
        color, loss = fused.render_train(target, rays, origin, direction, s["sdf"], s["data"], R, interval, K,
                                         s["sdf_grad"], s["data_grad"], mode, s["transmittance"], loss=s["loss"],
                                         tlist=tlist, order=order)
        out = dict(color=color, loss=loss, sdf_grad=s["sdf_grad"], data_grad=s["data_grad"])
        return dict(out, tlist=tlist) if tlist is not None else out
    if kind == "autograd":
        rays, origin, direction, target = s["batch"]
        model = s["model"]
        model.zero_grad(set_to_none=True)
        color = model(rays, origin, direction)
        loss = F.mse_loss(color, target)
        loss.backward()
        return dict(color=color.detach(), loss=loss.detach(), sdf_grad=model.sdfGrid.grad,
                    data_grad=model.renderData.grad)
    if kind == "separable":
        rays, origin, direction, target = s["batch"]
        model = s["model"]
        model.zero_grad(set_to_none=True)
        color, loss = model.train_step(target, rays, origin, direction)
        return dict(color=color, loss=loss, x=model.xLayer.grad, y=model.yLayer.grad, z=model.zLayer.grad,
                    offset=model.offset.grad, data_grad=model.renderData.grad)
    if kind == "ops":
        model, q = s["model"], s["model"].quadricGrid
        model.zero_grad(set_to_none=True)
        color = model(s["camera"].GetRayPoints())
        loss = F.mse_loss(color, s["target"])
        loss.backward()
        return dict(color=color.detach(), loss=loss.detach(), x=q.xLayer.grad, y=q.yLayer.grad, z=q.zLayer.grad,
                    offset=q.offset.grad, data_grad=model.renderData.grad)
    if kind in ("frame", "frame_proposal"):
        cam = s["camera"]
        cam.GenerateRayPoints(s["mask"])
        render = s["net"].render if kind == "frame_proposal" else fused.render_forward
        color = render(cam.rayList, cam.originList, cam.dirList, s["sdf"], s["data"], R, interval, K, "fixed",
                       s["transmittance"])
        return cam.whole_image(color)
    if kind == "adam":
        s["opt"].step()
        out = {}
        for name, p in s["params"].items():
            st = s["opt"].state[p]
            out[name] = dict(param=p.detach(), m=st["exp_avg"], v=st["exp_avg_sq"])
            if s["copies"] is not None:
                out[name]["copy"] = s["copies"][p]
        return out
    net = s["net"]
    net.grad.zero_()
    loss = net.gradients(s["points"])
    return dict(loss=loss, grad=net.grad)


# ----------------------------------------------------------------------------- work

def work(case):
    """Inputs read once, outputs written once.  A ray crosses about one unit of length inside the
    volume, half of a uniform march's samples carry weight, and each of those needs its cell
    and the 8 corner rows around it, of which the touched ones are read once."""
    kind, R = case["kind"], case["R"]
    if kind == "mlp_train":
        return dict(bytes=16.0 * case["points"] + 6 * 6280, flops=36864.0 * case["points"])
    V, cells = (R + 1.0) ** 3, float(R) ** 3
    if kind == "adam":
        n = 8 * cells + 32 * V
        return dict(bytes=n * (32 + (2 if case["storage"] == "bf16" else 0)), flops=12.0 * n)
    C = _channels(case)
    b = 2 if case.get("storage") == "bf16" else 4
    rays = float(case["rays"] if "rays" in case else case["size"] ** 2)
    samples = rays / _interval(case)
    active = samples / 2
    if kind in ("train_list", "frame_proposal"):
        samples = active = 24.0 * rays
    if kind == "separable":
        cell_read, cell_out = 0.0, 0.0
    elif kind == "ops":
        cell_read, cell_out = 0.0, 0.0
    else:
        cell_read = 8 * b * cells * (1 - math.exp(-2 * samples / cells))
        cell_out = 32 * cells
    read = rays * 52 + cell_read + C * b * V * (1 - math.exp(-8 * active / V))
    flops = samples * 60 + active * (16 * C + 12 * C)
    if kind in ("train_list", "frame_proposal"):
        flops += 64 * 0.75 * rays * 12288
    if kind in ("frame", "frame_proposal"):
        return dict(bytes=read, flops=flops)
    return dict(bytes=read + cell_out + 4 * C * V, flops=flops + active * 40 * C)


# ----------------------------------------------------------------------------- float64

def _f32(x):
    return x.to(torch.float32)


def _fma(a, b, c):
    """float32 fused multiply-add (the float64 product of two float32 is exact)."""
    return _f32(a.to(F64) * b.to(F64) + c.to(F64))


def _scalar(v, like):
    return torch.full((), float(v), dtype=torch.float32, device=like.device)


def _march(origin, direction, j, interval):
    """SDF sample j of each ray in float32: origin + (direction j) interval.  [B, J, 3]"""
    return _fma(direction.unsqueeze(1) * j.view(1, -1, 1).float(), _scalar(interval, origin), origin.unsqueeze(1))


def _midpoint(origin, direction, j, interval):
    t = (j.float() + 0.5) * _scalar(interval, origin)
    return _fma(direction.unsqueeze(1), t.view(1, -1, 1), origin.unsqueeze(1))


def _cell_of(p, R):
    """Cell index and local coordinates in [-1, 1)^3 of float32 points."""
    q = (p + 1.0) * (R / 2.0)
    c = torch.floor(q)
    u = q * 2.0 - (2.0 * c + 1.0)
    c = c.long()
    return c, u.to(F64)


def _quadric(a, u):
    """Value and gradient (in local coordinates) of the quadric of each cell row a."""
    value = (a[:, 0:3] * u * u + a[:, 3:6] * u).sum(1) + a[:, 6]
    return value, 2 * a[:, 0:3] * u + a[:, 3:6]


def _basis(v, sh):
    x, y, z = v.unbind(1)
    c1, c4, c6, c8 = 0.48860251190291992, 1.0925484305920792, 0.31539156525252, 0.54627421529603959
    b = [torch.full_like(x, 0.28209479177387814), c1 * x, c1 * y, c1 * z, c4 * x * z, c4 * x * y,
         c6 * (2 * y * y - z * z - x * x), c4 * y * z, c8 * (z * z - x * x)]
    if sh == 3:
        a3, b3, cc, d3, e3 = (math.sqrt(35 / (32 * math.pi)), math.sqrt(105 / (4 * math.pi)),
                              math.sqrt(21 / (32 * math.pi)), math.sqrt(7 / (16 * math.pi)),
                              math.sqrt(105 / (16 * math.pi)))
        b += [a3 * x * (3 * z * z - x * x), b3 * x * y * z, cc * x * (4 * y * y - z * z - x * x),
              d3 * y * (2 * y * y - 3 * z * z - 3 * x * x), cc * z * (4 * y * y - z * z - x * x),
              e3 * y * (z * z - x * x), a3 * z * (z * z - 3 * x * x)]
    return torch.stack(b, 1)


def _shade(normal, view, row, sh, compat):
    """Reflection shading.  The reference mode reads SH coefficient i from channels i..i+2, and
    its gradient writes it to channels 3i..3i+2."""
    nb = 9 if sh == 2 else 16
    r = view - 2 * (view * normal).sum(1, keepdim=True) * normal
    b = _basis(r, sh)
    packed = row[:, :3 * nb].reshape(-1, nb, 3)
    if compat:
        read = torch.stack([row[:, i:i + 3] for i in range(9)], 1).detach()
        spec = (b.unsqueeze(-1) * read).sum(1) + (b.detach().unsqueeze(-1) * (packed - packed.detach())).sum(1)
    else:
        spec = (b.unsqueeze(-1) * packed).sum(1)
    diffuse, metal, ao = row[:, 3 * nb:3 * nb + 3], row[:, 3 * nb + 3:3 * nb + 4], row[:, 3 * nb + 4:3 * nb + 5]
    return (diffuse * (1 - metal) + spec * metal) * ao


def _exact_render(count, origin, direction, R, interval, cell_rows, data, sh, compat, target=None, grads=None,
                  tlist=None):
    """Colours [N, 3] in float64 and, with a target, the loss sum; ``grads`` (the gradient grids
    of the cells and of the rows) receive the gradient of the mean squared error.  ``cell_rows``
    gives the 7 coefficients at flat cell indices."""
    n, dev = count.shape[0], count.device
    C = data.shape[1]
    color = torch.zeros((n, 3), dtype=F64, device=dev)
    loss = torch.zeros((), dtype=F64, device=dev)
    hit = torch.nonzero(count >= 2).flatten()
    base_R = R if compat else R + 1  # the reference addresses a cell's base vertex by the cell's index
    nv = R + 1
    order = hit[torch.argsort(count[hit])]
    per = max(1, int(4e8 // (C * 8 * 40)))  # active samples gathered at a time
    start = 0
    while start < order.numel():
        longest = 33 if tlist is not None else int(count[order[min(order.numel() - 1, start + 4095)]])
        ids = order[start:start + max(64, min(4096, per * 4 // longest))]
        start += ids.numel()
        o, d, cnt = origin[ids], direction[ids], count[ids]
        if tlist is not None:
            t = tlist[ids]
            ends = o.to(F64).unsqueeze(1) + d.to(F64).unsqueeze(1) * t.unsqueeze(-1)
            mids = o.to(F64).unsqueeze(1) + d.to(F64).unsqueeze(1) * (0.5 * (t[:, 1:] + t[:, :-1])).unsqueeze(-1)
            cnt = torch.full_like(cnt, 33)
        else:
            j = torch.arange(int(cnt.max()), device=dev)
            ends, mids = _march(o, d, j, interval), _midpoint(o, d, j[:-1], interval)
        B, S = ends.shape[0], ends.shape[1]
        live = torch.arange(S, device=dev).unsqueeze(0) < cnt.unsqueeze(1)  # SDF samples
        # SDF at the interval ends
        c1, u1 = _cell_of(ends[live], R)
        i1 = c1[:, 0] + c1[:, 1] * R + c1[:, 2] * R * R
        a1 = cell_rows(i1).requires_grad_(grads is not None)
        value, g1 = _quadric(a1, u1)
        s = value / torch.linalg.norm(g1, dim=1) / R
        ok = torch.ones_like(s, dtype=torch.bool) if compat else torch.isfinite(s) & (s.abs() <= 4.0)
        sdf = torch.zeros((B, S), dtype=F64, device=dev).masked_scatter(live, torch.where(ok, s, torch.zeros_like(s)))
        good = torch.zeros((B, S), dtype=torch.bool, device=dev).masked_scatter(live, ok)
        e = torch.exp(-K * sdf)
        x = (e[:, 1:] - e[:, :-1]) / (1 + e[:, 1:])
        on = good[:, 1:] & good[:, :-1] & (x > 0)
        alpha = torch.where(on, x, torch.zeros_like(x))
        T = torch.cumprod(torch.cat([torch.ones_like(alpha[:, :1]), 1 - alpha[:, :-1]], 1), 1)
        # colour of the samples that carry weight
        cr, ur = _cell_of(mids[on], R)
        ir = cr[:, 0] + cr[:, 1] * R + cr[:, 2] * R * R
        ar = cell_rows(ir).requires_grad_(grads is not None)
        nr = _quadric(ar, ur)[1]
        normal = nr / torch.linalg.norm(nr, dim=1, keepdim=True)
        w = (ur + 1) / 2
        v0 = cr[:, 0] + cr[:, 1] * base_R + cr[:, 2] * base_R * base_R
        corners, row = [], None
        for z in (0, 1):
            for y in (0, 1):
                for xx in (0, 1):
                    wt = ((w[:, 0] if xx else 1 - w[:, 0]) * (w[:, 1] if y else 1 - w[:, 1])
                          * (w[:, 2] if z else 1 - w[:, 2])).unsqueeze(1)
                    v = v0 + xx + y * nv + z * nv * nv
                    corners.append((v, wt))
                    part = data[v].to(F64) * wt
                    row = part if row is None else row + part
        row.requires_grad_(grads is not None)
        view = d.to(F64).unsqueeze(1).expand(B, S - 1, 3)[on]
        rgb = _shade(normal, view, row, sh, compat)
        weight = (alpha * T)[on]
        which = torch.nonzero(on)[:, 0]
        col = torch.zeros((B, 3), dtype=F64, device=dev).index_add(0, which, rgb * weight.unsqueeze(1))
        color[ids] = col.detach()
        if grads is not None:
            err = col.detach() - target[ids].to(F64)
            ga, gr, grow = torch.autograd.grad(col, (a1, ar, row), 2 * err / (3 * n))
            grads[0][:, :7].index_add_(0, i1, ga)
            grads[0][:, :7].index_add_(0, ir, gr)
            for v, wt in corners:
                grads[1].index_add_(0, v, grow * wt)
    if target is not None:
        loss = ((color - target.to(F64)) ** 2).sum()
    return color, loss


def _stored_rows(cells):
    """Reader of dense cells: 7 coefficients, a bf16 cell's a6 in two parts."""
    def rows(i):
        a = cells[i].to(F64)
        if cells.dtype == torch.bfloat16:
            a[:, 6] += a[:, 7]
        return a[:, :7].clone()
    return rows


def _layer_cells(x, y, z, offset):
    """[R, R, R, 7] cells of the separable grid (the reference's recurrences, in float64)."""
    def axis(a0, off):
        zero = a0.new_zeros(1)
        a3 = off + torch.cumsum(torch.cat([zero, 2 * a0[:-1] + 2 * a0[1:]]), 0)
        return a3, torch.cumsum(torch.cat([zero, 3 * a0[:-1] + a0[1:] + 2 * a3[:-1]]), 0)

    R = x.shape[0]
    (x3, x6), (y4, y6), (z5, z6) = axis(x, offset[0]), axis(y, offset[1]), axis(z, offset[2])

    def along(v, dim):
        shape = [1, 1, 1]
        shape[dim] = R
        return v.view(shape).expand(R, R, R)

    return torch.stack([along(x, 2), along(y, 1), along(z, 0), along(x3, 2), along(y4, 1), along(z5, 0),
                        along(x6, 2) + along(y6, 1) + along(z6, 0) + offset[3]], -1)


def _exact_layers(case, seed, count, origin, direction, target, mean):
    R = case["R"]
    layers = [v.to(_device()).to(F64).requires_grad_(True) for v in _layers(R, seed)]
    cells = _layer_cells(*layers).reshape(-1, 7)
    data = _appearance(R, 32, seed, torch.float32)
    grads = (torch.zeros((R ** 3, 7), dtype=F64, device=data.device),
             torch.zeros(data.shape, dtype=F64, device=data.device))
    flat = cells.detach()
    color, loss = _exact_render(count, origin, direction, R, _interval(case), lambda i: flat[i].clone(), data, 2, True,
                                target, grads)
    gx, gy, gz, go = torch.autograd.grad(cells, layers, grads[0])
    if mean:
        loss = loss / color.numel()
    return color, loss, gx, gy, gz, go, grads[1]


def _ray_cut(case, seed):
    """Every pixel's ray of the camera in the reference's float32: sample count, first in-box
    march point, direction."""
    a, dev, interval = _camera_args(case, seed), _device(), _interval(case)
    n = case["size"] ** 2
    one = torch.zeros((), dtype=torch.float32, device=dev)
    rot = [_scalar(v, one) for v in np.asarray(a.rotation, np.float32)]
    tr = [_scalar(v, one) for v in np.asarray(a.translation, np.float32)]
    pid = torch.arange(n, device=dev)
    px, py = (pid % a.width).float() + 0.5, (pid // a.width).float() + 0.5

    def world(depth):
        z = _scalar(depth, one).expand(n)
        x = (px + _scalar(a.cx, one)) / _scalar(a.fx, one) * z
        y = (py + _scalar(a.cy, one)) / _scalar(a.fy, one) * z
        return torch.stack([_fma(rot[3 * i + 2], z, _fma(rot[3 * i], x, rot[3 * i + 1] * y)) + tr[i]
                            for i in range(3)], 1)

    near, far = world(a.near), world(a.far)
    d = far - near
    length = torch.sqrt(_fma(d[:, 2], d[:, 2], _fma(d[:, 0], d[:, 0], d[:, 1] * d[:, 1])))
    d = d / length.unsqueeze(1)
    f = far - near
    end = torch.where(d[:, 0] != 0, f[:, 0] / d[:, 0],
                      torch.where(d[:, 1] != 0, f[:, 1] / d[:, 1], f[:, 2] / d[:, 2]))
    steps = torch.floor(end / _scalar(interval, one)).clamp_min(0).long()
    count = torch.zeros(n, dtype=torch.long, device=dev)
    origin = torch.zeros((n, 3), dtype=torch.float32, device=dev)
    for s in range(0, n, 32768):
        e = min(n, s + 32768)
        j = torch.arange(int(steps[s:e].max()), device=dev)
        p = _march(near[s:e], d[s:e], j, interval)
        inside = (p.abs() < _scalar(0.9999, one)).all(-1) & (j.unsqueeze(0) < steps[s:e].unsqueeze(1))
        count[s:e] = inside.sum(1)
        first = inside.to(torch.int8).argmax(1)
        origin[s:e] = torch.where(inside.any(1, keepdim=True), p[torch.arange(e - s, device=dev), first],
                                  torch.zeros_like(near[s:e]))
    count = torch.where(count < 2, torch.zeros_like(count), count)
    return count, origin, d


def _exact_samples(w, count, origin, direction, interval, mix):
    """The 33 fine SDF positions of each ray from the network's densities at 64 coarse points."""
    n = count.shape[0]
    length = (count - 1).clamp_min(0).to(F64) * float(np.float32(interval))
    delta = (length / 64).unsqueeze(1)
    t = (torch.arange(64, device=count.device, dtype=F64) + 0.5) * delta
    out = torch.zeros((n, 33), dtype=F64, device=count.device)
    k = torch.arange(1, 32, device=count.device, dtype=F64) / 32
    for s in range(0, n, 16384):
        e = min(n, s + 16384)
        p = origin[s:e].to(F64).unsqueeze(1) + direction[s:e].to(F64).unsqueeze(1) * t[s:e].unsqueeze(-1)
        y = _hidden(w, p) @ w[6208:6272] + w[6272]
        keep = torch.exp(-F.softplus(y) * (count[s:e] >= 2).unsqueeze(1) * delta[s:e])
        T = torch.cumprod(torch.cat([torch.ones_like(keep[:, :1]), keep[:, :-1]], 1), 1)
        wt = T * (1 - keep)
        total = wt.sum(1, keepdim=True)
        pdf = torch.where(total > 0, (1 - mix) * wt / total.clamp_min(1e-300) + mix / 64, torch.full_like(wt, 1 / 64))
        cdf = torch.cumsum(pdf, 1)
        cdf = torch.cat([torch.zeros_like(cdf[:, :1]), cdf / cdf[:, -1:]], 1)
        lo = (torch.searchsorted(cdf, k.expand(e - s, 31).contiguous(), right=True) - 1).clamp(0, 63)
        a, b = cdf.gather(1, lo), cdf.gather(1, lo + 1)
        out[s:e, 1:32] = (lo + (k - a) / (b - a)) * delta[s:e]
        out[s:e, 32] = length[s:e]
    return torch.minimum(out, length.unsqueeze(1))


def exact(case, seed):
    kind, R = case["kind"], case["R"]
    dev = _device()
    if kind == "mlp_train":
        w = _network(seed).to(dev).to(torch.bfloat16).to(F64).requires_grad_(True)
        pts = _points(case, seed).to(F64)
        total, grad = 0.0, torch.zeros_like(w)
        for q in pts.split(65536):
            y = _hidden(w, q[:, :3]) @ w[6208:6272] + w[6272]
            e = torch.log1p(F.softplus(y)) - torch.log1p(q[:, 3])
            loss = (torch.where(e < 0, 4.0, 1.0) * e * e).sum() / pts.shape[0]
            grad += torch.autograd.grad(loss, w)[0]
            total = total + loss.detach()
        return dict(loss=total.reshape(1), grad=grad)
    if kind == "adam":
        out = {}
        for i, (name, p) in enumerate(_adam_grids(case, seed).items()):
            g, m, v = _moments(p.shape, seed + i)
            o = dict(param=torch.empty(p.shape, dtype=F64, device=dev), m=None, v=None, copy=None)
            o["m"], o["v"] = torch.empty_like(o["param"]), torch.empty_like(o["param"])
            for s in range(0, p.shape[0], 1 << 22):
                sl = slice(s, s + (1 << 22))
                gg, mm, vv = g[sl].to(F64), m[sl].to(F64), v[sl].to(F64)
                mm = mm + 0.1 * (gg - mm)
                vv = 0.999 * vv + 0.001 * gg * gg
                o["m"][sl], o["v"][sl] = mm, vv
                o["param"][sl] = p[sl].to(F64) - 1e-2 / (1 - 0.9 ** 21) * mm / (
                    torch.sqrt(vv) / math.sqrt(1 - 0.999 ** 21) + 1e-8)
            if case["storage"] == "f32":
                del o["copy"]
            out[name] = o
        return out
    if kind in ("frame", "frame_proposal"):
        count, origin, direction = _ray_cut(case, seed)
        cells, data = _grids(case, seed, 0.001)
        tlist = None
        if kind == "frame_proposal":
            w = _network(seed).to(dev).to(torch.bfloat16).to(F64)
            tlist = _exact_samples(w, count, origin, direction, _interval(case), 0.05)
        color, _ = _exact_render(count, origin, direction, R, _interval(case), _stored_rows(cells), data, case["sh"],
                                 False, tlist=tlist)
        return color.view(case["size"], case["size"], 3)
    if kind == "ops":
        count, origin, direction = _ray_cut(case, seed)
        target = torch.rand((case["size"] ** 2, 3), generator=_generator(seed, 6), device=dev)
        color, loss, gx, gy, gz, go, gd = _exact_layers(case, seed, count, origin, direction, target, True)
        return dict(color=color, loss=loss, x=gx, y=gy, z=gz, offset=go, data_grad=gd.view(R + 1, R + 1, R + 1, 32))
    rays, origin, direction, target = _batch(case, seed)
    count = rays[:, 0].long()
    if kind == "separable":
        color, loss, gx, gy, gz, go, gd = _exact_layers(case, seed, count, origin, direction, target, False)
        return dict(color=color, loss=loss.reshape(1), x=gx, y=gy, z=gz, offset=go, data_grad=gd)
    cells, data = _grids(case, seed, 0.01)
    if kind == "autograd" and case["storage"] == "bf16":
        cells, data = _cells_bf16(_cells(R, seed, 0.01)), data
    tlist = None
    if kind == "train_list":
        w = _network(seed).to(dev).to(torch.bfloat16).to(F64)
        tlist = _exact_samples(w, count, origin, direction, _interval(case), 0.25)
    grads = (torch.zeros(cells.shape, dtype=F64, device=dev), torch.zeros(data.shape, dtype=F64, device=dev))
    compat = case.get("mode", "fixed") == "compat"
    color, loss = _exact_render(count, origin, direction, R, _interval(case), _stored_rows(cells), data, case["sh"],
                                compat, target, grads, tlist)
    if kind == "autograd":
        return dict(color=color, loss=loss / color.numel(), sdf_grad=grads[0], data_grad=grads[1])
    if tlist is None:
        return dict(color=color, loss=loss.reshape(1), sdf_grad=grads[0], data_grad=grads[1])
    # the network's bf16 arithmetic moves a sample across cells of a noisy grid now and then, so
    # the gradients have no value that is meaningful entry by entry
    return dict(color=color, loss=loss.reshape(1), sdf_grad=None, data_grad=None, tlist=tlist)
