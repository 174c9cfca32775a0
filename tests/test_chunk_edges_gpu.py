"""Rays whose render samples end at, before and after a 32-sample chunk's edge: the SDF sample that
one chunk hands to the next, in the train pass and in the forward + backward passes, against the
float64 oracle (image 1e-5 absolute, gradients 1e-4 relative, as the other fused tests), and the
loss, a sum of partial sums.  Its bound: at most 64 additions per warp, 128 per partial sum and 6
of the final tree and of the caller's value, each within 2^-24 of a sum of positive terms, and the
colours' own 1e-5."""
import numpy as np
import pytest
import torch

import oracle.oracle as O
from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"
COUNTS = (0, 2, 3, 32, 33, 34, 64, 65, 66, 97)  # SDF samples; a ray renders one fewer


@pytest.mark.parametrize("sh,storage", [(2, "f32"), (3, "f32"), (2, "bf16")])
@pytest.mark.parametrize("passes", ["train", "backward"])
def test_chunk_edges_vs_oracle(passes, sh, storage):
    from qsdvr_b200 import fused, scenes
    from qsdvr_b200.camera import Camera

    R, k, interval = 24, 6.0, 4.0 / 256
    cam = Camera(scenes.look_at((2.0, -3.1, 1.4), 24, 24, 70.0, 2.0, 6.0), interval, R)
    cam.GenerateRayPoints(torch.ones(24 * 24, dtype=torch.bool))
    full = cam.rayList[:, 0].cpu().numpy()
    n = np.minimum(np.resize(COUNTS, full.size), full)  # truncated rays, a mix of lengths
    n[n < 2] = 0
    nr = np.maximum(n - 1, 0)
    rays = np.stack([n, np.cumsum(n) - n, nr, np.cumsum(nr) - nr], 1).astype(np.int32)
    assert {31, 32, 33, 63, 64, 65} <= set(nr.tolist())
    o, d = cam.originList, cam.dirList
    inp = {a: torch.from_numpy(b) for a, b in
           O.generate_ray_points(rays, o.cpu().numpy(), d.cpu().numpy(), interval, R).items()}
    inp["rayList"] = torch.from_numpy(rays).long()
    cells = fused.pad_grid7(scenes.sphere_grid(R, 0.55, 0.01, seed=5).reshape(-1, 7)).to(DEV)
    data = scenes.appearance(R, seed=5, sh_degree=sh).to(DEV)
    target = torch.rand((n.size, 3), generator=torch.Generator().manual_seed(6)).to(DEV)
    stored, tr = (cells, data), "product"
    g7 = cells[:, :7].cpu()
    if storage == "bf16":
        stored, tr = (fused.sdf_cells_bf16(cells), data.to(torch.bfloat16)), "log"
        g7, data = O.sdf_cells_decode(stored[0]), stored[1].float()
    g7, dd = g7.double().requires_grad_(), data.double().cpu().requires_grad_()
    img = O.render(g7, dd, inp, k, False, sh)
    mse = ((img - target.double().cpu()) ** 2).mean()
    wg, wd = torch.autograd.grad(mse, (g7, dd))

    rt = torch.from_numpy(rays).to(DEV)
    sg = torch.zeros(cells.shape, device=DEV)
    dg = torch.zeros(data.shape, device=DEV)
    args = (rt, o, d, *stored, R, interval, k)
    if passes == "train":
        color, loss = fused.render_train(target, *args, sg, dg, "fixed", tr)
        want = mse.item() * img.numel()
        assert abs(loss.item() - want) <= (64 + 128 + 6) * 2.0 ** -24 * want + 2e-5 * img.numel() * want ** 0.5
    else:
        color = fused.render_forward(*args, "fixed", tr)
        fused.render_backward(2.0 / target.numel() * (color - target), *args, sg, dg, "fixed", tr)
    assert (color.cpu().double() - img.detach()).abs().max().item() < 1e-5
    assert rel_err(sg[:, :7].cpu(), wg) < 1e-4
    assert rel_err(dg.cpu(), wd) < 1e-4
