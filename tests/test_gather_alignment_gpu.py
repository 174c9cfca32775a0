"""The gather's 32-byte loads against the 16-byte ones that serve an appearance grid at a 16-byte
boundary: the same colours bit for bit, and gradients that differ by the order of their float
atomics only (at most a few hundred additions per entry: 1e-5 of the largest), for each storage, degree and
kernel variant."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _at16(t):
    """A copy of t that starts 16 bytes past a 512-byte boundary."""
    n = 16 // t.element_size()
    buf = torch.empty(t.numel() + n, dtype=t.dtype, device=DEV)
    out = buf[n:].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 32 == 16
    return out


@pytest.mark.parametrize("sh,storage,mode,variant", [
    (2, "f32", "compat", "plain"), (2, "f32", "fixed", "merge"), (2, "f32", "compat", "separable"),
    (3, "f32", "fixed", "plain"), (2, "bf16", "fixed", "plain"), (3, "bf16", "fixed", "plain"),
    (3, "bf16", "fixed", "merge")])
def test_unaligned_grid_matches_aligned(sh, storage, mode, variant):
    from qsdvr_b200 import fused, scenes
    from qsdvr_b200.camera import Camera

    R, k, interval = 20, 5.0, 4.0 / 128
    cam = Camera(scenes.look_at((1.8, -3.2, 1.3), 40, 40, 60.0, 2.0, 6.0), interval, R)
    cam.GenerateRayPoints(torch.ones(1600, dtype=torch.bool))
    cells = fused.pad_grid7(scenes.sphere_grid(R, 0.55, 0.01, seed=5).reshape(-1, 7)).to(DEV)
    data = scenes.appearance(R, seed=5, sh_degree=sh).to(DEV)
    if storage == "bf16":
        cells, data = fused.sdf_cells_bf16(cells), data.to(torch.bfloat16)
    target = torch.rand((1600, 3), generator=torch.Generator().manual_seed(6)).to(DEV)
    layers = None
    if variant == "separable":
        g = torch.Generator().manual_seed(7)
        layers = fused.separable_tables(*(1 + 0.05 * torch.randn(R, generator=g).to(DEV) for _ in range(3)),
                                        torch.tensor([-20.0, 5.0, 30.0, -40.0], device=DEV))
        cells = None
    outs = []
    for d in (data, _at16(data)):
        args = (cam.rayList, cam.originList, cam.dirList, cells, d, R, interval, k)
        fwd = fused.render_forward(*args, mode, sdf_layers=layers)
        sg = torch.zeros(layers.shape if layers is not None else cells.shape, device=DEV)
        dg = torch.zeros(data.shape, device=DEV)
        color, _ = fused.render_train(target, *args, sg, dg, mode, sdf_layers=layers, merge=variant == "merge")
        sb, db = torch.zeros_like(sg), torch.zeros_like(dg)
        fused.render_backward(2.0 / target.numel() * (color - target), *args, sb, db, mode, sdf_layers=layers,
                              merge=variant == "merge")
        outs.append((fwd, color, sg, dg, sb, db))
    a, b = outs
    assert a[1].isfinite().all() and a[3].abs().max() > 0
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    for x, y in zip(a[2:], b[2:]):
        assert rel_err(y.cpu(), x.cpu()) < 1e-5
