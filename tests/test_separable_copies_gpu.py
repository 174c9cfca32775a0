"""The separable table gradient through the workspace's copies, through a workspace without room for
them and without a workspace (one ray per block): the same colours bit for bit, and table gradients
that differ by the order of float additions only (1e-5 of the component's largest entry, the bar of
the other comparisons of float atomics)."""
import ctypes

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("R", [9, 33])
@pytest.mark.parametrize("passes", ["train", "backward"])
def test_copies_match_direct(R, passes):
    from qsdvr_b200 import _lib, fused, scenes
    from qsdvr_b200.camera import Camera

    interval, k = 4.0 / 128, 5.0
    cam = Camera(scenes.look_at((1.8, -3.2, 1.3), 70, 70, 105.0, 2.0, 6.0), interval, R)
    cam.GenerateRayPoints(torch.ones(4900, dtype=torch.bool))
    g = torch.Generator().manual_seed(R)
    tables = fused.separable_tables(*(1 + 0.05 * torch.randn(R, generator=g).to(DEV) for _ in range(2)),
                                    0.05 * torch.randn(R, generator=g).to(DEV),
                                    torch.tensor([2.0 - 2 * R, 2.0 - 2 * R, R, 0.8 * R * R], device=DEV))
    data = scenes.appearance(R, seed=5).to(DEV)
    target = torch.rand((4900, 3), generator=g).to(DEV)
    rays = (cam.rayList, cam.originList, cam.dirList)
    grad_color = torch.rand((4900, 3), generator=g).to(DEV)
    outs = []
    for kind in ("copies", "short", "none"):
        color = torch.zeros((4900, 3), device=DEV)
        tg, dg, loss = torch.zeros_like(tables), torch.zeros_like(data), torch.zeros(1, device=DEV)
        a = fused.make_args(*rays, None, data, R, interval, k, color=color, target=target, grad_color=grad_color,
                            data_grad=dg, loss=loss, grad_scale=0.01, persistent=False, sdf_layers=tables,
                            sdf_layers_grad=tg)
        need = int(_lib.lib().qsdvr_render_workspace_size(ctypes.byref(a)))
        copies = 64 * (3 * R + 1) * 16
        size = {"copies": need, "short": need - copies, "none": 0}[kind]
        ws = torch.empty(max(size, 1), dtype=torch.uint8, device=DEV).fill_(0xff)
        if size:
            a.workspace, a.workspace_bytes = ws.data_ptr(), size
        _lib.call("qsdvr_render_" + passes, ctypes.byref(a),
                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        outs.append((color, tg, dg))
    assert outs[0][1].isfinite().all() and outs[0][1][:, :3].abs().max() > 0
    for color, tg, dg in outs[1:]:
        assert torch.equal(color, outs[0][0])
        for c in range(3):
            assert rel_err(tg[:, c].cpu(), outs[0][1][:, c].cpu()) < 1e-5
        assert rel_err(dg.cpu(), outs[0][2].cpu()) < 1e-5
