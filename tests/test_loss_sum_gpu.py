"""The loss that a train pass accumulates: the squared errors of the colours that it returns, summed
over warps, partial sums and a tree, added to what the caller's loss held.  All terms are positive, so
the sum is off by at most its longest chain of additions in units of 2^-24: a warp's rays (of 10000 over
2368 warps fewer than 64, three terms each), a partial sum's warps (74), 6 of the tree and the last.
A single ray's share of the loss is an order above that."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("persistent", [True, False])
@pytest.mark.parametrize("sh,storage", [(2, "f32"), (3, "bf16")])
def test_loss_is_the_sum_over_the_returned_colours(sh, storage, persistent):
    from qsdvr_b200 import fused, scenes
    from qsdvr_b200.camera import Camera

    R, interval, n, held = 24, 4.0 / 128, 10000, 0.75
    cam = Camera(scenes.look_at((1.8, -3.2, 1.3), 100, 100, 140.0, 2.0, 6.0), interval, R)
    cam.GenerateRayPoints(torch.ones(n, dtype=torch.bool))
    cells = fused.pad_grid7(scenes.sphere_grid(R, 0.55, 0.01, seed=5).reshape(-1, 7)).to(DEV)
    data = scenes.appearance(R, seed=5, sh_degree=sh).to(DEV)
    if storage == "bf16":
        cells, data = fused.sdf_cells_bf16(cells), data.to(torch.bfloat16)
    target = torch.rand((n, 3), generator=torch.Generator().manual_seed(6)).to(DEV)
    sg, dg = torch.zeros(cells.shape, device=DEV), torch.zeros(data.shape, device=DEV)
    loss = torch.full((1,), held, device=DEV)
    color, out = fused.render_train(target, cam.rayList, cam.originList, cam.dirList, cells, data, R, interval, 5.0, sg,
                                    dg, "fixed", loss=loss, persistent=persistent)
    assert out.data_ptr() == loss.data_ptr()
    want = held + ((color - target).double() ** 2).sum().item()
    # without the persistent grid every ray adds to the caller's loss by itself: a chain of n additions,
    # whose roundings are of either sign (8 standard deviations of n of them)
    chain = 3 * 64 + 74 + 6 + 1 if persistent else 8 * (n / 3) ** 0.5 + 4
    assert abs(loss.item() - want) <= chain * 2.0 ** -24 * want
