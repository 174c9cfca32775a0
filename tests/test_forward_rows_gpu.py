"""The forward pass of larger fp32 degree-2 batches loads its rows in 16-byte pieces: the same colours
and opacities, bit for bit, as the same rays in parts that are below that kernel's line."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
LINE = 4096  # rays


@pytest.mark.parametrize("form", ["persistent", "plain", "list", "ordered", "unaligned"])
@pytest.mark.parametrize("mode,transmittance", [("compat", "product"), ("fixed", "product"), ("fixed", "log")])
@pytest.mark.parametrize("R,n", [(3, LINE), (20, LINE + 1), (61, 10000)])
def test_large_batch_matches_its_parts(R, n, mode, transmittance, form):
    from qsdvr_b200 import fused, proposal, scenes
    from qsdvr_b200.camera import Camera

    interval = 4.0 / 150
    cam = Camera(scenes.look_at((1.8, -3.2, 1.3), 101, 100, 140.0, 2.0, 6.0), interval, R)
    cam.GenerateRayPoints(torch.ones(10100, dtype=torch.bool))
    rays, o, d = (t[-n:].contiguous() for t in (cam.rayList, cam.originList, cam.dirList))
    rays, _ = proposal.with_offsets(rays)
    cells = fused.pad_grid7(scenes.sphere_grid(R, 0.55, 0.01, seed=5).reshape(-1, 7)).to(DEV)
    data = scenes.appearance(R, seed=5).to(DEV)
    if form == "unaligned":
        buf = torch.empty(data.numel() + 4, device=DEV)
        buf[4:].copy_(data.reshape(-1))
        data = buf[4:].view(data.shape)
        assert data.data_ptr() % 32 == 16
    tlist = proposal.uniform_tlist(rays, interval) if form == "list" else None

    def render(i, j):
        part = rays[i:j].contiguous()
        alpha = torch.zeros(n * 132, device=DEV)  # at most 2 sqrt(3) / interval + 2 samples a ray
        t = tlist[i:j].contiguous() if tlist is not None else None
        if t is not None:  # 32 samples a ray
            part[:, 3] = 32 * torch.arange(i, j, dtype=torch.int32, device=DEV)
        order = torch.arange(j - i - 1, -1, -1, dtype=torch.int32, device=DEV) if form == "ordered" else None
        color = fused.render_forward(part, o[i:j].contiguous(), d[i:j].contiguous(), cells, data, R, interval, 5.0,
                                     mode, transmittance, persistent=form != "plain", tlist=t, sample_alpha=alpha,
                                     order=order)
        return color, alpha

    color, alpha = render(0, n)
    parts = [render(i, min(i + LINE - 1, n)) for i in range(0, n, LINE - 1)]
    assert torch.equal(color, torch.cat([c for c, _ in parts]))
    assert torch.equal(alpha, sum(a for _, a in parts))
    assert color.isfinite().all() and color.abs().max() > 0 and alpha.max() > 0
