"""The ray order that the differentiable renders take for large batches: where the rule says so, and
gradients equal to those in batch order up to the order of their float atomics (1e-5 of the largest
entry, the bar of the other comparisons of float atomics; colours bit for bit)."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_rule():
    from qsdvr_b200 import fused

    def taken(n, R, channels=32):
        rays = torch.zeros((n, 4), dtype=torch.int32, device=DEV)
        o = torch.zeros((n, 3), device=DEV)
        data = torch.empty(((R + 1) ** 3, channels), device=DEV)
        return fused.gradient_order(rays, o, o, 0.01, data, R) is not None

    assert taken(16384, 128) and not taken(16383, 128)
    assert not taken(65536, 64) and not taken(16384, 256) and taken(32768, 256)


@pytest.mark.parametrize("model", ["f32", "bf16", "separable"])
def test_ordered_gradients_match_batch_order(model, monkeypatch):
    from qsdvr_b200 import fused, scenes
    from qsdvr_b200.camera import Camera

    R, interval = 112, 4.0 / 128  # 113^3 rows of 64 bytes (bf16): 92 MB
    cam = Camera(scenes.look_at((1.8, -3.2, 1.3), 130, 130, 180.0, 2.0, 6.0), interval, R)
    cam.GenerateRayPoints(torch.ones(130 * 130, dtype=torch.bool))
    rays = (cam.rayList, cam.originList, cam.dirList)
    target = torch.rand((130 * 130, 3), generator=torch.Generator().manual_seed(6)).to(DEV)
    if model == "separable":
        m = fused.SeparableRenderGrid(R, interval=interval)
        with torch.no_grad():
            m.offset.copy_(torch.tensor([2.0 - 2 * R, 2.0 - 2 * R, R, 0.8 * R * R]))
            m.zLayer.zero_()
    else:
        m = fused.DenseRenderGrid(R, 5.0, interval, mode="fixed", storage=model,
                                  sdf_grid=scenes.sphere_grid(R, 0.55, 0.0, device=DEV),
                                  data=scenes.appearance(R, seed=5, device=DEV))
    real, seen, outs = fused.gradient_order, [], []

    def noting(*args):
        order = real(*args)
        seen.append(order is not None)
        return order

    for rule in (noting, lambda *args: None):
        monkeypatch.setattr(fused, "gradient_order", rule)
        m.zero_grad(set_to_none=True)
        color = m(*rays)
        ((color - target) ** 2).mean().backward()
        outs.append((color.detach(), *(p.grad for p in m.parameters())))
    assert seen == [True]
    assert torch.equal(outs[0][0], outs[1][0])
    for a, b in zip(outs[0][1:], outs[1][1:]):
        assert a.abs().max() > 0 and rel_err(a.cpu(), b.cpu()) < 1e-5
    monkeypatch.setattr(fused, "gradient_order", noting)
    with torch.no_grad():  # no gradients, no order
        assert torch.equal(m(*rays), outs[0][0])
    assert seen == [True]
