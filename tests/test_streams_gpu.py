"""Renders that share a device.  Modules of different configuration on two streams at once: each gets
the colours of its own single-stream run bit for bit, and its gradients up to the order of the float
atomics (1e-5 of the largest entry).  A captured step and later renders: the step's replay."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _models(R, interval):
    from qsdvr_b200 import fused, scenes

    def dense(storage, sh):
        return fused.DenseRenderGrid(R, 5.0, interval, mode="fixed", storage=storage,
                                     sdf_grid=scenes.sphere_grid(R, 0.55, 0.0, device=DEV), sh_degree=sh,
                                     data=scenes.appearance(R, seed=5, sh_degree=sh, device=DEV))

    return dense("f32", 2), dense("bf16", 3)


def _batches(R, interval):
    from qsdvr_b200 import scenes
    from qsdvr_b200.camera import Camera

    out = []
    for eye, size in (((1.8, -3.2, 1.3), 200), ((-2.1, -2.9, 1.6), 256)):
        cam = Camera(scenes.look_at(eye, size, size, 1.4 * size, 2.0, 6.0), interval, R)
        cam.GenerateRayPoints(torch.ones(size * size, dtype=torch.bool))
        out.append((cam.rayList, cam.originList, cam.dirList))
    return out


def test_two_modules_on_two_streams():
    R, interval = 112, 4.0 / 128
    models, batches = _models(R, interval), _batches(R, interval)
    grads = [tuple(p.requires_grad for p in m.parameters()) for m in models]
    assert all(all(g) for g in grads)

    def step(m, batch):
        m.zero_grad(set_to_none=True)
        color = m(*batch)
        (color ** 2).mean().backward()
        return (color.detach(), *(p.grad for p in m.parameters()))

    want = [step(m, b) for m, b in zip(models, batches)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in models]
    for _ in range(5):
        got = [None, None]
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i] = step(models[i], batches[i])
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert torch.equal(g[0], w[0])
            for a, b in zip(g[1:], w[1:]):
                assert rel_err(a.cpu(), b.cpu()) < 1e-5


def test_captured_step_outlives_larger_renders():
    """A captured training step replays the same colours and loss after separable models with larger
    workspaces have rendered and the allocator's free memory has been given back and overwritten."""
    from qsdvr_b200 import fused

    R, interval = 64, 4.0 / 128
    rays, o, d = _batches(R, interval)[0]
    m = _models(R, interval)[0]
    target = torch.rand((rays.shape[0], 3), generator=torch.Generator().manual_seed(1)).to(DEV)
    sg, dg = torch.zeros_like(m.sdfGrid), torch.zeros_like(m.renderData)
    loss = torch.zeros(1, device=DEV)

    def step():
        loss.zero_()
        order = fused.ray_order(rays, o, d, interval)
        return fused.render_train(target, rays, o, d, m.sdfGrid.detach(), m.renderData.detach(), R, interval, 5.0, sg, dg,
                                  "fixed", loss=loss, order=order)[0]

    want, want_loss = step().clone(), loss.item()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        color = step()
    for big in (96, 160):
        sep = fused.SeparableRenderGrid(big, interval=interval)
        sep.train_step(target, rays, o, d)
        del sep
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filled = torch.full((1 << 28,), 0xFF, dtype=torch.uint8, device=DEV)
    color.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(color, want)
    # the same positive terms in another order, each sum of at most 512 (a warp), 128 and 6 additions
    assert abs(loss.item() - want_loss) <= 2 * (512 + 128 + 6) * 2.0 ** -24 * want_loss
    assert bool((filled == 0xFF).all())
