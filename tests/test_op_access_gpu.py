"""Per-op backward kernels at the alignments their accesses branch on: the shader's rows at 32- and
16-byte boundaries (the same bits), and the quadric gradients of even and odd cells in a buffer at an
8- and at a 4-byte boundary (one sample per cell, so no order of additions: the same bits)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _at(t, floats):
    buf = torch.zeros(t.numel() + floats, device=DEV)
    out = buf[floats:].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("n", [1, 127, 129])
@pytest.mark.parametrize("mode", ["compat", "fixed"])
def test_shader_rows_at_16_bytes(n, mode):
    from qsdvr_b200 import qsdvr as qs

    g = torch.Generator().manual_seed(n)
    nrm, view, gout, spec = (torch.randn((n, 3), generator=g).to(DEV) for _ in range(4))
    data = torch.randn((n, 32), generator=g).to(DEV)
    outs = []
    for shift_in, shift_out in ((0, 0), (4, 0), (0, 4), (4, 4)):
        d = _at(data, shift_in)
        ng, dg = torch.zeros((n, 3), device=DEV), _at(torch.zeros((n, 32), device=DEV), shift_out)
        qs.ShaderBackward(gout, nrm, view, d, spec, ng, dg, mode=mode)
        outs.append((ng, dg))
    assert outs[0][1].abs().max() > 0
    for ng, dg in outs[1:]:
        assert torch.equal(ng, outs[0][0]) and torch.equal(dg, outs[0][1])


@pytest.mark.parametrize("op", ["sdf", "normal"])
def test_cell_gradients_at_4_bytes(op):
    from qsdvr_b200 import qsdvr as qs

    R = 5
    g = torch.Generator().manual_seed(3)
    grid = torch.randn((R, R, R, 7), generator=g).to(DEV)
    index = torch.arange(R ** 3, dtype=torch.int32, device=DEV)  # one sample per cell, even and odd
    pts = (2 * torch.rand((R ** 3, 3), generator=g) - 1).to(DEV)
    gout = torch.randn(R ** 3 if op == "sdf" else (R ** 3, 3), generator=g).to(DEV)
    gout[::7] = 0.0
    outs = []
    for shift in (0, 1, 2, 3):
        gg = _at(torch.zeros_like(grid), shift)
        if op == "sdf":
            qs.SampleSDFBackward(gout, grid, pts, index, gg, R)
        else:
            qs.SampleNormalBackward(gout, grid, pts, index, gg)
        outs.append(gg)
    assert (outs[0].reshape(-1, 7)[1][:6] != 0).all() and not outs[0].reshape(-1, 7)[::7].any()
    for gg in outs[1:]:
        assert torch.equal(gg, outs[0])
