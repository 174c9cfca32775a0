"""The separable layers' kernels (LayerToGrid forward and backward, the fused renderer's tables
and their adjoint) at the edges of their blocking: grids below one warp, around warps and
blocks, and the largest R the entry points take.

The recurrences are the reference's host loops in float32, one rounding per operation
(kernel/surface.cu:161-178, :301-334), so a float32 numpy loop gives the same bits.  The backward's
sums run in another order: with positive gradients every partial sum is positive, and each result
is off by at most (additions in its chain) * 2^-24 of its value: at most 1184 block sums, 1406 rows
per block, 16 warp and tile steps and two recurrences of R steps with up to three additions each.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
F = np.float32


def _layers(R, seed):
    r = np.random.default_rng(seed)
    return [r.uniform(-0.5, 0.5, R).astype(F) for _ in range(3)] + [r.uniform(-1, 1, 4).astype(F)]


def _axis(a0, off):
    a3, a6 = np.empty_like(a0), np.empty_like(a0)
    a3[0], a6[0] = off, 0
    for i in range(1, len(a0)):
        a3[i] = (F(2) * a0[i - 1] + F(2) * a0[i]) + a3[i - 1]
        a6[i] = ((F(3) * a0[i - 1] + a0[i]) + F(2) * a3[i - 1]) + a6[i - 1]
    return a3, a6


def _reverse(g0, g3, g6):
    """The reference's reverse loops, in the inputs' precision."""
    g0, g3, g6 = g0.copy(), g3.copy(), g6.copy()
    two, three = g0.dtype.type(2), g0.dtype.type(3)
    for i in range(len(g0) - 1, 0, -1):
        g0[i] += g6[i]
        g0[i - 1] += three * g6[i]
        g3[i - 1] += two * g6[i]
        g6[i - 1] += g6[i]
    for i in range(len(g0) - 1, 0, -1):
        g0[i] += two * g3[i]
        g0[i - 1] += two * g3[i]
        g3[i - 1] += g3[i]
    return g0, g3, g6


@pytest.mark.parametrize("R", [1, 2, 31, 33, 65, 257])
def test_layer_to_grid_edges(R):
    from qsdvr_b200 import qsdvr as qs

    x, y, z, off = _layers(R, R)
    out = torch.empty((R, R, R, 7), device=DEV)
    qs.LayerToGridForward(out, *(torch.from_numpy(v) for v in (x, y, z, off)))
    (x3, x6), (y4, y6), (z5, z6) = _axis(x, off[0]), _axis(y, off[1]), _axis(z, off[2])
    want = np.empty((R, R, R, 7), F)
    want[..., 0], want[..., 3] = x, x3
    want[..., 1], want[..., 4] = y[:, None], y4[:, None]
    want[..., 2], want[..., 5] = z[:, None, None], z5[:, None, None]
    want[..., 6] = ((x6 + y6[:, None]) + z6[:, None, None]) + off[3]
    assert np.array_equal(out.cpu().numpy(), want)

    g7 = np.random.default_rng(R + 1).uniform(0.5, 1.0, (R, R, R, 7)).astype(F)
    got = [torch.empty(R) for _ in range(3)] + [torch.empty(4)]
    qs.LayerToGridBackward(torch.from_numpy(g7).to(DEV), *got)
    g = g7.astype(np.float64)
    tol = (1184 + 1406 + 16 + 6 * R) * 2.0 ** -24
    for axis, (c0, c3, keep) in enumerate(((0, 3, 2), (1, 4, 1), (2, 5, 0))):
        other = tuple(a for a in range(3) if a != keep)
        g0, g3, _ = _reverse(*(g[..., c].sum(other) for c in (c0, c3, 6)))
        np.testing.assert_allclose(got[axis].numpy(), g0, rtol=tol)
        np.testing.assert_allclose(got[3][axis].item(), g3[0], rtol=tol)
    np.testing.assert_allclose(got[3][3].item(), g[..., 6].sum(), rtol=tol)


@pytest.mark.parametrize("R", [1, 2, 32, 33, 1290])
def test_separable_tables_and_adjoint_edges(R):
    from qsdvr_b200 import fused

    layers = _layers(R, R + 7)
    tables = fused.separable_tables(*(torch.from_numpy(v).to(DEV) for v in layers)).cpu().numpy()
    want = np.zeros((3 * R + 1, 4), F)
    for a in range(3):
        a3, a6 = _axis(layers[a], layers[3][a])
        want[a * R:(a + 1) * R, :3] = np.stack([layers[a], a3, a6], 1)
    want[3 * R, 0] = layers[3][3]
    assert np.array_equal(tables, want)

    tg = np.random.default_rng(R + 8).uniform(-1, 1, (3 * R + 1, 4)).astype(F)
    got = fused.separable_grad(torch.from_numpy(tg).to(DEV))
    for a in range(3):
        g0, g3, g6 = _reverse(*(np.ascontiguousarray(tg[a * R:(a + 1) * R, c]) for c in range(3)))
        assert np.array_equal(got[a].cpu().numpy(), g0)
        assert got[3][a].item() == g3[0]
        if a == 0:
            assert got[3][3].item() == g6[0]
