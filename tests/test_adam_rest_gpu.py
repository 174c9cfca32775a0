"""The dense Adam kernel's ends: the elements past the last group of 8 go with the same launch, and
untouched rows (gradient and moments 0) keep their parameters bit for bit where the formula does."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("grad", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [3, 4, 8, 4 * 512 * 8 - 1, 4 * 512 * 8 + 7])
def test_one_launch(n, grad):
    from torch.profiler import ProfilerActivity, profile

    from qsdvr_b200.optim import adam_step

    p, m, v = (torch.rand(n, device=DEV) for _ in range(3))
    g = torch.rand(n, device=DEV).to(grad)
    adam_step(p, g, m, v, 1, 1e-2, zero_grad=False)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        adam_step(p, g, m, v, 2, 1e-2, zero_grad=False)
        torch.cuda.synchronize()
    launched = [e.name for e in prof.events() if "adam" in e.name]
    assert len(launched) == 1, launched


@pytest.mark.parametrize("state", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("copy", [None, "plain", "cells"])
@pytest.mark.parametrize("lr,eps", [(1e-2, 1e-8), (1e-2, 0.0), (-1e-2, 1e-8), (0.0, 1e-8)])
def test_untouched_rows_match_groups_of_four(state, copy, lr, eps):
    """Against the kernel that serves 16-byte aligned buffers, which computes every element: the same
    values and signs of 0, NaN for NaN (0 / 0 with eps = 0), for rows of zeros, of negative zeros and
    of zeros but one element."""
    from qsdvr_b200.optim import adam_step

    rows, gen = 96, torch.Generator(device=DEV).manual_seed(3)
    p, g, m, v = (torch.randn((rows, 8), generator=gen, device=DEV) for _ in range(4))
    p[::3, :2] = torch.tensor([0.0, -0.0], device=DEV)
    p[8] = torch.inf
    g[::2], m[::2], v[::2] = 0.0, 0.0, 0.0
    g[2::8], m[4::16] = -0.0, -0.0
    g[6, 3], m[14, 5], v[22, 7] = 1e-3, 1e-3, 1e-3
    v = v.abs()
    outs = []
    for offset in (0, 4):  # 4 floats: not 32-byte aligned, the kernel of groups of 4
        t = [torch.empty(rows * 8 + 16, device=DEV, dtype=d)[k:k + rows * 8] for d, k in
             ((torch.float32, offset), (torch.float32, offset), (state, 8 if state is torch.bfloat16 else offset),
              (state, 8 if state is torch.bfloat16 else offset))]
        for buf, x in zip(t, (p, g, m, v)):
            buf.copy_(x.reshape(-1))
        c = torch.full((rows * 8,), 7.0, dtype=torch.bfloat16, device=DEV) if copy else None
        for step in (3, 4):
            adam_step(*t, step, lr, eps=eps, param_bf16=c, zero_grad=step == 4, sdf_cells=copy == "cells")
        outs.append(t + ([c] if copy else []))
    for a, b in zip(*outs):
        assert torch.equal(a.isnan(), b.isnan())
        assert torch.equal(a.nan_to_num(0.5), b.nan_to_num(0.5))
        assert torch.equal(a.signbit() & ~a.isnan(), b.signbit() & ~b.isnan())
