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
