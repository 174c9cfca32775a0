"""LayerToGridForward with host layers only queues its work: it returns while earlier work of the
stream is still running, and the grid is that of the layers at the time of the call."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("R", [1, 16, 128, 256])
def test_host_layers_do_not_wait(R):
    from qsdvr_b200 import qsdvr

    gen = torch.Generator().manual_seed(R)
    layers = [torch.randn(n, generator=gen) for n in (R, R, R, 4)]
    want = torch.empty((R, R, R, 7), device=DEV)
    qsdvr.LayerToGridForward(want, *layers)
    out = torch.empty_like(want)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    torch.cuda._sleep(200_000_000)  # about 0.1 s
    done.record()
    qsdvr.LayerToGridForward(out, *layers)
    waited = done.query()
    for t in layers:
        t.zero_()  # the copy has left the host tensors
    torch.cuda.synchronize()
    assert not waited
    assert torch.equal(out, want)
