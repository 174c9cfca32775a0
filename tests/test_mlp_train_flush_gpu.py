"""The proposal network's gradient flush: vector REDs into an aligned gradient buffer and scalar
ones into a buffer that is only 4-byte aligned, at one point, one point past a tile and several
tiles per CTA, against the float64 oracle (2e-3 norm-wise: the kernel and the oracle round the same
values to bf16, as in tests/test_proposal_gpu.py)."""
import ctypes

import numpy as np
import pytest
import torch

import oracle.proposal as OP
from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 129, 80000])
def test_flush_alignment(n, offset):
    from qsdvr_b200 import proposal
    from qsdvr_b200._lib import call

    w = proposal.init_params(3, "cpu")
    w[6144:6208] = 0.05
    w[6272] = 0.3
    r = np.random.default_rng(n)
    pts = np.concatenate([r.uniform(-1, 1, (n, 3)), r.exponential(2.0, (n, 1))], 1).astype(np.float32)
    p, params = torch.from_numpy(pts).to(DEV), w.to(DEV).to(torch.bfloat16)
    buf = torch.zeros(proposal.N_PARAMS + 4, device=DEV)
    grad, loss = buf[offset:offset + proposal.N_PARAMS], torch.zeros(1, device=DEV)
    assert grad.data_ptr() % 16 == 4 * offset
    call("qsdvr_mlp_train", ctypes.c_void_p(p.data_ptr()), n, ctypes.c_void_p(params.data_ptr()), 4.0,
         ctypes.c_void_p(grad.data_ptr()), ctypes.c_void_p(loss.data_ptr()),
         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    want, want_loss = OP.train_gradients(w.numpy(), pts, 4.0)
    got = grad.cpu().numpy().astype(np.float64)
    assert abs(loss.item() - want_loss) <= 1e-4 * max(1.0, want_loss)
    for lo, hi in ((0, 2048), (2048, 6144), (6144, 6208), (6208, 6272), (6272, 6273)):
        assert rel_err(got[lo:hi], want[lo:hi]) < 2e-3, (lo, hi)
    assert not buf[:offset].any() and not buf[offset + 6273:].any()
