"""The dense Adam kernel (8 elements a thread, 32-byte accesses) against the kernel that serves
buffers with 16-byte alignment only: the same bits in every output, for each type of gradient, state
and copy, at the edges of groups of 4, of groups of 8 and of blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _at(t, offset):
    """A copy of t that starts `offset` bytes past a 512-byte boundary."""
    n = offset // t.element_size()
    buf = torch.empty(t.numel() + n, dtype=t.dtype, device=DEV)
    buf[n:].copy_(t)
    assert buf[n:].data_ptr() % 512 == offset
    return buf[n:]


@pytest.mark.parametrize("n", [1, 4, 7, 8, 12, 15, 4095, 4096, 4097, 8 * 512 * 3 + 13])
@pytest.mark.parametrize("grad,state,copy", [("f32", "f32", None), ("f32", "f32", "plain"), ("bf16", "f32", "plain"),
                                             ("f32", "bf16", "plain"), ("bf16", "bf16", None), ("f32", "f32", "cells"),
                                             ("f32", "bf16", "cells")])
def test_dense_matches_groups_of_four(n, grad, state, copy):
    from qsdvr_b200.optim import adam_step

    if copy == "cells":
        n = 8 * ((n + 7) // 8)
    types = {"f32": torch.float32, "bf16": torch.bfloat16}
    gen = torch.Generator(device=DEV).manual_seed(n)

    def rand(scale):
        return scale * torch.randn(n, generator=gen, device=DEV)

    p, g, m, v = rand(1.0), rand(0.1), rand(0.05), rand(0.05) ** 2
    g[::3] = 0.0
    outs = []
    for offset in (0, 16):  # 16: not 32-byte aligned, the kernel of groups of 4
        t = [_at(p, offset), _at(g.to(types[grad]), offset), _at(m.to(types[state]), offset),
             _at(v.to(types[state]), offset)]
        c = torch.zeros(n, dtype=torch.bfloat16, device=DEV) if copy else None
        for step in (3, 4):
            adam_step(*t, step, 1e-2, param_bf16=c, zero_grad=step == 4, sdf_cells=copy == "cells")
        outs.append(t + ([c] if copy else []))
    assert not outs[0][1].any() and not torch.equal(outs[0][0], p)
    for a, b in zip(*outs):
        assert torch.equal(a, b)
