"""What camera.gather_rays refuses: its kernel reads int64 indices, int32 [P,4] records and float32
[P,3] tables of one device."""
import pytest
import torch

DEV = "cuda"


def _tables(P, device):
    return (torch.arange(4 * P, dtype=torch.int32, device=device).reshape(P, 4),
            torch.rand((P, 3), device=device), torch.rand((P, 3), device=device))


def test_refuses_other_types_and_host_tensors():
    from qsdvr_b200.camera import gather_rays

    rays, o, d = _tables(6, "cpu")
    pix = torch.tensor([4, 0, 5])
    with pytest.raises(TypeError, match="rays|rayList"):
        gather_rays(pix, rays.long(), o, d)
    with pytest.raises(ValueError, match="expected a CUDA tensor"):
        gather_rays(pix, rays, o, d)


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["int32", "host", "strided", "pixels2d", "rays3", "strided rays", "origin", "dir64",
                                  "host dir"])
def test_refuses_on_the_device(case):
    from qsdvr_b200.camera import gather_rays

    rays, o, d = _tables(6, DEV)
    pix = torch.tensor([4, 0, 5], device=DEV)
    bad = {"int32": (pix.int(), rays, o, d), "host": (pix.cpu(), rays, o, d),
           "strided": (torch.arange(6, device=DEV)[::2], rays, o, d), "pixels2d": (pix.reshape(3, 1), rays, o, d),
           "rays3": (pix, rays[:, :3].contiguous(), o, d), "strided rays": (pix, rays.t().contiguous().t(), o, d),
           "origin": (pix, rays, o[:4], d), "dir64": (pix, rays, o, d.double()), "host dir": (pix, rays, o, d.cpu())}
    with pytest.raises((TypeError, ValueError)):
        gather_rays(*bad[case])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [0, 1, 255, 256, 257])
def test_matches_indexing(n):
    from qsdvr_b200.camera import gather_rays

    tables = _tables(300, DEV)
    pix = torch.randperm(300, generator=torch.Generator().manual_seed(n))[:n].to(DEV)
    for got, t in zip(gather_rays(pix, *tables), tables):
        assert torch.equal(got, t[pix])
