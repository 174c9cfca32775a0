"""RayCut's bisected in-box runs against the C oracle's sample-by-sample march, bit for bit, where a
run can end in an unusual way: rays along an axis (a direction component of exactly 0), a camera
inside the volume, a far plane inside it or in front of it, steps of 1 and of several hundred
thousand samples; and the rays a Camera keeps against plain indexing."""
import numpy as np
import pytest
import torch

import oracle.oracle as O
from conftest import oracle_camera

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _along_axis(axis, sign, size, near, far, distance):
    """A camera on an axis, looking along it (its centre pixel's ray has two zero components)."""
    from qsdvr_b200.qsdvr import CameraArgs

    f = np.zeros(3)
    f[axis] = sign
    right = np.roll(np.abs(f), 1)
    a = CameraArgs()
    a.width = a.height = size
    a.rotation = np.stack([right, np.cross(f, right), f], 1).reshape(-1)
    a.translation = -distance * f
    a.fx = a.fy = 1.3 * size
    a.cx = a.cy = -size / 2.0
    a.near, a.far = near, far
    a.pixelCount = size * size
    return a


CASES = [(axis, sign, 33, 2.0, 6.0, 4.0, 4 / 256) for axis in (0, 1, 2) for sign in (-1, 1)] + [
    (0, 1, 33, 0.01, 3.0, 0.2, 1 / 64),   # camera inside the volume
    (2, -1, 33, 2.0, 4.1, 4.0, 1 / 64),   # the far plane inside it
    (1, 1, 33, 2.0, 2.9, 4.0, 1 / 64),    # the far plane in front of it
    (2, 1, 33, 0.5, 4.0, 4.0, 3.0),       # one march step
    (0, -1, 5, 2.0, 6.0, 4.0, 1.1e-5),    # 360 thousand
]


@pytest.mark.parametrize("axis,sign,size,near,far,distance,interval", CASES)
def test_bisected_run_matches_the_march(axis, sign, size, near, far, distance, interval):
    from qsdvr_b200 import qsdvr as qs
    from qsdvr_b200.camera import Camera

    args = _along_axis(axis, sign, size, near, far, distance)
    P = size * size
    mask = np.random.default_rng(axis + size).random(P) < 0.8
    rays = torch.zeros((P, 4), dtype=torch.int32, device=DEV)
    origin, direction = torch.zeros((P, 3), device=DEV), torch.zeros((P, 3), device=DEV)
    qs.RayCut(args, torch.from_numpy(mask), rays, origin, direction, interval)
    want, wo, wd, S, M = O.ray_cut(oracle_camera(args), mask, interval)
    np.testing.assert_array_equal(direction.cpu().numpy(), wd)
    np.testing.assert_array_equal(rays.cpu().numpy().view(np.uint32), want)
    np.testing.assert_array_equal(origin.cpu().numpy(), wo)
    assert (args.sdfCount, args.renderCount) == (S, M)

    for order in ("pixels", "tiles"):
        cam = Camera(args, interval, 64, device=DEV)
        cam.GenerateRayPoints(torch.from_numpy(mask), order=order)
        pix = cam.pixel_index
        assert torch.equal(pix.sort().values, torch.from_numpy(np.flatnonzero(mask)).to(DEV))
        assert torch.equal(cam.rayList, rays[pix]) and torch.equal(cam.originList, origin[pix])
        assert torch.equal(cam.dirList, direction[pix])


def test_gather_rays_flags_a_pixel_outside():
    from qsdvr_b200 import _lib
    from qsdvr_b200.camera import gather_rays

    _lib.device_error()
    rays = torch.ones((4, 4), dtype=torch.int32, device=DEV)
    o, d = torch.ones((4, 3), device=DEV), torch.ones((4, 3), device=DEV)
    got = gather_rays(torch.tensor([3, 4, -1], device=DEV), rays, o, d)
    assert [t[0].sum().item() for t in got] == [4, 3, 3] and not any(t[1:].any() for t in got)
    assert _lib.device_error() & _lib.DEVERR_INDEX
    assert all(t.shape[0] == 0 for t in gather_rays(torch.empty(0, dtype=torch.int64, device=DEV), rays, o, d))
