"""Scratch memory of the render entry points: calls that are in flight together (two streams, two
threads) must not share it.  Checked on the host, without launching: the addresses and sizes that a
launch gets, with a second call made while the first one has not returned."""
import torch


def _overlap(a, b):
    return a[0] < b[0] + b[1] and b[0] < a[0] + a[1]


def test_ray_order_calls_in_flight_have_their_own_scratch(monkeypatch):
    from qsdvr_b200 import fused

    rays = torch.zeros((100, 4), dtype=torch.int32)
    o = torch.zeros((100, 3))
    seen = []

    def launch(dev, name, *args):
        seen.append(args[-2:])  # (address, bytes)
        if len(seen) == 1:
            fused.ray_order(rays, o, o, 0.01)

    monkeypatch.setattr(fused, "_check_batch", lambda rays, *_: (rays.device, rays.shape[0]))
    monkeypatch.setattr(fused, "launch", launch)
    fused.ray_order(rays, o, o, 0.01)
    assert len(seen) == 2 and not _overlap(*seen)
