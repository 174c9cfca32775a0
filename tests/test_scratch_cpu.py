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


def test_render_calls_in_flight_have_their_own_workspace(monkeypatch):
    """Arguments that are still held (by another stream's call, or by a captured graph) keep a
    workspace that later calls of the same or of a larger need neither use nor replace."""
    from contextlib import nullcontext
    from types import SimpleNamespace

    from qsdvr_b200 import fused

    def need(ref):  # a separable render's workspace holds the copies of its table gradient as well
        a = ref._obj
        return 4096 + (64 * 16 * (3 * a.reso + 1) if a.sdf_layers else 0)

    monkeypatch.setattr(fused._lib, "lib", lambda: SimpleNamespace(qsdvr_render_workspace_size=need))
    monkeypatch.setattr(fused, "_check_batch", lambda rays, *_: (rays.device, rays.shape[0]))
    monkeypatch.setattr(fused, "on_device", lambda dev: nullcontext())
    rays, o = torch.zeros((10, 4), dtype=torch.int32), torch.zeros((10, 3))

    def args(R, separable):
        data = torch.zeros(((R + 1) ** 3, 32))
        if separable:
            return fused.make_args(rays, o, o, None, data, R, 0.01, 5.0, sdf_layers=torch.zeros((3 * R + 1, 4)))
        return fused.make_args(rays, o, o, torch.zeros((R ** 3, 8)), data, R, 0.01, 5.0)

    held = [args(*form) for form in ((4, False), (4, False), (4, True), (8, True), (8, False))]
    spans = [(a.workspace, a.workspace_bytes) for a in held]
    assert [s[1] for s in spans] == [4096, 4096, 4096 + 1024 * 13, 4096 + 1024 * 25, 4096]
    for i, a in enumerate(held):
        # still the memory of a live tensor, and nobody else's
        assert a.scratch.data_ptr() == a.workspace and a.scratch.numel() == a.workspace_bytes
        assert not any(_overlap(spans[i], s) for s in spans[:i])
