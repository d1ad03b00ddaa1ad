"""The page-locked record staging of a device that is named without an index belongs to the device
that is current (host only)."""
import torch

from tomography_local_demo_b200 import recon as R


def test_each_current_device_has_its_own_ring(monkeypatch):
    monkeypatch.setattr(R, "_STAGING", {})
    monkeypatch.setattr(R, "_RecordStaging", object)
    rings = {}
    for current in (0, 1, 0, 1):
        monkeypatch.setattr(torch.cuda, "current_device", lambda: current)
        ring = R._staging(torch.device("cuda"))
        assert rings.setdefault(current, ring) is ring
        assert R._staging(torch.device("cuda", current)) is ring
        assert R._staging("cuda:%d" % current) is ring
    assert rings[0] is not rings[1]
