"""A disk population on the device that there is no memory for the once-per-unordered-pair rows of (256 MB at
N = 65 536): it is taken all the same and evaluated by the ordered kernel, whose partial rows need less
than a quarter of that."""
import pytest
import torch

from conftest import normalized_error
from pointvortex_b200 import ics
from pointvortex_b200.kernel import DiskKernel, VortexSystem

pytestmark = pytest.mark.gpu


def test_upload_when_memory_is_short():
    n = 65536
    x, y, g = ics.disk(n, 1, 1.0, 0.9)
    k = DiskKernel(1.0)
    k.uploadDeviceState(VortexSystem(x, y, g))
    assert k.statePlan()["symmetric"]
    want = k.evaluateDeviceState()
    k.close()
    k = DiskKernel(1.0)
    k.uploadDeviceState(VortexSystem(*ics.disk(64, 1, 1.0, 0.9)))
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(free - (160 << 20), dtype=torch.uint8, device="cuda")
    try:
        k.uploadDeviceState(VortexSystem(x, y, g))
        plan = k.statePlan()
        f = k.evaluateDeviceState()
    finally:
        del held
        torch.cuda.empty_cache()
    assert not plan["symmetric"] and plan["rows"] * n * 16 < 64 << 20, plan
    assert normalized_error(f.x, f.y, want.x, want.y).max() <= 1e-12
    k.uploadDeviceState(VortexSystem(x, y, g))  # with the memory there again
    assert k.statePlan()["symmetric"]
