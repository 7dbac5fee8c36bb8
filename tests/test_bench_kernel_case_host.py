"""bench.py's velocity evaluations with the kernel faked (no device): the ordered arm asks for fewer targets
than vortices, which is what always takes the ordered-pair kernel, and counts those targets' pairs."""
import numpy as np
import pytest


@pytest.mark.parametrize("ordered", [False, True])
def test_ordered_arm_is_a_range(monkeypatch, ordered):
    import bench
    import pointvortex_b200 as pv
    import torch
    n, calls = 64, []

    class Fake:
        def __init__(self, *args, **kw):
            pass

        def uploadDeviceState(self, system):
            pass

        def statePlan(self):
            return {"symmetric": 1}

        def evaluate(self, x, y, g):
            calls.append(("host", 0, x.size))

        def evaluateRange(self, x, y, g, core, begin, end):
            calls.append(("host", begin, end))

        def evaluateDeviceState(self):
            calls.append(("state", 0, n))

        def setProfiling(self, on):
            pass

        def resetKernelStats(self):
            pass

        def kernelStats(self):
            return {"velocity": (3, 3, 3.0), "near": (0, 0, 0.0)}

    monkeypatch.setattr(pv, "PeriodicBoxKernel", Fake)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    r = bench.run_kernel_case(f"periodic:{n}", 3, ordered=ordered)
    assert len(calls) == 5 and len(set(calls)) == 1
    targets = n - 1 if ordered else n
    assert calls[0] == (("host" if ordered else "state"), 0, targets)
    assert r["kernel"] == ("ordered" if ordered else "symmetric")
    assert np.isclose(r["pairs_per_s"], targets * (n - 1) / 1e-3)
