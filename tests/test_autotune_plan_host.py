"""The autotuner's timing of the ordered-pair kernel with the kernel faked (no device): it evaluates fewer
targets than vortices, since an evaluation of all of them runs the once-per-unordered-pair form where that
is planned, whatever the entry says."""
import pytest

from pointvortex_b200 import autotune


@pytest.mark.parametrize("geometry,name", [("infinite", "InfinitePlaneKernel"),
                                           ("periodic", "PeriodicBoxKernel"), ("disk", "DiskKernel")])
def test_times_a_range(monkeypatch, geometry, name):
    from pointvortex_b200 import kernel
    n, calls = 128, []

    class Fake:
        def __init__(self, *args, **kw):
            pass

        def uploadDeviceState(self, system):
            pass

        def evaluateDeviceState(self):
            calls.append(("all", autotune_entry()))

        def evaluateRange(self, x, y, g, core, begin, end):
            calls.append((x.size, begin, end, autotune_entry()))

        def setProfiling(self, on):
            pass

        def resetKernelStats(self):
            pass

        def kernelStats(self):
            return {"velocity": (2, 2, 6.0)}

        def close(self):
            pass

    def autotune_entry():
        return autotune.get_entry(autotune.GEOMETRIES[geometry], 0, 7)

    monkeypatch.setattr(kernel, name, Fake)
    saved = autotune_entry()
    try:
        assert autotune._time_plan(geometry, 0, n, 4, 2) == 3.0
    finally:
        autotune.set_entry(autotune.GEOMETRIES[geometry], 0, 7, saved)
    assert calls == [(n, 0, n - 1, 4)] * 3
