"""The sizes that the tuner of the once-per-unordered-pair form times (steps faked, no device): one of each
bucket, and none that the ordered choice would serve by whole steps in one launch."""
import re
import os

from conftest import ROOT
from pointvortex_b200 import autotune


def test_sizes_are_beyond_the_small_steps(monkeypatch):
    header = open(os.path.join(ROOT, "pointvortex_b200", "csrc", "pv_internal.h")).read()
    limit = int(re.search(r"kSmallStepsMaxN = (\d+);", header).group(1))
    assert autotune.SMALL_STEPS_MAX_N == limit
    timed = []
    monkeypatch.setattr(autotune, "_time_steps", lambda g, p, n, s: timed.append(n) or 1.0)
    monkeypatch.setattr(autotune, "_grid_ctas", lambda g, p, n: timed.append(n) or 4)
    keys = [(g, p, b) for g in (0, 1) for p in (0, 1) for b in range(11, 14)]
    saved = {k: (autotune.get_symmetric_entry(*k), autotune.get_symmetric_grid(*k)) for k in keys}
    try:
        entries = autotune.tune_symmetric(range(11, 14), evals=3)
    finally:
        for k, (entry, grid) in saved.items():
            autotune.set_symmetric_entry(*k, *entry)
            autotune.set_symmetric_grid(*k, grid)
    assert min(timed) > limit and {n.bit_length() - 1 for n in timed} == {11, 12, 13}
    assert {(e["log2_n"], e["n"]) for e in entries} == {(11, 3072), (12, 4096), (13, 8192)}
