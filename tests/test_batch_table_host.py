"""The batch table and its tuner on the host (timings faked, no device): an entry reads back as what it is,
so that a table can be put back, and the tuner times the built-in rule beside the ordered items and
leaves a size without an entry where the rule is faster. The tests share the table, and each finds it as
it was before the one that ran first."""
import json

import pytest

from pointvortex_b200 import autotune


@pytest.mark.parametrize("key", [(0, 0, 10), (1, 0, 9), (2, 0, 12), (1, 1, 12)])
def test_an_entry_reads_back_as_itself(key):
    autotune.set_batch_entry(*key, 0)
    assert autotune.stored_batch_entry(*key) == 0
    autotune.set_batch_entry(*key, 2)
    assert autotune.stored_batch_entry(*key) == autotune.get_batch_entry(*key) == 2
    autotune.set_batch_entry(*key, autotune.stored_batch_entry(*key))
    assert autotune.stored_batch_entry(*key) == 2
    autotune.set_batch_entry(*key, 0)
    assert autotune.stored_batch_entry(*key) == 0


def test_what_a_test_restores_from_the_effective_value_is_undone():
    for key in [(0, 0, 10), (2, 0, 12)]:
        autotune.set_batch_entry(*key, autotune.get_batch_entry(*key))
        assert autotune.stored_batch_entry(*key) != 0


def test_and_the_next_test_finds_the_table_without_entries():
    for key in [(0, 0, 10), (2, 0, 12)]:
        assert autotune.stored_batch_entry(*key) == 0


@pytest.mark.parametrize("rule_ms", [0.5, 1.5])
def test_the_tuner_times_the_built_in_rule(monkeypatch, tmp_path, rule_ms):
    """Ordered items take 1 ms or more, the rule rule_ms for FP64 and 2 ms for FP32C."""
    timed = []

    def fake(geometry, precision, n, attempts):
        entry = autotune.stored_batch_entry(autotune.GEOMETRIES[geometry],
                                            autotune.PRECISIONS[precision], n.bit_length() - 1)
        timed.append((geometry, precision, entry))
        if entry == 0:
            return rule_ms if precision == "fp64" else 2.0
        return 1.0 if entry == 2 else 3.0

    monkeypatch.setattr(autotune, "_time_batch", fake)
    entries = autotune.tune_batch(range(9, 11), attempts=2)
    assert {(g, p, 0) for g in autotune.GEOMETRIES for p in autotune.PRECISIONS} <= set(timed)
    for e in entries:
        want = 0 if e["precision"] == "fp64" and rule_ms < 1.0 else 2
        key = (autotune.GEOMETRIES[e["geometry"]], autotune.PRECISIONS[e["precision"]], e["log2_n"])
        assert e["per_thread"] == autotune.stored_batch_entry(*key) == want, e
    path = tmp_path / "table.json"  # and a file of them loads as it was written
    path.write_text(json.dumps({"batch": entries}))
    for e in entries:
        autotune.set_batch_entry(autotune.GEOMETRIES[e["geometry"]],
                                 autotune.PRECISIONS[e["precision"]], e["log2_n"], 1)
    assert autotune.load(str(path)) == len(entries)
    for e in entries:
        key = (autotune.GEOMETRIES[e["geometry"]], autotune.PRECISIONS[e["precision"]], e["log2_n"])
        assert autotune.stored_batch_entry(*key) == e["per_thread"]
