"""bench.py's line: a few kilobytes with every key a reader of the record needs,
whatever the legs carry; their details are apart."""
import json

import bench


def _line():
    leg = {"value": 1.5, "unit": "iterations/s", "rows": [{"a": 1.0 / 3.0, "b": "x" * 40}] * 200}
    line = {k: 1.0 / 3.0 for k in bench.LINE_KEYS}
    line["config"] = {"model": "m" * 200, "note": "n" * 600}
    line["cpu_baseline"] = {"sample": "s" * 400, "parity": {k: 1.0 / 3.0 for k in "abcdefgh"}, "note": "n" * 400}
    line["roofline"] = {"kernel": "k" * 300, "peak_source": "p" * 100, "hbm": {k: 1.0 / 3.0 for k in "abcdef"}}
    for k in ("mixed", "trust_region", "refine", "matched_cost", "variable_intrinsics", "batched", "serving"):
        line[k] = dict(leg)
    return line


def test_the_record_is_short_and_has_what_it_must():
    line = _line()
    record, details = bench.split_line(line)
    assert len(json.dumps(record)) < bench.LINE_BYTES
    assert set(bench.LINE_KEYS) <= set(record)
    assert record["legs"] == {"mixed": 1.5, "trust_region": 1.5, "refine": 1.5}
    assert set(record) - {"legs"} | set(details) == set(line)


def test_a_leg_that_did_not_run_has_no_number():
    line = _line()
    line["mixed"] = None
    assert "mixed" not in bench.split_line(line)[0]["legs"]
