"""What bench.py prints: one JSON line, the last and short enough to be read from
the end of a log, whatever the number of configurations; everything else on lines
of its own before it."""
import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
import bench  # noqa: E402


def result():
    check = {"ok": True, "max_err_over_bound": 0.5, "against": "a" * 150}
    batch = {k: 1.25 for k in bench.BATCH_KEYS} | {"chosen": {"note": "n" * 900}, "check": check}
    return {"metric": bench.METRIC, "value": 1634.5, "unit": "GB/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "config": {"workload": "w" * 300}, "roofline": {"note": "r" * 430}, "e2e": {"value": 5.0, "p": "e" * 680},
            "cpu_baseline": {"sample": "c" * 190}, "check": check, "batched": batch, "batched_i32": batch,
            "configs": [{"config": i, "us": 1.0, "check": "x" * 400} for i in range(61)], "configs_checked": "61/61"}


def test_one_short_json_line_at_the_end():
    res = result()
    lines = bench.output_lines(res)
    assert [i for i, l in enumerate(lines) if l.startswith("{")] == [len(lines) - 1]
    assert len(lines[-1]) < 4000 and all("\n" not in l for l in lines)
    last = json.loads(lines[-1])
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "config", "roofline", "e2e", "cpu_baseline",
              "check", "configs_checked"):
        assert last[k] == res[k]
    assert last["batched"]["queue_learned_ms"] == 1.25 and last["batched"]["check_ok"] is True


def test_nothing_is_lost_before_it():
    res = result()
    lines = bench.output_lines(res)
    assert [json.loads(l[7:]) for l in lines if l.startswith("config ")] == res["configs"]
    for k in ("batched", "batched_i32"):
        assert [json.loads(l.split(" ", 1)[1]) for l in lines if l.startswith(k + " ")] == [res[k]]


def test_a_result_without_them_is_one_line():
    assert bench.output_lines({"impl": "reference", "unavailable": "why"}) == [
        '{"impl": "reference", "unavailable": "why"}']
