"""CPU test of bench.py's JSON line: one line that its readers can take whole, however long the legs' results are."""
import json

import bench

LINE = {"metric": "m", "value": 1.0, "unit": "Mrays/s", "n_gpus": 1, "steps": 20, "warmup": 5, "ms_per_step": 2.0,
        "config": {"model": "x"}, "e2e": {"value": 1.0, "h2d_bytes_per_step": 1}, "gpu_launches": 40,
        "autotune": {"best": "b", "fastest_ms": [["a", 1.0]] * 10}}


def _legs(runs):
    run = {"rel_mse": 0.123456789, "ms": {"min": 1.0, "runs": [1.0, 2.0, 3.0]}, "deep": {"a": {"b": {"c": 1.0}}}}
    return {"city_frame": {"ms": 6.6, "rays": 1}, "residency": {"best": "0.150/1", "sweep": {str(i): run for i in range(runs)},
                                                              "frames": [[1.0] * 20] * runs}}


def test_short_legs_stay_whole():
    assert json.loads(bench.fit_line(LINE, _legs(3))) == {**LINE, **json.loads(json.dumps(_legs(3)))}


def test_long_legs_are_cut():
    for runs in (100, 300, 5000):
        text = bench.fit_line(LINE, _legs(runs))
        assert len(text) <= bench.LINE_LIMIT and "\n" not in text
        got = json.loads(text)
        assert {k: got[k] for k in LINE} == LINE
        assert set(got) == set(LINE) | {"city_frame", "residency"}
        assert got["city_frame"]["ms"] == 6.6


def test_long_autotune_is_cut_last():
    line = dict(LINE, autotune={"best": "b", "configs": 402, "legacy_ms": {str(i): 1.0 for i in range(3000)}})
    got = json.loads(bench.fit_line(line, _legs(3)))
    assert got["autotune"] == {"best": "b", "configs": 402, "legacy_ms": {}} and got["value"] == 1.0
