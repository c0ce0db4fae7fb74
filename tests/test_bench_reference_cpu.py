"""bench.py --impl reference without gsbn's kernels: one line that says so, and
none of this repository's code timed in their place."""
import json
import sys

import bench
from oracle import sim


def test_without_the_reference(monkeypatch, capsys):
    monkeypatch.setattr(sim, "ref_available", lambda: False)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--gpus", "1", "--steps", "20", "--warmup", "5"])
    for key in ("RANK", "WORLD_SIZE", "LOCAL_RANK"):
        monkeypatch.delenv(key, raising=False)
    bench.main()
    lines = capsys.readouterr().out.strip().splitlines()
    assert len(lines) == 1
    out = json.loads(lines[0])
    assert set(out) == {"impl", "unavailable"} and out["impl"] == "reference"
    assert "\n" not in out["unavailable"] and out["unavailable"]
