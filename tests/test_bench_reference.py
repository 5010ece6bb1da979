"""bench.py where the reference could not be built (its sources are not part of the repository)."""
import json
import sys

import bench
import oracle


def lines(monkeypatch, capsys, *args):
    monkeypatch.setattr(oracle, "ref_available", lambda: False)
    monkeypatch.setattr(oracle, "REF_PATH", "/nonexistent/libumappp_ref.so")
    monkeypatch.setattr(oracle, "_ref", None)
    monkeypatch.setattr(sys, "argv", ["bench.py", *args])
    for name in ("RANK", "WORLD_SIZE"):
        monkeypatch.delenv(name, raising=False)
    bench.main()
    return [json.loads(x) for x in capsys.readouterr().out.splitlines()]


def test_reference_arm_says_so(monkeypatch, capsys):
    out = lines(monkeypatch, capsys, "--impl", "reference", "--steps", "1")
    assert len(out) == 1 and out[0]["impl"] == "reference" and "not built" in out[0]["unavailable"]


def test_line_is_printed_without_the_reference(monkeypatch, capsys):
    monkeypatch.setattr(bench, "run_ours", lambda args, rank, world: {"metric": "m", "value": 1.5})
    out = lines(monkeypatch, capsys, "--no-batch", "--no-precision")
    assert len(out) == 1 and out[0]["value"] == 1.5 and "not built" in out[0]["cpu_baseline"]["unavailable"]
