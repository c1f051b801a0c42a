"""bench.py's reference arm: a build that is not there is reported as such, a
file lost on the way is an error."""
from __future__ import annotations

import json
import sys

import pytest

ARGS = ["bench.py", "--impl", "reference", "--candidates", "1", "--cells-lo", "4000", "--cells-hi", "5000",
        "--steps", "1", "--warmup", "0"]


def test_missing_build_is_reported(monkeypatch, capsys, tmp_path):
    import bench
    from oracle import ref
    monkeypatch.setattr(sys, "argv", ARGS)
    monkeypatch.setattr(ref, "EXE_FAST", tmp_path / "none")
    assert bench.main() == 0
    line = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "not present" in line["unavailable"]


def test_a_lost_file_is_an_error(monkeypatch):
    import bench
    from oracle import ref

    def lost(*a, **k):
        raise FileNotFoundError("mesh.bin")

    monkeypatch.setattr(sys, "argv", ARGS)
    monkeypatch.setattr(ref, "EXE_FAST", type(ref.EXE_FAST)(__file__))
    monkeypatch.setattr(ref, "write_binary_mesh", lost)
    with pytest.raises(FileNotFoundError):
        bench.main()
