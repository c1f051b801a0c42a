"""Plan of the block ILU sweeps on the CPU (tests/sweep_plan_check.cpp): every
value is where the kernel reads it, for all cluster sizes and ragged graphs."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ is needed to compile the check")
def test_every_value_is_in_its_slot(tmp_path):
    exe = tmp_path / "sweep_plan_check"
    csrc = ROOT / "optimisation2forme_b200" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-D_GLIBCXX_ASSERTIONS", f"-I{csrc}",
                    str(ROOT / "tests" / "sweep_plan_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
