"""Block ILU sweeps whose waits run out, on the CPU (sweep_giveup_check.cpp:
the kernel's synchronisation in random order)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ is needed to compile the check")
def test_waits_that_run_out_leave_the_protocol_sound(tmp_path):
    exe = tmp_path / "sweep_giveup_check"
    csrc = ROOT / "optimisation2forme_b200" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-D_GLIBCXX_ASSERTIONS", f"-I{csrc}",
                    str(ROOT / "tests" / "sweep_giveup_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
