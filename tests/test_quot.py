"""The branch-free quotients and square roots of the FP64 kernels
(csrc/qdiv.h) against IEEE arithmetic, on the CPU (tests/quot_check.cpp)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ is needed to compile the check")
def test_quotients_and_roots_are_correctly_rounded(tmp_path):
    exe = tmp_path / "quot_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'optimisation2forme_b200' / 'csrc'}",
                    str(ROOT / "tests" / "quot_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
