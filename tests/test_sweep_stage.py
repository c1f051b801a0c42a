"""Packing, staging and reading of the block ILU sweeps' operands, on the CPU
(sweep_stage_check.cpp), with the layout's constants taken from ilu.cuh."""
from __future__ import annotations

import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "optimisation2forme_b200" / "csrc"


def _constants() -> dict:
    text = (CSRC / "ilu.cuh").read_text() + (CSRC / "sweep_plan.hpp").read_text()
    env: dict = {}
    for name in ("kSweepChunks", "kSweepRec", "kSweepSlots", "kSweepBars", "kStageRing", "kSweepWindow", "kStageSlots",
                 "kStageChunkDoubles", "kStageChunksFwd", "kStageChunksBwd", "kStageBwdD", "kStageDoubles", "kStageOwn"):
        m = re.search(rf"constexpr\s+int\s+{name}\s*=\s*([^;]+);", text)
        assert m, name
        env[name] = int(eval(m.group(1), {}, env))
    return env


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ is needed to compile the check")
def test_every_read_finds_its_own_element(tmp_path):
    k = _constants()
    exe = tmp_path / "sweep_stage_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-D_GLIBCXX_ASSERTIONS", f"-DSTAGE_RING={k['kStageRing']}",
                    f"-DSTAGE_CHUNK={k['kStageChunkDoubles']}", f"-DSTAGE_BWD_D={k['kStageBwdD']}",
                    f"-DSTAGE_DOUBLES={k['kStageDoubles']}", f"-DSTAGE_OWN={k['kStageOwn']}", f"-I{CSRC}",
                    str(ROOT / "tests" / "sweep_stage_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
