"""The block sweeps wait on barriers that count stores from other thread
blocks of the cluster: every such wait acquires at cluster scope (the default
of the instruction is the block's own)."""
from __future__ import annotations

import re
from pathlib import Path

ILU = Path(__file__).resolve().parents[1] / "optimisation2forme_b200" / "csrc" / "ilu.cuh"


def test_waits_acquire_at_cluster_scope():
    waits = re.findall(r"mbarrier\.(?:try|test)_wait[\w.:]*", ILU.read_text())
    assert waits
    for w in waits:
        assert ".acquire.cluster." in w, w
