"""The block ILU sweeps (a cluster of thread blocks walking a schedule)
against the waiting sweeps (rows in plain level order, no schedule): the
arithmetic of a row is the same, so some iterations of the adjoint solve give
the same lambda bit for bit -- at each cluster size, on triangles and
quadrilaterals, with few and with ragged rows."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from conftest import desc_of, small_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_surface,n_layers,triangles", [
    (12, 3, True), (13, 5, False),       # less than a chunk per level
    (96, 25, True), (90, 61, False),     # one block
    (200, 50, True),                     # two
    (270, 136, True), (290, 201, False),  # four
    (420, 260, True),                    # eight
])
def test_block_sweeps_equal_waiting_sweeps(n_surface, n_layers, triangles):
    from optimisation2forme_b200 import SimulationParams, Solver
    p = SimulationParams(viscosity=1.8e-5, inflow_velocity=0.6, aoa_deg=2.0, cfl_number=0.5, final_time=10.0,
                         limiter_k=5.0, verbosity=0, adjoint_sweeps="block")
    with Solver(p, desc=desc_of(small_mesh(triangles=triangles, n_surface=n_surface, n_layers=n_layers, seed=3))) as s:
        s.initialize_freestream()
        s.time_loop(20)
        s.compute_residual()
        got = []
        for mode in ("block", "waiting", "block"):
            s.set_params(dataclasses.replace(p, adjoint_sweeps=mode))
            s.compute_residual()
            got.append(s.solve_adjoint_system(beta=0.1, tol=1e-10, max_iter=12, restart=12, raise_on_failure=False))
        assert np.all(np.isfinite(got[0]["lambda"])) and np.any(got[0]["lambda"] != 0.0)
        for other in got[1:]:
            assert other["iters"] == got[0]["iters"]
            assert np.array_equal(other["lambda"].view(np.int64), got[0]["lambda"].view(np.int64))
