"""A value held back (test hook) lets the waits of the block ILU sweeps run
out: the solve returns O2F_ERR_CUDA, and after the hook is cleared the same
context solves to the same lambda as before."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import desc_of, small_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_surface,n_layers,triangles", [
    (12, 3, True), (90, 61, False),  # one block
    (200, 50, True),                 # two
    (270, 136, True),                # four
    (420, 260, True),                # eight
])
def test_a_held_back_value_is_an_error_and_the_next_solve_is_not(n_surface, n_layers, triangles):
    from optimisation2forme_b200 import O2FError, SimulationParams, Solver
    p = SimulationParams(viscosity=1.8e-5, inflow_velocity=0.6, aoa_deg=2.0, cfl_number=0.5, final_time=10.0,
                         limiter_k=5.0, verbosity=0, adjoint_sweeps="block")
    solve = dict(beta=0.1, tol=1e-10, max_iter=12, restart=12)
    with Solver(p, desc=desc_of(small_mesh(triangles=triangles, n_surface=n_surface, n_layers=n_layers, seed=3))) as s:
        s.initialize_freestream()
        s.time_loop(20)
        s.compute_residual()
        ref = s.solve_adjoint_system(**solve, raise_on_failure=False)
        for _ in range(2):
            s.debug_ilu_stall(True, spin_limit=500, selected=True)
            with pytest.raises(O2FError) as e:
                s.solve_adjoint_system(**solve)
            assert e.value.status == "O2F_ERR_CUDA" and "dependency wait" in str(e.value)
            s.debug_ilu_stall(False)
            again = s.solve_adjoint_system(**solve, raise_on_failure=False)
            assert again["iters"] == ref["iters"]
            assert np.array_equal(again["lambda"].view(np.int64), ref["lambda"].view(np.int64))
