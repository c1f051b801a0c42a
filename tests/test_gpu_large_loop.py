"""The time loop of meshes beyond the tile kernels (separate kernels with the
wave speed, norm and step control folded into the stages) against the batched
loop: state, time, steps, history, and the loop's stops."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal, desc_of, perturbed_freestream, small_mesh

pytestmark = pytest.mark.gpu


def _same(a, b):
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(np.where(nan, 0.0, a).view(np.int64), np.where(nan, 0.0, b).view(np.int64))


@pytest.mark.parametrize("n_surface,n_layers,triangles", [(360, 262, True), (440, 425, False)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_large_loop_equals_the_batched_loop(n_surface, n_layers, triangles, precision):
    from optimisation2forme_b200 import Batch, SimulationParams, Solver
    m = small_mesh(triangles=triangles, n_surface=n_surface, n_layers=n_layers, seed=5)
    p = SimulationParams(viscosity=1.8e-5, inflow_velocity=0.6, aoa_deg=1.5, cfl_number=0.3, final_time=1e30,
                         limiter_k=5.0, verbosity=0, precision=precision)
    with Solver(p, desc=desc_of(m)) as a, Solver(p, desc=desc_of(m)) as b, Batch([b]) as batch:
        assert 180000 <= a.n_cells < 200000
        U = perturbed_freestream(a.n_cells, p, seed=1)

        def both(steps, drop=0.0):
            ra = a.time_loop(steps, residual_drop=drop, raise_on_failure=False)
            rb = batch.time_loop(steps, residual_drop=drop)[0]
            assert ra["steps"] == rb["steps"] and ra["t"] == rb["t"] and ra["status"] == rb["status"]
            assert _same(a.get_state(), b.get_state())
            n = ra["steps"]
            h = batch.history(0, n) if n else np.zeros(0)
            # the same squares in another order: 2 n eps, n terms a partial sum
            assert np.all(np.abs(ra["history"] - h) <= 1e-12 * np.abs(h))
            return ra

        for s in (a, b):
            s.set_state(U)
        full = both(7)
        assert full["steps"] == 7 and full["t"] > 0.0 and full["status"] == "OK"
        assert np.all(full["history"] > 0.0)
        if precision == "fp64":
            for name in ("edge_LR", "edge_tau", "edge_F", "vertex_U", "R"):
                assert bits_equal(a.debug(name), b.debug(name)), name
        # a residual drop that the loop meets on the way
        for s in (a, b):
            s.set_state(U)
        k = int(np.argmin(full["history"]))
        assert k > 0
        stopped = both(7, drop=float(full["history"][k] / full["history"][0]) * (1.0 + 1e-9))
        assert 0 < stopped["steps"] <= 7
        # a state that is not finite
        q = U.copy()
        q[4 * 1000 + 3] = np.nan
        for s in (a, b):
            s.set_state(q)
        assert both(7)["status"] == "O2F_ERR_NONFINITE"
        for s in (a, b):
            s.set_state(U)
        assert both(3)["steps"] == 3
