"""The block sweeps' plan and buffers are made for solves that use them: not
for a context that sweeps the other way, and at the first solve after a
change."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from conftest import desc_of, small_mesh

pytestmark = pytest.mark.gpu


def test_waiting_sweeps_make_no_plan():
    import ctypes

    from optimisation2forme_b200 import SimulationParams, Solver, _lib

    def device_bytes(s):
        info = _lib.MeshInfo()
        _lib.check(_lib.lib().o2f_get_info(s._h, ctypes.byref(info)))
        return info.device_bytes

    p = SimulationParams(viscosity=1.8e-5, inflow_velocity=0.6, aoa_deg=2.0, cfl_number=0.5, final_time=10.0,
                         limiter_k=5.0, verbosity=0, adjoint_sweeps="waiting")
    with Solver(p, desc=desc_of(small_mesh(triangles=True, n_surface=96, n_layers=25, seed=3))) as s:
        s.initialize_freestream()
        s.time_loop(20)
        got, held = [], []
        for mode in ("waiting", "auto", "waiting", "block"):
            s.set_params(dataclasses.replace(p, adjoint_sweeps=mode))
            s.compute_residual()
            got.append(s.solve_adjoint_system(beta=0.1, tol=1e-10, max_iter=12, restart=12, raise_on_failure=False))
            held.append(device_bytes(s))
        # at least the factor blocks in sweep order, 2 x 512 B and 128 B a row
        assert held[1] - held[0] >= 1152 * s.n_cells
        assert held[3] == held[2] == held[1]
        for other in got[1:]:
            assert other["iters"] == got[0]["iters"]
            assert np.array_equal(other["lambda"].view(np.int64), got[0]["lambda"].view(np.int64))
