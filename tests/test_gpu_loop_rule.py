"""Which kernels the time loop runs on (tiles: 6 launches a step, separate
kernels: 17) by size and precision, and that both give the batched loop's
bits; on meshes beyond the tiles, the loop's step control too."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal, desc_of, perturbed_freestream, small_mesh

pytestmark = pytest.mark.gpu


def _params(**kw):
    from optimisation2forme_b200 import SimulationParams
    return SimulationParams(viscosity=1.8e-5, inflow_velocity=0.6, aoa_deg=1.5, cfl_number=0.3, final_time=1e30,
                            limiter_k=5.0, verbosity=0, **kw)


# cells a wave of tiles holds: 75,776
@pytest.mark.parametrize("n_surface,n_layers,lo,hi,tiles", [
    (260, 140, 70000, 75776, ("fp64", "fp32")),
    (280, 140, 75777, 132608, ("fp64",)),
    (340, 210, 132609, 151552, ("fp64", "fp32")),
    (350, 236, 151553, 179999, ("fp64",)),
])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_kernels_by_size_and_precision(n_surface, n_layers, lo, hi, tiles, precision):
    from optimisation2forme_b200 import Batch, Solver
    m = small_mesh(triangles=True, n_surface=n_surface, n_layers=n_layers, seed=5)
    p = _params(precision=precision)
    with Solver(p, desc=desc_of(m)) as a, Solver(p, desc=desc_of(m)) as b:
        assert lo <= a.n_cells <= hi
        U = perturbed_freestream(a.n_cells, p, seed=1)
        a.set_state(U)
        b.set_state(U)
        before = a.timing()["kernel_launches"]
        ra = a.time_loop(16)
        per_step = (a.timing()["kernel_launches"] - before) / 16
        assert per_step < 8 if precision in tiles else per_step > 15
        with Batch([b]) as batch:
            rb = batch.time_loop(16)[0]
        assert ra["steps"] == rb["steps"] == 16 and ra["t"] == rb["t"]
        assert bits_equal(a.get_state(), b.get_state())
