"""The time loop's tile kernels and the branch-free FP64 arithmetic
(optimisation2forme_b200/csrc/kernels_tile.cuh, qdiv.h) where they can go
wrong: states whose quotients leave the fast path's range against the CPU
oracle, and the tile kernels against the separate kernels (the batched loop)
at ragged tile counts, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal, desc_of, perturbed_freestream, small_mesh
from oracle import cpu

pytestmark = pytest.mark.gpu


def _params(**kw):
    from optimisation2forme_b200 import SimulationParams
    d = dict(viscosity=1.8e-5, inflow_velocity=0.6, aoa_deg=0.0, cfl_number=0.3, final_time=1e30, limiter_k=5.0,
             verbosity=0)
    d.update(kw)
    return SimulationParams(**d)


def _states(nc, p):
    U = perturbed_freestream(nc, p, seed=3)
    fs = np.tile(perturbed_freestream(1, p, amp=0.0), nc)
    yield "uniform", fs
    for name, f in (("supersonic", 6.0), ("backwards", -6.0)):
        q = U.reshape(-1, 4).copy()
        q[:, 3] += 0.5 * (f * f - 1.0) * (q[:, 1] ** 2 + q[:, 2] ** 2) / q[:, 0]
        q[:, 1:3] *= f
        yield name, q.reshape(-1)
    yield "tiny", U * 1e-130
    yield "huge", U * 1e130
    q = U.reshape(-1, 4).copy()
    q[5::97] *= 1e-220
    q[11::89] *= 1e120
    yield "uneven", q.reshape(-1)
    q = U.reshape(-1, 4).copy()
    q[3::50, 3] *= 0.05  # negative pressure
    q[7::61, 2] = 0.0
    yield "negative pressure", q.reshape(-1)
    q = U.reshape(-1, 4).copy()
    q[9, 0] = 0.0
    q[31, 1] = np.nan
    yield "not numbers", q.reshape(-1)


def _same(a, b):
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(np.where(nan, 0.0, a).view(np.int64), np.where(nan, 0.0, b).view(np.int64))


@pytest.mark.parametrize("triangles", [True, False])
@pytest.mark.parametrize("limiter", ["venkatakrishnan", "barth_jespersen"])
def test_residual_outside_the_fast_range_equals_the_oracle(triangles, limiter):
    from optimisation2forme_b200 import HostMesh, Solver
    m = small_mesh(triangles=triangles, n_surface=40, n_layers=9, seed=2)
    p = _params(limiter=limiter)
    o = cpu.Oracle(HostMesh(desc=desc_of(m)), p)
    with Solver(p, desc=desc_of(m)) as s:
        for name, U in _states(s.n_cells, p):
            s.set_state(U)
            with np.errstate(all="ignore"):
                ref = o.residual(U)
            assert _same(s.compute_residual(), ref["R"]), name
            assert _same(s.debug("edge_LR"), ref["edge_LR"].reshape(-1)), name


# a single ragged tile; one full tile; one cell more than a tile's multiple
# (16 columns of 8 cells = 128); several; quadrilaterals
@pytest.mark.parametrize("n_surface,n_layers,triangles", [
    (8, 8, True), (12, 8, False), (28, 12, False), (60, 33, True), (120, 41, False),
])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_tile_loop_equals_separate_kernels(n_surface, n_layers, triangles, precision):
    from optimisation2forme_b200 import Batch, Solver
    m = small_mesh(triangles=triangles, n_surface=n_surface, n_layers=n_layers, seed=5)
    p = _params(precision=precision, aoa_deg=1.5)
    with Solver(p, desc=desc_of(m)) as a, Solver(p, desc=desc_of(m)) as b:
        U = perturbed_freestream(a.n_cells, p, seed=1)
        a.set_state(U)
        b.set_state(U)
        ra = a.time_loop(7)
        with Batch([b]) as batch:
            rb = batch.time_loop(7)[0]
        assert ra["steps"] == rb["steps"] == 7 and ra["t"] == rb["t"]
        assert bits_equal(a.get_state(), b.get_state())
        for name in ("edge_LR", "edge_tau", "edge_F", "vertex_U", "R"):
            if precision == "fp64":
                assert bits_equal(a.debug(name), b.debug(name)), name
        assert a.lift_drag(0.1) == b.lift_drag(0.1)


def test_a_vertex_of_many_cells():
    """More cells about a vertex than the kernels hold in registers."""
    from optimisation2forme_b200 import Batch, HostMesh, Solver
    n = 13
    t = np.linspace(0.0, 2 * np.pi, n, endpoint=False)
    xy = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(t), np.sin(t)], axis=1)]).reshape(-1)
    ring = np.arange(n)
    m = dict(node_xy=xy, segments=np.stack([1 + ring, 1 + (ring + 1) % n], axis=1),
             segment_bc=np.full(n, ord("f"), dtype=np.uint8), cell_offsets=np.arange(0, 3 * n + 1, 3),
             cell_nodes=np.stack([0 * ring, 1 + ring, 1 + (ring + 1) % n], axis=1).reshape(-1))
    p = _params()
    o = cpu.Oracle(HostMesh(desc=desc_of(m)), p)
    with Solver(p, desc=desc_of(m)) as a, Solver(p, desc=desc_of(m)) as b:
        U = perturbed_freestream(n, p, seed=4)
        a.set_state(U)
        assert bits_equal(a.compute_residual(), o.residual(U)["R"])
        b.set_state(U)
        a.time_loop(3)
        with Batch([b]) as batch:
            batch.time_loop(3)
        assert bits_equal(a.get_state(), b.get_state())
