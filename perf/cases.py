"""The work whose speed is measured: what a program that uses this framework
has it do, through its public entry points, over the sizes it does it at.

A user of the framework builds a ``Solver`` per airfoil mesh, marches the flow
(``time_loop``, alone or in a ``Batch``), solves the adjoint and takes the
shape gradient (``solve_adjoint_system``, ``compute_shape_gradient``,
``optimize_shape``), and trains and queries the warm-start ``Network``.  The
kinds below are those calls; sizes are the ones of ``meshgen.config_mesh``,
of ``bench.py``'s candidates (30k-77k cells) and of the tests (2k-20k cells).

  residual   load a state, one residual, read it back
  rk3        load a state, a run of SSP-RK3 steps, read state and history back
  batch      the same for several candidates of uneven sizes in one batch
  adjoint    residual of a loaded state, forces, adjoint solve (to the
             tolerance, or a bounded number of iterations of it: a whole
             solve of a fine mesh takes seconds), shape gradient
  adjoints   the same for several candidates at once, a host thread and a
             stream for each
  optimise   residual, then ``optimize_shape`` as one call
  train      Adam steps of the warm-start network on a data set it holds
  predict    the network's values at every cell of a mesh

Flows follow the configurations (M 0.5-0.85, AoA 0-4 deg, the reference's
viscosity, thermal time-step bound, Venkatakrishnan K = 5) and states are
made from the seed: freestream with a boundary layer at the wall, a dipole,
acoustic pulses, a shear layer and, from M 0.7 up, a shock.  The adjoint is
taken about a state that the time loop has reached: those kinds start near the
freestream and take some steps (in plain torch) when the inputs are made.
"""
from __future__ import annotations

import functools
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

BETA = 0.1
NAMES = ["m", "p", "t"]
GAMMA, RHO, P0, CP, PR, MU = 1.4, 1.225, 101325.0, 1005.0, 0.71, 1.8e-5

# ---------------------------------------------------------------------------
# Cases


def _grid(cells: int, triangles: bool = True) -> tuple[int, int]:
    """(surface points, layers) of an O-grid of about `cells` cells."""
    per = 2 if triangles else 1
    ni = max(48, int(round(math.sqrt(2 * cells / per) / 2)) * 2)
    return ni - 4, max(8, int(round(cells / (per * ni))))


def listed():
    return [
        # The smallest call: one residual of a coarse mesh of quadrilaterals
        # (the reference's own cell type) with the Barth-Jespersen limiter.
        dict(name="residual_4k_quads_bj", kind="residual", n_surface=92, n_layers=43, triangles=False,
             limiter="barth_jespersen", precision="fp64", first_height=1e-3, mach=0.5, aoa=0.0),
        # The small configuration (NACA 2412, ~20k triangles, M 0.6, AoA 2):
        # many short steps.
        dict(name="rk3_20k", kind="rk3", n_surface=200, n_layers=50, triangles=True, limiter="venkatakrishnan",
             precision="fp64", first_height=2e-3, mach=0.6, aoa=2.0, steps=300),
        # Quadrilaterals of an ordinary, odd size.
        dict(name="rk3_quads_57k", kind="rk3", n_surface=337, n_layers=171, triangles=False,
             limiter="venkatakrishnan", precision="fp64", first_height=1e-3, mach=0.7, aoa=1.0, steps=150),
        # The large transonic configuration: 2.0M triangles, first cell 1e-4
        # chord, M 0.85, in FP64.
        dict(name="rk3_2m", kind="rk3", n_surface=1400, n_layers=715, triangles=True, limiter="venkatakrishnan",
             precision="fp64", first_height=1e-4, mach=0.85, aoa=1.25, steps=60),
        # The mixed-precision configuration: ~500k triangles, FP32 residual.
        dict(name="rk3_fp32_500k", kind="rk3", n_surface=700, n_layers=357, triangles=True,
             limiter="venkatakrishnan", precision="fp32", first_height=1e-4, mach=0.65, aoa=2.5, steps=150),
        # Eight candidates of uneven sizes, as the benchmark batches them.
        dict(name="batch_8_candidates", kind="batch", count=8, cells_lo=30000, cells_hi=77000, mesh_seed=3,
             precision="fp64", steps=60),
        # The adjoint and gradient of one benchmark candidate: FP32 Jacobian
        # blocks, FP64 refinement.
        dict(name="adjoint_75k_mixed", kind="adjoint", n_surface=270, n_layers=136, triangles=True,
             first_height=1e-3, mach=0.72, aoa=1.7, adjoint_precision="fp32", tol=1e-8, iterations=60),
        # The same of a mesh beyond the candidates' sizes, all in FP64.
        dict(name="adjoint_300k", kind="adjoint", n_surface=546, n_layers=273, triangles=True, first_height=1e-3,
             mach=0.6, aoa=2.0, adjoint_precision="fp64", tol=1e-8, iterations=30),
        # Eight candidates' adjoints at once (the benchmark's fast path).
        dict(name="adjoints_8_at_once", kind="adjoints", count=8, cells_lo=30000, cells_hi=77000, mesh_seed=5,
             adjoint_precision="fp32", tol=1e-8, iterations=40),
        # One whole shape-gradient evaluation of a coarse mesh to the default
        # tolerance.
        dict(name="optimise_5k", kind="optimise", n_surface=96, n_layers=25, triangles=True, first_height=2e-3,
             mach=0.6, aoa=2.0, adjoint_precision="fp64", tol=1e-6),
        # Warm-start network: training at the benchmark's batch size on the
        # points of a few fields, and the prediction for one candidate.
        dict(name="train_4096", kind="train", points=200000, batch=4096, steps=60),
        dict(name="predict_75k", kind="predict", points=74528, max_batch=16384),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["residual", "rk3", "rk3", "rk3", "batch", "adjoint", "adjoint", "adjoints", "optimise",
                       "train", "predict"])
    flow = dict(mach=round(rng.uniform(0.5, 0.85), 3), aoa=round(rng.uniform(0.0, 4.0), 3))
    tri = rng.random() < 0.75
    limiter = "venkatakrishnan" if rng.random() < 0.75 else "barth_jespersen"
    precision = "fp64" if rng.random() < 0.7 else "fp32"
    if kind == "residual":
        ns, nl = _grid(int(_log(rng, 2000, 1000000)), tri)
        return dict(kind=kind, n_surface=ns, n_layers=nl, triangles=tri, limiter=limiter, precision=precision,
                    first_height=1e-3, **flow)
    if kind == "rk3":
        cells = int(_log(rng, 2400, 1900000))
        ns, nl = _grid(cells, tri)
        return dict(kind=kind, n_surface=ns, n_layers=nl, triangles=tri, limiter=limiter, precision=precision,
                    first_height=1e-3 if cells < 300000 else 2e-4, steps=max(20, min(300, 30000000 // cells)), **flow)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 24), cells_lo=20000, cells_hi=rng.randint(30000, 90000),
                    mesh_seed=rng.randrange(1000), precision=precision, steps=rng.randint(20, 60))
    if kind == "adjoint":
        cells = int(_log(rng, 5000, 400000))
        ns, nl = _grid(cells, tri)
        return dict(kind=kind, n_surface=ns, n_layers=nl, triangles=tri, first_height=1e-3,
                    adjoint_precision=rng.choice(["fp64", "fp32"]), tol=1e-8,
                    iterations=max(20, min(60, 9000000 // cells)), **flow)
    if kind == "adjoints":
        return dict(kind=kind, count=rng.randint(2, 15), cells_lo=20000, cells_hi=rng.randint(30000, 90000),
                    mesh_seed=rng.randrange(1000), adjoint_precision="fp32", tol=1e-8,
                    iterations=rng.randint(15, 30))
    if kind == "optimise":
        ns, nl = _grid(int(_log(rng, 2400, 8000)), tri)
        return dict(kind=kind, n_surface=ns, n_layers=nl, triangles=tri, first_height=2e-3,
                    adjoint_precision=rng.choice(["fp64", "fp32"]), tol=1e-6,
                    mach=round(rng.uniform(0.5, 0.65), 3), aoa=flow["aoa"])
    if kind == "train":
        return dict(kind=kind, points=rng.randint(20000, 400000), batch=int(_log(rng, 256, 16384)),
                    steps=rng.randint(10, 60))
    return dict(kind=kind, points=int(_log(rng, 1000, 400000)), max_batch=rng.choice([4096, 16384]))


# ---------------------------------------------------------------------------
# Inputs


def _sections(case) -> list[dict]:
    """One mesh and flow for each context of the case."""
    if "n_surface" in case:
        return [dict(m=0.02, p=0.4, t=0.12, n_surface=case["n_surface"], n_layers=case["n_layers"],
                     triangles=case["triangles"], first_height=case["first_height"], seed=0, mach=case["mach"],
                     aoa=case["aoa"])]
    rng = np.random.default_rng(case["mesh_seed"])
    out = []
    for i in range(case["count"]):
        m, p, t = float(rng.uniform(0, 0.06)), float(rng.uniform(0.2, 0.6)), float(rng.uniform(0.08, 0.18))
        mach, aoa = float(rng.uniform(0.5, 0.8)), float(rng.uniform(0.0, 4.0))
        cells = float(rng.uniform(case["cells_lo"], case["cells_hi"]))
        ni = max(64, int(round(np.sqrt(cells) / 2)) * 2)
        out.append(dict(m=m, p=p, t=t, n_surface=ni - 4, n_layers=max(8, int(round(cells / (2 * ni)))),
                        triangles=True, first_height=1e-3, seed=case["mesh_seed"] * 1000 + i, mach=mach, aoa=aoa))
    return out


@functools.lru_cache(maxsize=64)
def _mesh_of(key) -> dict:
    from optimisation2forme_b200.meshgen import OGridSpec, naca_ogrid
    return naca_ogrid(OGridSpec(growth=1.1, **dict(key)))


def _mesh(sec: dict) -> dict:
    return _mesh_of(tuple(sorted((k, v) for k, v in sec.items() if k not in ("mach", "aoa"))))


def _state(sec: dict, mesh: dict, seed: int) -> np.ndarray:
    """A flow field about the section, [4 * n_cells]."""
    rng = np.random.default_rng([seed, mesh["cell_nodes"].size])
    xy = mesh["node_xy"].reshape(-1, 2)
    ni = int((mesh["segment_bc"] == ord("w")).sum())
    wall = np.linalg.norm(xy.reshape(-1, ni, 2) - xy[:ni], axis=2).reshape(-1)  # distance along the grid line
    n = 3 if sec["triangles"] else 4
    nodes = mesh["cell_nodes"].reshape(-1, n)
    c, d = xy[nodes].mean(axis=1), wall[nodes].mean(axis=1)
    x, y = c[:, 0] - 0.855, c[:, 1]
    a0 = math.sqrt(GAMMA * P0 / RHO)
    U = sec["mach"] * a0
    al = math.radians(sec["aoa"])
    r2 = x * x + y * y + 0.05
    k = rng.uniform(0.02, 0.05)
    u = U * (math.cos(al) - k * (x * x - y * y) / (r2 * r2))  # a dipole's far field
    v = U * (math.sin(al) - 2 * k * x * y / (r2 * r2))
    q = 1.0 - 0.5 * GAMMA * sec["mach"] ** 2 * ((u * u + v * v) / (U * U) - 1.0) * 0.5
    p = P0 * np.clip(q, 0.6, 1.6)
    for _ in range(4):  # pulses
        x0, y0, s = rng.uniform(-1.0, 1.5), rng.uniform(-0.8, 0.8), rng.uniform(0.1, 0.4)
        g = rng.uniform(-0.04, 0.04) * np.exp(-((x - x0) ** 2 + (y - y0) ** 2) / (s * s))
        p = p * (1.0 + g)
        u = u + U * g
        v = v + 0.5 * U * g
    if sec["mach"] >= 0.7:  # a shock above the section
        xs = rng.uniform(0.0, 0.25)
        p = p * (1.0 + 0.12 * np.tanh((x - xs) / 0.03) * np.exp(-((y - 0.3) / 0.4) ** 2))
    u = u * (1.0 + 0.03 * np.tanh(y / 0.2) * np.exp(-0.1 * (x - 1.0) ** 2))  # shear layer
    bl = np.tanh(d / rng.uniform(0.02, 0.05))
    u, v = u * bl, v * bl
    rho = RHO * (p / P0) ** (1.0 / GAMMA)
    return np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], axis=1).reshape(-1)


def _start(case, sec, mesh, seed: int) -> np.ndarray:
    """The state the case's calls begin with."""
    U = _state(sec, mesh, seed)
    if case["kind"] not in ("adjoint", "adjoints", "optimise"):
        return U
    x = _exact_of(sec, "venkatakrishnan")
    q = x.fs + 0.02 * (torch.as_tensor(U, device=x.dev).reshape(-1, 4) - x.fs)
    return x.march(q, 30 if case["kind"] == "optimise" else 12)[0].reshape(-1).cpu().numpy()


def _solver(case, sec, mesh, stream=None):
    from optimisation2forme_b200 import SimulationParams, Solver, mesh_desc
    prm = SimulationParams(viscosity=MU, inflow_velocity=sec["mach"], aoa_deg=sec["aoa"], cfl_number=0.4,
                           final_time=1e30, limiter_k=5.0, dt_mode="thermal",
                           limiter=case.get("limiter", "venkatakrishnan"), precision=case.get("precision", "fp64"),
                           adjoint_precision=case.get("adjoint_precision", "fp64"), verbosity=0)
    return Solver(prm, desc=mesh_desc(mesh["node_xy"], mesh["segments"], mesh["segment_bc"], mesh["cell_offsets"],
                                      mesh["cell_nodes"]), stream=stream)


def _points(n: int, seed: int) -> tuple[np.ndarray, np.ndarray]:
    """Standardised network inputs and smooth targets."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, 7)).astype(np.float32)
    f = rng.standard_normal((7, 8)).astype(np.float32)
    y = np.sin(x @ f) + 0.3 * np.cos(2.0 * x[:, :1]) * x[:, 1:2]
    return x, y.astype(np.float32)


def _weights(n: int, seed: int) -> np.ndarray:
    """Parameters of a trained network's magnitude, in o2f_mlp's layout."""
    rng = np.random.default_rng([seed, n])
    out = []
    for i, o in ((128, 256), (256, 256), (256, 256), (256, 256), (256, 16)):
        w = rng.standard_normal((o, i)) * math.sqrt(2.0 / i)
        b = 0.1 * rng.standard_normal(o)
        w[8 if o == 16 else o:] = 0.0
        b[8 if o == 16 else o:] = 0.0
        out += [w.reshape(-1), b]
    p = np.concatenate(out).astype(np.float32)
    assert p.size == n
    return p


def _network(case, seed):
    from optimisation2forme_b200.warmstart import Network
    net = Network(max_batch=max(128, case.get("max_batch", case.get("batch", 128))), freq_scale=1.0, seed=0)
    net.set_params(_weights(net.n_params, seed))
    return net


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, y = _points(case["points"], seed)
        net = _network(case, seed)
        net.set_data(x, y)
        return dict(case=case, net=net, w=_weights(net.n_params, seed), seed=seed)
    if kind == "predict":
        return dict(case=case, net=_network(case, seed), x=_points(case["points"], seed)[0])
    secs = _sections(case)
    meshes = [_mesh(s) for s in secs]
    U = [_start(case, s, m, seed) for s, m in zip(secs, meshes)]
    streams = [torch.cuda.Stream() for _ in secs] if kind == "adjoints" else [None] * len(secs)
    solvers = [_solver(case, s, m, st.cuda_stream if st else None) for s, m, st in zip(secs, meshes, streams)]
    st = dict(case=case, secs=secs, solvers=solvers, streams=streams, U=U)
    if kind == "batch":
        from optimisation2forme_b200 import Batch
        st["batch"] = Batch(solvers)
    if kind == "adjoints":
        st["pool"] = ThreadPoolExecutor(max_workers=len(secs))
    for s, u in zip(solvers, U):
        s.set_state(u)
    return st


# ---------------------------------------------------------------------------
# One pass


def _shape(sec):
    from optimisation2forme_b200._lib import ShapeParams
    return ShapeParams(0.355, 1.0, sec["m"], sec["p"], sec["t"])


def _adjoint(case, s, sec) -> dict:
    s.compute_residual()
    f = s.lift_drag(BETA)
    a = s.solve_adjoint_system(BETA, tol=case["tol"], max_iter=case["iterations"], restart=500,
                               raise_on_failure=False)
    g = s.compute_shape_gradient(NAMES, _shape(sec), beta=BETA)
    return dict(forces=np.array(f), lam=a["lambda"], iters=a["iters"], grad=g)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "residual":
        s = state["solvers"][0]
        s.set_state(state["U"][0])
        return dict(R=s.compute_residual())
    if kind == "rk3":
        s = state["solvers"][0]
        s.set_state(state["U"][0])
        r = s.time_loop(case["steps"])
        return dict(U=s.get_state(), history=r["history"], t=r["t"], steps=r["steps"])
    if kind == "batch":
        for s, u in zip(state["solvers"], state["U"]):
            s.set_state(u)
        r = state["batch"].time_loop(case["steps"])
        return dict(U=[s.get_state() for s in state["solvers"]],
                    t=np.array([x["t"] for x in r]),
                    steps=np.array([x["steps"] for x in r]))
    if kind == "adjoint":
        return _adjoint(case, state["solvers"][0], state["secs"][0])
    if kind == "adjoints":
        return list(state["pool"].map(lambda z: _adjoint(case, *z), zip(state["solvers"], state["secs"])))
    if kind == "optimise":
        s = state["solvers"][0]
        s.compute_residual()
        f = s.lift_drag(BETA)
        r = s.optimize_shape(NAMES, _shape(state["secs"][0]), beta=BETA, tol=case["tol"])
        return dict(forces=np.array(f), J=r["J"], iters=r["iters"], grad=r["grad"])
    if kind == "train":
        net = state["net"]
        net.set_params(state["w"])
        loss = net.train(case["steps"], batch=case["batch"], lr=1e-3, seed=state["seed"])
        return dict(loss=loss, params=net.params()[0])
    return dict(Y=state["net"].predict(state["x"]))


# ---------------------------------------------------------------------------
# Work


def _counts(case):
    for sec in _sections(case):
        ni, per = 2 * (sec["n_surface"] // 2) + 4, 2 if sec["triangles"] else 1
        nc, nv = per * ni * sec["n_layers"], ni * (sec["n_layers"] + 1)
        corners = nc * (3 if per == 2 else 4)
        yield nc, (corners + 2 * ni) // 2, nv, corners


def work(case):
    kind = case["kind"]
    if kind in ("train", "predict"):
        n = 128 * 256 + 3 * 256 * 256 + 256 * 8
        if kind == "train":
            return {"bytes": case["steps"] * (case["batch"] * 60.0 + 28.0 * n),
                    "flops": 6.0 * n * case["batch"] * case["steps"]}
        return {"bytes": case["points"] * 60.0 + 2.0 * n, "flops": 2.0 * n * case["points"]}
    w = 4 if case.get("precision") == "fp32" else 8
    total = 0.0
    for nc, ne, nv, corners in _counts(case):
        geometry = nc * (16 + 3 * w) + ne * (16 + 5 * w) + nv * 4 + corners * (4 + w)  # of one residual
        residual = geometry + nc * 8 * w  # state in, residual out
        if kind == "residual":
            total += residual
        elif kind in ("rk3", "batch"):  # three residuals a step; state and old state in, state out
            total += case["steps"] * (3 * geometry + nc * 32 * 8)
        else:
            iters = case.get("iterations", 150)
            blk = 4 if case["adjoint_precision"] == "fp32" else 8
            product = ne * (32 * blk + 17) + nc * (8 + 16 + 64)
            sweeps = nc * 64 + (nc + 2 * ne) * 128  # factor blocks, vector in and out
            total += iters * (2 * (product + sweeps) + 12 * 32 * nc)
            total += 8 * residual + ne * 320  # state's and perturbed residuals, blocks
    return {"bytes": float(total), "flops": 0.0}


# ---------------------------------------------------------------------------
# The same in 64 bits, in plain torch


class _Exact:
    """Residual and forces of a mesh (reference formulas, in the order that
    suits arrays)."""

    def __init__(self, sec, mesh, limiter):
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = functools.partial(torch.as_tensor, device=dev)
        n = 3 if sec["triangles"] else 4
        xy = t(mesh["node_xy"]).reshape(-1, 2)
        cn = t(mesh["cell_nodes"]).reshape(-1, n)
        nv, nc = xy.shape[0], cn.shape[0]
        self.nc, self.nv, self.n = nc, nv, n
        a0 = math.sqrt(GAMMA * P0 / RHO)
        ux, uy = (sec["mach"] * a0 * f(math.radians(sec["aoa"])) for f in (math.cos, math.sin))
        self.axes = (math.cos(math.radians(sec["aoa"])), math.sin(math.radians(sec["aoa"])))
        self.fs = t(np.array([RHO, RHO * ux, RHO * uy, P0 / (GAMMA - 1) + 0.5 * RHO * (ux * ux + uy * uy)]))
        self.q_inf = 0.5 * RHO * (ux * ux + uy * uy)
        # cells
        X = xy[cn]

        def cross(p, q):
            return p[:, 0] * q[:, 1] - q[:, 0] * p[:, 1]

        self.vol = 0.5 * cross(X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]).abs()
        if n == 4:
            self.vol = self.vol + 0.5 * cross(X[:, 1] - X[:, 2], X[:, 3] - X[:, 2]).abs()
        self.ctr = X.mean(dim=1)
        self.eps = (5.0 * torch.sqrt(self.vol / math.pi)) ** 3
        self.limiter = limiter
        # edges: the first cell that has one is its left cell
        a, b = cn, torch.roll(cn, -1, dims=1)
        key = torch.minimum(a, b) * nv + torch.maximum(a, b)
        uniq, inv = torch.unique(key.reshape(-1), return_inverse=True)
        ne = uniq.numel()
        owner = torch.arange(nc, device=dev).repeat_interleave(n)
        cl = torch.full((ne,), nc, device=dev).scatter_reduce(0, inv, owner, "amin")
        cr = torch.full((ne,), -1, device=dev).scatter_reduce(0, inv, owner, "amax")
        inner = cr != cl
        self.cl, self.inner, self.cr = cl, inner, torch.where(inner, cr, cl)
        self.v0, self.v1 = uniq // nv, uniq % nv
        seg, bc = t(mesh["segments"]).reshape(-1, 2), t(mesh["segment_bc"])
        self.vwall = torch.zeros(nv, dtype=torch.bool, device=dev)
        self.vfar = torch.zeros(nv, dtype=torch.bool, device=dev)
        self.vwall[seg[bc == ord("w")].reshape(-1)] = True
        self.vfar[seg[bc == ord("f")].reshape(-1)] = True
        sk = seg.min(dim=1).values * nv + seg.max(dim=1).values
        at = torch.searchsorted(uniq, sk)
        self.ewall = torch.zeros(ne, dtype=torch.bool, device=dev)
        self.efar = torch.zeros(ne, dtype=torch.bool, device=dev)
        self.ewall[at[bc == ord("w")]] = True
        self.efar[at[bc == ord("f")]] = True
        d = xy[self.v0] - xy[self.v1]
        self.len = torch.linalg.norm(d, dim=1)
        nrm = torch.stack([d[:, 1], -d[:, 0]], dim=1) / self.len[:, None]
        self.ectr = 0.5 * (xy[self.v0] + xy[self.v1])
        flip = ((self.ctr[cl] - self.ectr) * nrm).sum(dim=1) < 0
        self.nrm = torch.where(flip[:, None], -nrm, nrm)  # toward the left cell
        per = self.len[inv].reshape(nc, n).sum(dim=1)
        self.min_h = float((2.0 * self.vol / per).min())
        # vertex weights over the cells about each vertex, by angle
        pv, pc = cn.reshape(-1), owner
        off = self.ctr[pc] - xy[pv]
        order = torch.argsort(torch.atan2(off[:, 1], off[:, 0]), stable=True)
        order = order[torch.argsort(pv[order], stable=True)]
        pv, pc, off = pv[order], pc[order], off[order]
        cnt = torch.bincount(pv, minlength=nv)
        start = torch.cumsum(cnt, 0) - cnt
        pos = torch.arange(pv.numel(), device=dev) - start[pv]
        m = cnt[pv]
        nxt, prv = start[pv] + (pos + 1) % m, start[pv] + (pos + m - 1) % m
        dist = torch.linalg.norm(off, dim=1)
        e = off / dist[:, None]

        def half(i, j):
            return torch.tan(0.5 * torch.acos((e[i] * e[j]).sum(dim=1).clamp(-1.0, 1.0)))

        me = torch.arange(pv.numel(), device=dev)
        w = (half(prv, me) + half(me, nxt)) / dist  # mean value
        bnd = (self.vwall | self.vfar)[pv]
        w = torch.where(bnd & (m > 4), 1.0 / dist, w)
        w = torch.where(m <= 2, torch.ones_like(w), w)
        w = torch.where(m == 3, cross(off[nxt], off[prv]), w)  # barycentric
        # as rows of each vertex, so that sums have one order
        self.fan = torch.zeros((nv, int(cnt.max())), dtype=torch.int64, device=dev)
        self.fan_w = torch.zeros(self.fan.shape, dtype=torch.float64, device=dev)
        self.fan[pv, pos], self.fan_w[pv, pos] = pc, w
        self.fan_w /= self.fan_w.sum(dim=1, keepdim=True)
        self.cell_edges = inv.reshape(nc, n)
        self.cell_sign = torch.where(cl[self.cell_edges] == torch.arange(nc, device=dev)[:, None], 1.0, -1.0).double()

    def at_vertices(self, f):
        return (self.fan_w[:, :, None] * f[self.fan]).sum(dim=1)

    def _bc(self, q, wall, far):
        still = torch.stack([q[:, 0], 0 * q[:, 0], 0 * q[:, 0],
                             q[:, 3] - 0.5 * (q[:, 1] ** 2 + q[:, 2] ** 2) / q[:, 0]], dim=1)
        q = torch.where(wall[:, None], still, q)
        return torch.where(far[:, None], self.fs, q)

    def to_cells(self, f):
        """Sum over each cell's edges of f, outward for the left cell."""
        return (self.cell_sign[:, :, None] * f[self.cell_edges]).sum(dim=1) / self.vol[:, None]

    def residual(self, U):
        cl, cr, inner = self.cl, self.cr, self.inner
        vq = self._bc(self.at_vertices(U), self.vwall, self.vfar)
        eq = self._bc(0.5 * (vq[self.v0] + vq[self.v1]), self.ewall, self.efar)
        nL = -self.nrm * self.len[:, None]  # outward of the left cell
        gx, gy = self.to_cells(eq * nL[:, :1]), self.to_cells(eq * nL[:, 1:])
        mn, mx = U.clone(), U.clone()
        for at, of in ((cl, cr), (cr, cl)):
            i = at[inner][:, None].expand(-1, 4)
            mn.scatter_reduce_(0, i, U[of[inner]], "amin")
            mx.scatter_reduce_(0, i, U[of[inner]], "amax")
        alpha = torch.ones_like(U)
        steps = {}
        for side, at in (("L", cl), ("R", cr)):
            dx = (self.ectr - self.ctr[at])
            step = gx[at] * dx[:, :1] + gy[at] * dx[:, 1:]
            steps[side] = step
            u = U[at]
            delta = (u + step) - u
            room = torch.where(delta > 0, mx[at] - u, mn[at] - u)
            tiny = delta.abs() < 2.220446049250313e-16
            if self.limiter == "venkatakrishnan":
                ep = self.eps[at][:, None]
                al = ((room * room + ep + 2 * room * delta) / (room * room + ep + 2 * delta * delta)).clamp(0.0, 1.0)
            else:
                al = (room / delta).clamp(max=1.0)
            al = torch.where(tiny, torch.ones_like(al), al)
            ok = torch.ones_like(inner) if side == "L" else inner
            alpha.scatter_reduce_(0, at[ok][:, None].expand(-1, 4), al[ok], "amin")
        L = U[cl] + alpha[cl] * steps["L"]
        R = U[cr] + alpha[cr] * steps["R"]
        mirror = L * torch.tensor([1.0, -1.0, -1.0, 1.0], dtype=torch.float64, device=self.dev)
        R = torch.where(self.ewall[:, None], mirror, torch.where(self.efar[:, None], self.fs.expand_as(L), R))
        F = self.hllc(L, R)
        out = -self.to_cells(F * self.len[:, None])
        # viscous terms
        r, u, v = U[:, 0], U[:, 1] / U[:, 0], U[:, 2] / U[:, 0]
        u_x, u_y = (gx[:, 1] - u * gx[:, 0]) / r, (gy[:, 1] - u * gy[:, 0]) / r
        v_x, v_y = (gx[:, 2] - v * gx[:, 0]) / r, (gy[:, 2] - v * gy[:, 0]) / r
        div = (2.0 / 3.0) * MU * (u_x + v_y)
        T_x = (GAMMA - 1) * ((gx[:, 3] * r - U[:, 3] * gx[:, 0]) / (r * r) - (u * u_x + v * v_x))
        T_y = (GAMMA - 1) * ((gy[:, 3] * r - U[:, 3] * gy[:, 0]) / (r * r) - (u * u_y + v * v_y))
        kap = MU * CP / PR
        vt = self.at_vertices(torch.stack([2 * MU * u_x - div, 2 * MU * v_y - div, MU * (u_y + v_x), -kap * T_x,
                                           -kap * T_y], dim=1))
        vt = torch.where((self.vwall | self.vfar)[:, None], torch.zeros_like(vt), vt)
        et = 0.5 * (vt[self.v0] + vt[self.v1])
        et = torch.where((self.ewall | self.efar)[:, None], torch.zeros_like(et), et)
        n0, n1 = nL[:, 0], nL[:, 1]
        sx, sy, qn = et[:, 0] * n0 + et[:, 2] * n1, et[:, 2] * n0 + et[:, 1] * n1, et[:, 3] * n0 + et[:, 4] * n1
        d = self.to_cells(torch.stack([sx, sy, qn], dim=1))
        out[:, 1] += d[:, 0]
        out[:, 2] += d[:, 1]
        out[:, 3] += u * d[:, 0] + v * d[:, 1] - d[:, 2]
        self.last = (L, et)
        return out

    def hllc(self, L, R):
        nx, ny = -self.nrm[:, 0], -self.nrm[:, 1]

        def side(q):
            u, v = (q[:, 1] * nx + q[:, 2] * ny) / q[:, 0], (q[:, 2] * nx - q[:, 1] * ny) / q[:, 0]
            p = (GAMMA - 1) * (q[:, 3] - 0.5 * q[:, 0] * (u * u + v * v))
            return q[:, 0], u, v, q[:, 3], p, torch.sqrt(GAMMA * p / q[:, 0])

        rl, ul, vl, el, pl, al = side(L)
        rr, ur, vr, er, pr, ar = side(R)
        sl, sr = torch.minimum(ul - al, ur - ar), torch.maximum(ul + al, ur + ar)
        ss = (pr - pl + rl * ul * (sl - ul) - rr * ur * (sr - ur)) / (rl * (sl - ul) - rr * (sr - ur))
        ps = pl + rl * (sl - ul) * (ss - ul)

        def star(r, u, v, e, p, s):
            k = r * (s - u) / (s - ss)
            es = ((s - u) * e - p * u + ps * ss) / (s - ss)
            return torch.stack([k * ss, k * ss * ss + ps, v * k * ss, (es + ps) * ss], dim=1)

        def plain(r, u, v, e, p):
            return torch.stack([r * u, r * u * u + p, r * u * v, (e + p) * u], dim=1)

        f = torch.where((ss >= 0)[:, None], star(rl, ul, vl, el, pl, sl), star(rr, ur, vr, er, pr, sr))
        f = torch.where((sl >= 0)[:, None], plain(rl, ul, vl, el, pl), f)
        f = torch.where((sr < 0)[:, None], plain(rr, ur, vr, er, pr), f)
        return torch.stack([f[:, 0], f[:, 1] * nx - f[:, 2] * ny, f[:, 1] * ny + f[:, 2] * nx, f[:, 3]], dim=1)

    def forces(self):
        L, et = self.last
        i = self.ewall
        q, n, A, s = L[i], self.nrm[i], self.len[i], et[i]
        p = (GAMMA - 1) * (q[:, 3] - 0.5 * (q[:, 1] ** 2 + q[:, 2] ** 2) / q[:, 0])
        fx = (-p * n[:, 0] + s[:, 0] * n[:, 0] + s[:, 2] * n[:, 1]) * A
        fy = (-p * n[:, 1] + s[:, 2] * n[:, 0] + s[:, 1] * n[:, 1]) * A
        ca, sa = self.axes

        def lift_drag(k):
            X, Y = fx[k].sum(), fy[k].sum()
            return float((Y * ca - X * sa) / self.q_inf), float((X * ca + Y * sa) / self.q_inf)

        cl, cd = lift_drag(torch.ones_like(fx, dtype=torch.bool))
        jl, jd = lift_drag(~(self.ectr[i, 0] > 1.3))
        return np.array([cl, cd, -jl + BETA * jd])

    def march(self, U, steps):
        mu = max(MU, MU * CP / PR * (GAMMA - 1))
        t, hist = 0.0, []
        for _ in range(steps):
            u, v = U[:, 1] / U[:, 0], U[:, 2] / U[:, 0]
            p = (GAMMA - 1) * (U[:, 3] - 0.5 * U[:, 0] * (u * u + v * v))
            wave = float((torch.hypot(u, v) + torch.sqrt(GAMMA * p / U[:, 0])).max())
            dt = min(0.4 * self.min_h / wave, 0.5 * self.min_h ** 2 / mu)
            U0 = U
            r = self.residual(U)
            hist.append(torch.linalg.norm(r[:, 0]))
            U = U0 + dt * r
            U = 0.75 * U0 + 0.25 * (U + dt * self.residual(U))
            U = (1.0 / 3.0) * U0 + (2.0 / 3.0) * (U + dt * self.residual(U))
            t += dt
        return U, torch.stack(hist).cpu().numpy(), t


@functools.lru_cache(maxsize=16)
def _exact_cached(key, limiter):
    sec = dict(key)
    return _Exact(sec, _mesh(sec), limiter)


def _exact_of(sec, limiter):
    return _exact_cached(tuple(sorted(sec.items())), limiter)


def _features(x, freq):
    arg = 2.0 * math.pi * (x[:, :2] @ freq.T)
    f = torch.cat([torch.sin(arg), torch.cos(arg), x], dim=1)
    return torch.nn.functional.pad(f, (0, 128 - f.shape[1]))


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        # the batches are drawn inside the call and their rounding feeds Adam's
        # signs: a 64-bit run of the same steps is another run
        return None
    if kind == "predict":
        net = _network(case, seed)  # for the Fourier frequencies, which it draws itself
        freq = torch.as_tensor(net.params()[1], dtype=torch.float64).reshape(-1, 2)
        p = torch.as_tensor(_weights(net.n_params, seed), dtype=torch.float64)
        net.close()
        h = _features(torch.as_tensor(_points(case["points"], seed)[0], dtype=torch.float64), freq)
        off = 0
        for k, (i, o) in enumerate(((128, 256), (256, 256), (256, 256), (256, 256), (256, 16))):
            w, b = p[off:off + i * o].reshape(o, i), p[off + i * o:off + i * o + o]
            off += i * o + o
            h = h @ w.T + b
            if k < 4:
                h = torch.nn.functional.silu(h)
        return dict(Y=h[:, :8].contiguous().numpy())
    secs = _sections(case)
    got = []
    for sec in secs:
        mesh = _mesh(sec)
        x = _exact_of(sec, case.get("limiter", "venkatakrishnan"))
        U = torch.as_tensor(_start(case, sec, mesh, seed), device=x.dev).reshape(-1, 4)
        if kind in ("rk3", "batch"):
            got.append(x.march(U, case["steps"]))
        else:
            got.append((x.residual(U), x))
    if kind == "residual":
        return dict(R=got[0][0].reshape(-1).cpu().numpy())
    if kind == "rk3":
        U, hist, t = got[0]
        return dict(U=U.reshape(-1).cpu().numpy(), history=hist, t=t, steps=None)
    if kind == "batch":
        return dict(U=[g[0].reshape(-1).cpu().numpy() for g in got], t=np.array([g[2] for g in got]), steps=None)
    # lambda and the gradient rest on difference quotients with steps of 1e-6,
    # whose own rounding is far above 64 bits: only the forces have such a value
    out = [dict(forces=x.forces(), lam=None, iters=None, grad=None) for _, x in got]
    if kind == "optimise":
        return dict(forces=out[0]["forces"], J=float(out[0]["forces"][2]), iters=None, grad=None)
    return out[0] if kind == "adjoint" else out
