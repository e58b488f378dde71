"""The forward-solve workloads this package is timed on.

Every case goes through the package's public calls (``ForwardModel.evaluate``,
``solve_batch``, ``Server``, ``Mesh.compute_wall_distance``) on the meshes of
the tests and the benchmark, or on meshes of the same families at other sizes.
A case is a dict of plain values; ``kind`` names the call:

  evaluate  one ForwardModel.evaluate of a cold channel, predictions included
  channel   solve_batch of cold plane channels, one theta per instance
  warm      solve_batch from a converged state (a chain's next proposals, or
            the re-solves of a warm finite-difference Jacobian), observed
  mix       solve_batch over channels of uneven size in one call
  step      solve_batch of the backward-facing step with permuted cell ids
  duct      solve_batch of the 3-D square duct with permuted cell ids
  served    requests through the resident Server
  wall      Mesh.compute_wall_distance on the device

A program keeps its meshes, cases (the device handles), servers and converged
start states; they are made once here too.  What changes from call to call is
theta, drawn from the seed.  Most solves are capped at an outer-iteration
count, as a stage of a long solve is: the cost of an outer iteration does not
change much along a solve.
"""
from __future__ import annotations

import functools
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "bayesian-turbulence-modeling_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import rans_sst_py as rs  # noqa: E402
from rans_sst_py._types import COEFF_DEFAULTS  # noqa: E402

ACTIVE = [8, 0, 1, 9, 2, 10]      # beta*, sigma_k1, sigma_w1, a1, beta1, kappa
CHANNEL_INIT = dict(u=(20.0, 0.0, 0.0), p=0.0, k=1e-2, omega=10.0)
MIX_NY = {"small": ((32, 180.0), (64, 180.0), (96, 395.0)),
          "large": ((64, 180.0), (128, 550.0), (256, 1000.0), (512, 2000.0))}
FIELDS = ("U", "p", "k", "omega", "nuT", "F1", "F2", "Pk", "CDkw", "Ub", "pb", "kb", "omegab")


def listed():
    return [
        # the smallest call: one likelihood evaluation of a coarse channel in
        # the reference's arithmetic, where latency is everything
        dict(name="evaluate_ch32", kind="evaluate", ny=32, re=180.0, precision="fp64", tol=1e-5, iters=1500),
        # one proposal of a Markov chain from its last converged state
        dict(name="chain_ch128", kind="warm", mesh="channel", precision="fp64", n=1, iters=120, step=0.02),
        # the 22 warm re-solves of a finite-difference Jacobian
        dict(name="jacobian_ch128", kind="warm", mesh="channel", precision="fp64", n=22, iters=80, step=5e-4),
        # a design sweep over theta in the reference's arithmetic
        dict(name="sweep_ch128_fp64", kind="channel", ny=128, re=550.0, precision="fp64", n=219, iters=60),
        # one mixed-precision solve, cold start to convergence
        dict(name="solve_ch64_mixed", kind="channel", ny=64, re=180.0, precision="mixed", n=1, iters=20000, tol=1e-8),
        # the benchmark's batch in mixed precision, both stages of a solve
        dict(name="sweep_ch128_mixed", kind="channel", ny=128, re=550.0, precision="mixed", n=219, iters=400),
        # one batch over meshes of uneven size
        dict(name="mix_64_to_512_mixed", kind="mix", sizes="large", precision="mixed", n=64, iters=100),
        # a chain proposal on an unstructured mesh (reference-order multigrid)
        dict(name="chain_bfs1920", kind="warm", mesh="bfs", precision="fp64", n=1, iters=12, step=0.02),
        # eight chains on that mesh side by side
        dict(name="chains8_bfs1920", kind="warm", mesh="bfs", precision="fp64", n=8, iters=12, step=0.02),
        # a large unstructured mesh on the whole device
        dict(name="step_123k", kind="step", a=32, precision="fp64", iters=5),
        # a large 3-D mesh, mixed precision
        dict(name="duct_74k_mixed", kind="duct", nx=32, ny=48, nz=48, precision="mixed", iters=8),
        # setup of a large mesh: distance to the nearest wall face
        dict(name="wall_123k", kind="wall", a=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["evaluate", "channel", "channel", "channel", "warm", "warm", "mix", "step", "duct", "served",
                       "wall"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "evaluate":
        return dict(kind=kind, ny=2 * rng.randint(8, 40), re=round(rng.uniform(120.0, 400.0), 1),
                    precision=precision, tol=1e-5, iters=rng.randint(300, 900))
    if kind == "channel":
        ny = 2 * _log_int(rng, 8, 200)
        n = _log_int(rng, 1, 256)
        most = 219 * 128 * 60 * (4 if precision == "mixed" else 1)
        iters = min(rng.randint(40, 300), max(8, most // (ny * max(n, 100))))
        return dict(kind=kind, ny=ny, re=round(180.0 * (ny / 32.0) ** 0.8, 1), precision=precision, n=n, iters=iters)
    if kind == "warm":
        mesh = rng.choice(["channel", "bfs"])
        n = _log_int(rng, 1, 200 if mesh == "channel" else 24)
        iters = rng.randint(20, 60) if mesh == "channel" else rng.randint(4, 10)
        return dict(kind=kind, mesh=mesh, precision="fp64", n=n, iters=iters, step=rng.choice([5e-4, 0.02]))
    if kind == "mix":
        return dict(kind=kind, sizes=rng.choice(["small", "large"]), precision=precision, n=_log_int(rng, 3, 120),
                    iters=rng.randint(20, 60))
    if kind == "step":
        a = _log_int(rng, 4, 31)
        return dict(kind=kind, a=a, precision="fp64", iters=rng.randint(2, 5))
    if kind == "duct":
        return dict(kind=kind, nx=rng.randint(4, 40), ny=2 * rng.randint(5, 22), nz=2 * rng.randint(5, 22),
                    precision=precision, iters=rng.randint(2, 5))
    if kind == "served":
        return dict(kind=kind, precision=precision, n=_log_int(rng, 2, 64), iters=rng.randint(40, 150))
    return dict(kind=kind, a=rng.randint(6, 31))


# ---- what a program keeps ----------------------------------------------------
def _settings(precision, iters, tol, force):
    s = rs.SolverSettings()
    s.verbose = False
    s.max_iterations = iters
    s.convergence_tol = tol
    s.precision = precision
    if force:
        s.body_force = rs.Vec3(1.0, 0.0, 0.0)
    return s


def _ratio(y1, n):
    """Growth ratio of n geometric cells over height 1 whose first cell is y1."""
    lo, hi = 1.0 + 1e-12, 3.0
    for _ in range(200):
        r = 0.5 * (lo + hi)
        lo, hi = (r, hi) if y1 * (r ** n - 1.0) / (r - 1.0) < 1.0 else (lo, r)
    return 0.5 * (lo + hi)


@functools.lru_cache(maxsize=None)
def _channel_mesh(ny, re):
    ratio = 1.08 if ny == 128 else _ratio(0.4 / re, ny // 2)
    m = rs.Mesh.make_channel_periodic_geometric(4, ny, 1.0, 1.0, ratio)
    m.compute_wall_distance()
    return m, rs.FlowBoundaryConditions.channel_defaults(m, 0.0, 0.0, 0.0)


@functools.lru_cache(maxsize=None)
def _channel_case(ny, re, precision, iters, tol):
    m, bcs = _channel_mesh(ny, re)
    return rs.Case(m, bcs, 1.0 / re, _settings(precision, iters, tol, True))


@functools.lru_cache(maxsize=None)
def _step_mesh(a, walls=True):
    m = rs.Mesh.make_backward_facing_step_2d(2 * a, 12 * a, 6 * a, 3 * a, 4.0, 30.0, 1.0, 3.0, 36000.0, 1.0)
    m = m.permuted(np.random.default_rng(7).permutation(m.n_cells()))
    if walls:
        m.compute_wall_distance(device=True)
    return m


STEP_NU = 1.0 / 36000.0
STEP_K = 1.5 * 0.01 ** 2
STEP_OMEGA = STEP_K / (100.0 * STEP_NU)


def _step_settings(precision, iters):
    s = _settings(precision, iters, 0.0, False)
    s.divergence_limit = 1e8
    s.alpha_u, s.alpha_p, s.alpha_k, s.alpha_omega = 0.3, 0.2, 0.4, 0.4
    s.inner_iterations = 300
    s.inner_tolerance = 1e-4
    s.turb_start_iter = 30
    s.turb_update_interval = 2
    return s


@functools.lru_cache(maxsize=2)
def _step_case(a, precision, iters):
    m = _step_mesh(a)
    bcs = rs.FlowBoundaryConditions.bfs_defaults(m, 1.0, STEP_K, STEP_OMEGA)
    return rs.Case(m, bcs, STEP_NU, _step_settings(precision, iters))


@functools.lru_cache(maxsize=2)
def _duct_case(nx, ny, nz, precision, iters):
    m = rs.Mesh.make_square_duct_periodic_3d(nx, ny, nz, 10.0, 2.0, 1.1)
    m = m.permuted(np.random.default_rng(17).permutation(m.n_cells()))
    m.compute_wall_distance(device=True)
    bcs = rs.FlowBoundaryConditions.channel_defaults(m, 0.0, 0.0, 0.0)
    return rs.Case(m, bcs, 1.0 / 300.0, _settings(precision, iters, 0.0, True))


def _observations(which):
    o = rs.ObservationOperator()
    if which == "channel":
        o.add_skin_friction("bottom_wall", rs.Vec3(0.5, 0.0, 0.5), 0.0066, 0.001, 1.0)
        o.add_skin_friction("top_wall", rs.Vec3(0.5, 2.0, 0.5), 0.0066, 0.001, 1.0)
        for y, u in ((0.001, 0.5), (0.01, 5.0), (0.1, 14.0), (0.5, 19.0), (1.0, 21.0)):
            o.add_velocity_profile(rs.Vec3(0.5, y, 0.5), 0, u, 0.5)
    else:
        o.add_velocity_profile(rs.Vec3(3.0, 0.3, 0.0), 0, -0.1, 0.05)
        o.add_skin_friction("bottom_wall_down", rs.Vec3(10.0, 0.0, 0.0), 0.002, 5e-4, 1.0)
        o.add_reattachment_length("bottom_wall_down", 6.0, 0.5)
    return o


@functools.lru_cache(maxsize=None)
def _warm_case(mesh, precision, iters):
    """A case and its converged state (the reference's, stored with the tests)."""
    z = np.load(os.path.join(ROOT, "tests", "golden",
                             "c1_chan550_4x128.npz" if mesh == "channel" else "bfs_perm_1920.npz"))
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "mesh.msh")
        with open(path, "wb") as fh:
            fh.write(z["mesh"].tobytes())
        m = rs.Mesh.load_from_file(path)
    m.wall_dist = np.ascontiguousarray(z["wall_dist"])
    if mesh == "channel":
        bcs = rs.FlowBoundaryConditions.channel_defaults(m, 0.0, 0.0, 0.0)
        s = _settings(precision, iters, 0.0, True)
    else:
        bcs = rs.FlowBoundaryConditions.bfs_defaults(m, 1.0, STEP_K, STEP_OMEGA)
        s = _step_settings(precision, iters)
        s.turb_start_iter = 0
    c = rs.Case(m, bcs, float(z["nu"]), s)
    c.set_observations(_observations(mesh))
    state = {f: np.ascontiguousarray(z["conv_" + f]) for f in FIELDS}
    state["turb_established"] = int(z["conv_turb_established"])
    return c, state


@functools.lru_cache(maxsize=None)
def _forward_model(ny, re, precision, iters, tol):
    m, bcs = _channel_mesh(ny, re)
    ps = rs.InferenceParameterSet.from_indices("six", ACTIVE)
    i = CHANNEL_INIT
    return ps, rs.ForwardModel(m, ps, _observations("channel"), bcs, 1.0 / re, _settings(precision, iters, tol, True),
                               u_init=rs.Vec3(*i["u"]), p_init=i["p"], k_init=i["k"], omega_init=i["omega"])


@functools.lru_cache(maxsize=None)
def _server():
    return rs.Server(max_slots=304, hbm_budget_bytes=4 << 30)


# ---- a call's own inputs -----------------------------------------------------
def _thetas(rng, n, spread):
    c = np.tile(np.asarray(COEFF_DEFAULTS, np.float64), (n, 1))
    c[:, ACTIVE] *= rng.uniform(1.0 - spread, 1.0 + spread, (n, len(ACTIVE)))
    return c


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = dict(kind=kind)
    if kind == "evaluate":
        ps, st["model"] = _forward_model(case["ny"], case["re"], case["precision"], case["iters"], case["tol"])
        base = np.array(ps.pack(rs.SSTCoefficients()))
        st["theta"] = list(base * rng.uniform(0.9, 1.1, len(ACTIVE)))
        return st
    if kind == "wall":
        m = _step_mesh(case["a"], False)
        # another numbering and another scale
        mesh = m.permuted(rng.permutation(m.n_cells()))
        scale = rng.uniform(0.5, 2.0)
        mesh.cell_center, mesh.face_center = mesh.cell_center * scale, mesh.face_center * scale
        st["mesh"] = mesh
        return st
    if kind == "channel":
        c = _channel_case(case["ny"], case["re"], case["precision"], case["iters"], case.get("tol", 0.0))
        st["cases"], st["inits"] = [c] * case["n"], [CHANNEL_INIT] * case["n"]
        st["theta"] = _thetas(rng, case["n"], 0.2)
    elif kind == "warm":
        c, state = _warm_case(case["mesh"], case["precision"], case["iters"])
        st["cases"], st["inits"] = [c] * case["n"], [state] * case["n"]
        st["theta"] = _thetas(rng, case["n"], case["step"])
    elif kind in ("mix", "served"):
        sizes = MIX_NY[case.get("sizes", "small")]
        cs = [_channel_case(ny, re, case["precision"], case["iters"], 0.0) for ny, re in sizes]
        st["cases"] = [cs[i % len(cs)] for i in range(case["n"])]
        st["inits"] = [CHANNEL_INIT] * case["n"]
        st["theta"] = _thetas(rng, case["n"], 0.2)
        if kind == "served":
            st["server"] = _server()
    elif kind == "step":
        st["cases"] = [_step_case(case["a"], case["precision"], case["iters"])]
        st["inits"] = [dict(u=(1.0, 0.0, 0.0), p=0.0, k=STEP_K, omega=STEP_OMEGA)]
        st["theta"] = _thetas(rng, 1, 0.1)
        # the start-up is laminar: another inlet-like start for another seed
        st["inits"][0]["u"] = (float(rng.uniform(0.9, 1.1)), 0.0, 0.0)
    elif kind == "duct":
        st["cases"] = [_duct_case(case["nx"], case["ny"], case["nz"], case["precision"], case["iters"])]
        st["inits"] = [dict(u=(float(rng.uniform(14.0, 16.0)), 0.0, 0.0), p=0.0, k=1e-2, omega=10.0)]
        st["theta"] = _thetas(rng, 1, 0.1)
    return st


def _collect(outs):
    """The states of a batch, one array per mesh size and field (at most four
    sizes), and what the solves report about themselves."""
    groups = {}
    for o in outs:
        groups.setdefault(o.state["U"].shape[0], []).append(o)
    res = {"status": np.array([int(o.status) for o in outs])}
    for cells, os_ in groups.items():
        r = res["cells_%d" % cells] = {}
        r["U"] = np.stack([o.state["U"] for o in os_])
        r["boundary"] = np.stack([np.concatenate([o.state[f].ravel() for f in ("Ub", "pb", "kb", "omegab")])
                                  for o in os_])
        for f in ("p", "k", "omega", "nuT", "F1", "F2", "Pk", "CDkw"):
            r[f] = np.stack([o.state[f] for o in os_])
        if os_[0].predictions is not None:
            r["predictions"] = np.array([o.predictions for o in os_])
            r["log_lik"] = np.array([o.log_lik for o in os_])
    return res


def run(state):
    kind = state["kind"]
    if kind == "evaluate":
        m = state["model"]
        m.clear_cache()   # a new chain: nothing to start from
        r = m.evaluate(state["theta"])
        return {"status": int(r.status), "log_lik": float(r.log_lik), "predictions": np.array(r.predictions),
                "fields": m.last_fields()}
    if kind == "wall":
        state["mesh"].compute_wall_distance(device=True)
        return state["mesh"].wall_dist
    if kind == "served":
        srv, left, done = state["server"], list(range(len(state["cases"]))), {}
        where = {}
        while len(done) < len(state["cases"]):
            while left:
                i = left[0]
                rid = srv.submit(state["cases"][i], state["theta"][i], init=state["inits"][i])
                if rid is None:
                    break
                where[rid] = left.pop(0)
            for rid, out in srv.poll(timeout_ms=20):
                done[where[rid]] = out
        return _collect([done[i] for i in range(len(state["cases"]))])
    return _collect(rs.solve_batch(state["cases"], state["theta"], inits=state["inits"]))


# ---- what a pass cannot do without -------------------------------------------
# Operations per cell and outer iteration: closure, gradients, assembly of the
# momentum, pressure and turbulence systems and corrections (about 900 with
# quadrilateral cells, 1400 with hexahedra), and the inner iterations (about
# 14 in all, 40 operations each).  Bytes: the case's geometry and the start
# state once, the final state once; between iterations a solve can stay on
# the chip.
def _cells(case):
    kind = case["kind"]
    if kind in ("evaluate", "channel"):
        return [4 * case["ny"]] * case.get("n", 1)
    if kind == "warm":
        return [512 if case["mesh"] == "channel" else 1920] * case["n"]
    if kind in ("mix", "served"):
        sizes = MIX_NY[case.get("sizes", "small")]
        return [4 * sizes[i % len(sizes)][0] for i in range(case["n"])]
    if kind == "duct":
        return [case["nx"] * case["ny"] * case["nz"]]
    return [120 * case["a"] ** 2]


def work(case):
    cells = _cells(case)
    if case["kind"] == "wall":
        faces = 2 * 14 * case["a"] + 3 * case["a"]
        return {"bytes": 8 * (4 * cells[0] + 3 * faces), "flops": 8 * cells[0] * faces}
    iters = case["iters"]
    if case.get("tol"):   # stops before its cap
        iters = 3000 if case["precision"] == "mixed" else min(iters, 1000)
    per_cell = 1400 if case["kind"] == "duct" else 900
    geometry = sum({c: 500 * c for c in cells}.values())
    return {"bytes": geometry + sum(2 * 96 * c for c in cells), "flops": (per_cell + 14 * 40) * iters * sum(cells)}


def exact(case, seed):
    """Wall distances have a value of their own.  The fields of a solve stopped
    at an outer-iteration count or at a residual do not: they depend on how far
    each inner Krylov or multigrid solve was taken, and the fixed point itself
    takes tens of thousands of outer iterations."""
    if case["kind"] != "wall":
        return None
    m = prepare(case, seed)["mesh"]
    walls = np.concatenate([faces for _, patch_type, faces in m.patches if patch_type == "wall"])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cc = torch.from_numpy(np.ascontiguousarray(m.cell_center)).to(dev)
    wf = torch.from_numpy(np.ascontiguousarray(m.face_center[walls])).to(dev)
    best = torch.full((cc.shape[0],), float("inf"), dtype=torch.float64, device=dev)
    for j in range(0, wf.shape[0], 64):
        best = torch.minimum(best, ((cc[:, None, :] - wf[None, j:j + 64, :]) ** 2).sum(-1).amin(1))
    return best.sqrt()
