"""Kernels whose paths depend on sizes, at the sizes where they can go wrong.

  * wall distance: FP32 search with FP64 measurement against the numpy brute
    force, bit for bit, at the edges of the shared-memory tile (1024 faces), of
    the candidate list (8 faces at the same distance) and of the warp, with
    coordinates far from the origin and beyond the FP32 range;
  * staging of a batch: states that several instances start from and results
    of meshes of uneven size equal the same solves one by one, bit for bit;
  * reference-order AMG sweeps (packed rows, one warp, one CTA) on meshes at the
    edges of their paths, against the oracle;
  * dense coarsest inverse on the grid: a pressure correction to 1e-10 takes
    about as many CG iterations as with an exact coarse solve.
"""
import ctypes as C

import numpy as np
import pytest

import cases
from rans_sst_py import Case, FlowBoundaryConditions, Mesh, solve, solve_batch
from rans_sst_py._forward import _init_struct
from rans_sst_py._lib import BtmHistory, check, dptr, lib, new_state, state_struct

pytestmark = pytest.mark.gpu

COEFF = np.array(cases.COEFF_DEFAULTS)
FIELDS = ("U", "p", "k", "omega", "nuT", "F1", "F2", "Pk", "CDkw", "Ub", "pb", "kb", "omegab")


def _device_distance(cc, wp):
    L = lib()
    L.btm_wall_distance.argtypes = [C.c_int32, C.POINTER(C.c_double), C.c_int32, C.POINTER(C.c_double),
                                    C.POINTER(C.c_double)]
    out = np.empty(len(cc))
    check(L.btm_wall_distance(len(cc), dptr(cc), len(wp), dptr(wp), dptr(out)))
    return out


@pytest.mark.parametrize("n_wall", [1, 7, 8, 9, 1023, 1024, 1025, 2500])
@pytest.mark.parametrize("n_cells", [1, 33, 257])
@pytest.mark.parametrize("kind", ["random", "offset", "equidistant", "near", "huge", "tiny"])
def test_wall_distance_bits(n_wall, n_cells, kind):
    rng = np.random.default_rng(n_wall * 1000 + n_cells)
    wp, cc = rng.uniform(-1, 1, (n_wall, 3)), rng.uniform(-1, 1, (n_cells, 3))
    if kind == "offset":
        wp, cc = wp + 1e6, cc + 1e6
    elif kind == "equidistant":   # every face at one distance of every cell on the axis
        a = np.linspace(0, 2 * np.pi, n_wall, endpoint=False)
        wp, cc = np.stack([np.cos(a), np.sin(a), 0 * a], 1), cc * np.array([0, 0, 1.0])
    elif kind == "near":
        cc = wp[rng.integers(0, n_wall, n_cells)] + 1e-9 * cc
    elif kind == "huge":
        wp, cc = wp * 1e30, cc * 1e30
    elif kind == "tiny":
        wp, cc = wp * 1e-30, cc * 1e-30
    wp, cc = np.ascontiguousarray(wp), np.ascontiguousarray(cc)
    d = cc[:, None, :] - wp[None, :, :]
    host = np.sqrt((d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]).min(1)
    assert np.array_equal(_device_distance(cc, wp), host)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_staging_equals_single_solves(precision):
    """Cold, host-warm (shared and own states) and device-warm instances of
    two meshes in one call."""
    made = []
    for m, b, nu, ini in (cases.periodic_channel(16, 120.0), cases.bfs_case()):
        s = cases.channel_settings(6, 0.0) if nu > 1e-3 else cases.bfs_settings(6, 0.0)
        s.precision = precision
        made.append((Case(m, b, nu, s), ini))
    first = [solve(c, COEFF, 0, ini) for c, ini in made]
    warm = [o.state for o in first]
    own = {k: (v * (1.0 + 1e-6) if isinstance(v, np.ndarray) else v) for k, v in warm[0].items()}
    plan = [(0, made[0][1]), (1, warm[1]), (0, warm[0]), (1, made[1][1]), (0, warm[0]), (0, own), (1, warm[1])]
    th = [COEFF * (1.0 + 0.01 * q) for q in range(len(plan))]
    batch = solve_batch([made[k][0] for k, _ in plan], th, inits=[i for _, i in plan])
    for q, (k, ini) in enumerate(plan):
        alone = solve(made[k][0], th[q], 0, ini)
        for f in FIELDS:
            assert np.array_equal(batch[q].state[f], alone.state[f]), (q, f)
        assert batch[q].iterations_run == alone.iterations_run
        assert batch[q].inner_iterations == alone.inner_iterations
        assert list(batch[q].last_residual) == list(alone.last_residual)
        assert batch[q].state["turb_established"] == alone.state["turb_established"]


@pytest.mark.parametrize("a", [12, 13, 14])
def test_grid_pressure_solve(a, oracle):
    """One cold iteration on meshes just above the one-CTA size (17,280 to
    23,520 cells; coarsest levels of different sizes modulo the panel width),
    inner solves to 1e-10, against the oracle: they agree to the inner
    tolerance times the conditioning of the systems (1e-7)."""
    m, b, nu, ini = cases.bfs_case(2 * a, 12 * a, 6 * a, 3 * a)
    s = cases.bfs_settings(1, 0.0)
    s.inner_tolerance = 1e-10
    s.inner_iterations = 1000
    out = solve(Case(m, b, nu, s), COEFF, 0, ini)
    ref, _ = oracle.solve(m, b, nu, s, COEFF, 0, **ini)
    for f in ("U", "p"):
        assert cases.rel_l2(out.state[f], ref[f]) < 1e-7, f
    assert out.inner_split[1] < 200


def _permuted_duct():
    m = Mesh.make_square_duct_periodic_3d(3, 8, 8, 10.0, 2.0, 1.2)
    m = m.permuted(np.random.default_rng(3).permutation(m.n_cells()))
    m.compute_wall_distance()
    b = FlowBoundaryConditions.channel_defaults(m, 0.0, 0.0, 0.0)
    return m, b, 1.0 / 150.0, dict(u=(15.0, 0.0, 0.0), p=0.0, k=1e-2, omega=10.0)


REFERENCE_AMG_MESHES = {
    "64 cells, all levels on one warp": lambda: cases.periodic_channel(16, 120.0),
    "72 cells, one level above the warp's": lambda: cases.periodic_channel(18, 120.0),
    "more than 32 wavefronts": lambda: cases.periodic_channel(64, 180.0),
    "hexahedra, level 0 from its CSR rows": _permuted_duct,
    "3,597 cells, wide coarse rows, long wavefronts": lambda: cases.bfs_case(11, 66, 33, 16),
}


@pytest.mark.parametrize("momentum", ["BiCGSTAB", "AMG"])
@pytest.mark.parametrize("name", sorted(REFERENCE_AMG_MESHES))
def test_reference_amg_sweeps(name, momentum, oracle):
    """Two cold iterations with the reference-order AMG (also as the momentum
    solver, where the velocity gradients are still needed), inner solves to
    1e-11, against the oracle: they agree to the inner tolerance times the
    conditioning of the systems (1e-8)."""
    m, b, nu, ini = REFERENCE_AMG_MESHES[name]()
    s = cases.channel_settings(2, 0.0) if nu > 1e-3 else cases.bfs_settings(2, 0.0)
    s.amg_order = "reference"
    s.momentum_solver = momentum
    s.inner_tolerance, s.inner_iterations = 1e-11, 400
    # (the allocation-free call: the launch shape by rule, no tuning probe)
    case, state, hist = Case(m, b, nu, s), new_state(m.n_cells(), m.n_boundary_faces()), BtmHistory()
    st, start = state_struct(state), _init_struct(ini, [])
    check(lib().btm_solve_noalloc(case.h, dptr(COEFF), 0, C.byref(start), C.byref(st), C.byref(hist)))
    ref, _ = oracle.solve(m, b, nu, s, COEFF, 0, **ini)
    for f in ("U", "k", "omega"):
        assert cases.rel_l2(state[f], ref[f]) < 1e-8, f
