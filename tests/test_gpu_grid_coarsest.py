"""Grid meshes whose coarsest multigrid level is swept, not inverted: coarsening
never joins separate pieces, so a mesh of more than 1024 of them ends on a
level of more than 1024 rows."""
import numpy as np
import pytest

import cases
from rans_sst_py import Case, FlowBoundaryConditions, Mesh, solve
from test_amg_hierarchy import hierarchy

COEFF = np.array(cases.COEFF_DEFAULTS)
NU, K_IN = 1.0 / 36000.0, 1.5 * 0.01 ** 2
OMEGA_IN = K_IN / (100.0 * NU)


def separate_steps(count: int, seed: int = 5) -> Mesh:
    """`count` backward-facing steps of 16 cells, each at its own scale, as one
    mesh with shuffled cell ids; a patch holds the faces of all of them."""
    one = Mesh.make_backward_facing_step_2d(2, 4, 2, 1, 4.0, 30.0, 1.0, 3.0, 36000.0, 1.0)
    one.compute_wall_distance()
    nC, nF, nI = one.n_cells(), one.n_faces(), one.n_internal
    rng = np.random.default_rng(seed)
    scale = rng.uniform(0.5, 2.0, count)
    # internal faces of all pieces, then the boundary faces patch by patch
    piece = np.repeat(np.arange(count), nI)
    face = np.tile(np.arange(nI), count)
    patches = []
    for name, kind, faces in one.patches:
        patches.append((name, kind, (len(face) + np.arange(count * len(faces))).astype(np.int32)))
        piece = np.concatenate([piece, np.repeat(np.arange(count), len(faces))])
        face = np.concatenate([face, np.tile(faces, count)])
    assert len(face) == count * nF
    m, s = Mesh(), scale[piece]
    m.owner = (one.owner[face] + nC * piece).astype(np.int32)
    nb = one.neighbour[face]
    m.neighbour = np.where(nb >= 0, nb + nC * piece, nb).astype(np.int32)
    m.face_patch, m.face_weight = one.face_patch[face], one.face_weight[face].copy()
    m.face_normal = one.face_normal[face].copy()
    m.face_center, m.face_d = one.face_center[face] * s[:, None], one.face_d[face] * s[:, None]
    m.face_area, m.face_delta = one.face_area[face] * s, one.face_delta[face] * s
    cells = np.repeat(scale, nC)
    m.cell_center = np.tile(one.cell_center, (count, 1)) * cells[:, None]
    m.cell_volume = np.tile(one.cell_volume, count) * cells ** 2
    m.wall_dist = np.tile(one.wall_dist, count) * cells
    m.patches, m.n_internal = patches, count * nI
    # each cell's faces, ascending
    of = np.concatenate([m.owner, m.neighbour[m.neighbour >= 0]])
    ids = np.concatenate([np.arange(len(face)), np.flatnonzero(m.neighbour >= 0)])
    order = np.lexsort((ids, of))
    m.cell_faces = ids[order].astype(np.int32)
    m.cell_face_offset = np.concatenate([[0], np.cumsum(np.bincount(of, minlength=count * nC))]).astype(np.int32)
    return m.permuted(rng.permutation(count * nC))


def _case():
    m = separate_steps(1100)
    return m, FlowBoundaryConditions.bfs_defaults(m, 1.0, K_IN, OMEGA_IN), dict(u=(1.0, 0.0, 0.0), p=0.0, k=K_IN,
                                                                              omega=OMEGA_IN)


def test_coarsest_level_is_too_large_to_invert():
    m, b, _ = _case()
    sizes = hierarchy(m, b, -1)[0]
    assert m.n_cells() > 16384 and len(sizes) > 1 and sizes[-1] > 1024


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_swept_coarsest_level(precision, oracle):
    """One cold iteration, inner solves to 1e-10, twice: the same bits, and in
    FP64 the oracle's state to the inner tolerance times the conditioning of the
    systems (1e-7).  The pieces are small, so the pressure solve needs few CG
    iterations as long as the coarsest level sees its own right-hand side."""
    m, b, ini = _case()
    s = cases.bfs_settings(1, 0.0)
    s.inner_tolerance, s.inner_iterations, s.precision = 1e-10, 1000, precision
    c = Case(m, b, NU, s)
    first, again = solve(c, COEFF, 0, ini), solve(c, COEFF, 0, ini)
    for f in ("U", "p", "k", "omega"):
        assert np.all(np.isfinite(first.state[f])), f
        assert np.array_equal(first.state[f], again.state[f]), f
    assert list(first.inner_split) == list(again.inner_split)
    if precision == "fp64":
        ref, _ = oracle.solve(m, b, NU, s, COEFF, 0, **ini)
        for f in ("U", "p"):
            assert cases.rel_l2(first.state[f], ref[f]) < 1e-7, f
        assert first.inner_split[1] < 200
