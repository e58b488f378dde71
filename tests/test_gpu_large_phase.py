"""The phase test hook runs on one CTA also for meshes whose solves take the
whole device: their coarsest multigrid level has up to 1024 rows."""
import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.linalg import spsolve

import cases
from rans_sst_py import Case
from test_amg_hierarchy import hierarchy
from test_gpu_parity import _dbg, _pack, _rand_state

pytestmark = pytest.mark.gpu


def test_amg_pcg_phase_on_a_large_mesh():
    """17,280 cells, a coarsest level above the one-CTA form's 32 rows: AMG-PCG on
    the mesh's pressure Laplacian (condition number 1.3e6) to 1e-9.  The true
    residual may be off the recursive one by rounding, 1.1e-16 times the condition
    number in each of some 50 iterations: 1e-8 in all; the error is at most the
    residual times the condition number."""
    m, b, nu, _ = cases.bfs_case(24, 144, 72, 36)
    sizes, _, (rp, col, val) = hierarchy(m, b, -1)
    assert m.n_cells() > 16384 and 32 < sizes[-1] <= 1024
    s = cases.bfs_settings(1, 0.0)
    s.inner_iterations, s.inner_tolerance = 200, 1e-9
    case = Case(m, b, nu, s)
    nC, nI = m.n_cells(), m.n_internal_faces()
    row = np.repeat(np.arange(nC), np.diff(rp))
    off = {(r, c): v for r, c, v in zip(row, col, val) if r != c}
    o, n = m.owner[:nI], m.neighbour[:nI]
    upper = np.array([off[x] for x in zip(o, n)])
    diag = np.zeros(nC)
    diag[row[row == col]] = val[row == col]
    rng = np.random.default_rng(3)
    src = rng.normal(size=nC)
    a = coo_matrix((np.concatenate([diag, upper, upper]),
                    (np.concatenate([np.arange(nC), o, n]), np.concatenate([np.arange(nC), n, o]))))
    exact = spsolve(a.tocsc(), src)
    out = _dbg(case, "amgpcg", _pack(m, _rand_state(m, rng, True),
                                     dict(diag=diag, upper=upper, lower=upper, source=src, x=np.zeros(nC))), nC + 4)
    iterations, final, _, converged = out[nC:]
    assert converged == 1 and final < 1e-9 and iterations < 200
    assert np.linalg.norm(a @ out[:nC] - src) < 1e-8 * np.linalg.norm(src)
    assert cases.rel_l2(out[:nC], exact) < 2e-2
