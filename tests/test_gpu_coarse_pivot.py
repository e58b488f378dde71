"""A coarsest multigrid level with a vanishing pivot: its rows are passed over."""
import numpy as np
import pytest
import scipy.sparse as sp
from scipy.sparse.linalg import spsolve

import cases
from rans_sst_py import Case
from test_amg_hierarchy import hierarchy
from test_gpu_parity import _dbg, _pack, _rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dead", [[0], [5], [17], [3, 11]])
def test_decoupled_empty_rows(dead):
    """The cells behind `dead` coarsest rows have no matrix entries and no source:
    AMG-PCG to 1e-10 solves the others (condition number below 1e6: to 1e-4) and
    leaves them at zero."""
    m, b, nu, _ = cases.bfs_case()
    sizes, maps, (rp, col, val) = hierarchy(m, b, -1)
    top = maps[0]
    for k in maps[1:]:
        top = k[top]
    assert sizes[-1] == 18 == top.max() + 1
    live = ~np.isin(top, dead)
    a = sp.csr_matrix((val, col, rp))
    nC, nI = m.n_cells(), m.n_internal
    o, n = m.owner[:nI], m.neighbour[:nI]
    upper = np.asarray(a[o, n]).ravel() * (live[o] & live[n])
    diag = a.diagonal() * live
    rng = np.random.default_rng(6)
    src = rng.normal(size=nC) * live
    s = cases.bfs_settings(1, 0.0)
    s.amg_order, s.inner_iterations, s.inner_tolerance = "multicolour", 300, 1e-10
    out = _dbg(Case(m, b, nu, s), "amgpcg", _pack(m, _rand_state(m, rng, True),
                                                  dict(diag=diag, upper=upper, lower=upper, source=src,
                                                       x=np.zeros(nC))), nC + 4)
    assert out[nC + 3] == 1
    k = np.flatnonzero(live)
    sub = (sp.diags(diag) + sp.coo_matrix((np.concatenate([upper, upper]),
                                           (np.concatenate([o, n]), np.concatenate([n, o]))), (nC, nC))).tocsc()[k][:, k]
    assert cases.rel_l2(out[:nC][k], spsolve(sub, src[k])) < 1e-4
    assert np.all(out[:nC][~live] == 0.0)
