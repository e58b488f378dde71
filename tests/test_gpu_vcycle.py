"""One V-cycle of the grid's multigrid (device_units.cu: unit_vcycle) against the
same cycle in numpy, on hierarchies that reach its branches: rows of more than 8
entries, aggregates of more than 4 members, and a coarsest level that is
inverted by the whole grid, inverted and applied by one thread a row, or swept."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import cases
from rans_sst_py import FlowBoundaryConditions, Mesh
from test_amg_hierarchy import hierarchy
from test_gpu_device_units import _d, units  # noqa: F401 (fixture)
from test_gpu_grid_coarsest import _case as separate_steps_case

WEIGHT, COARSE_SWEEPS = 0.7, 50


def _colours(a):
    """Greedy in row order: no two coupled rows of a colour."""
    col = np.full(a.shape[0], -1)
    for i in range(a.shape[0]):
        used = set(col[a.indices[a.indptr[i]:a.indptr[i + 1]]])
        k = 0
        while k in used:
            k += 1
        col[i] = k
    order = np.argsort(col, kind="stable").astype(np.int32)
    return np.concatenate([[0], np.cumsum(np.bincount(col))]).astype(np.int32), order


class Level:
    def __init__(self, a, agg=None):
        a.sort_indices()
        self.a, self.n, self.agg = a, a.shape[0], agg
        self.off, self.rows = _colours(a)
        self.rd = 1.0 / a.diagonal()
        if agg is not None:
            self.p = sp.csr_matrix((np.ones(self.n), (np.arange(self.n), agg)))
            self.agg_mem = np.argsort(agg, kind="stable").astype(np.int32)
            self.agg_off = np.concatenate([[0], np.cumsum(np.bincount(agg))]).astype(np.int32)
        rest = (a - sp.diags(a.diagonal())).tocsr()
        self.parts = [(r, rest[r]) for r in np.split(self.rows, self.off[1:-1])]

    def sweep(self, x, b, reverse):
        for r, m in (reversed(self.parts) if reverse else self.parts):
            x[r] = (b[r] - m @ x) * self.rd[r]


def levels(m, b, grid):
    """The library's hierarchy of the mesh, values by Galerkin products."""
    _, maps, (rp, col, val) = hierarchy(m, b, grid)
    out, a = [], sp.csr_matrix((val, col, rp))
    for agg in maps + [None]:
        out.append(Level(a.copy(), agg))
        if agg is not None:
            a = (out[-1].p.T @ a @ out[-1].p).tocsr()
    return out


def vcycle(lev, b, inverse):
    x, rhs = [np.zeros(l.n) for l in lev], [b] + [None] * (len(lev) - 1)

    def jacobi(l, b, x):
        return x + WEIGHT * l.rd * (b - l.a @ x)

    for q, l in enumerate(lev[:-1]):
        if q == 0:
            l.sweep(x[0], b, False)
            l.sweep(x[0], b, False)
        else:
            x[q] = jacobi(l, rhs[q], WEIGHT * l.rd * rhs[q])
        rhs[q + 1] = l.p.T @ (rhs[q] - l.a @ x[q])
    if inverse is not None:
        x[-1] = inverse @ rhs[-1]
    else:
        for s in range(COARSE_SWEEPS):
            lev[-1].sweep(x[-1], rhs[-1], s % 2 == 1)
    for q in range(len(lev) - 2, -1, -1):
        l = lev[q]
        x[q] = x[q] + l.p @ x[q + 1]
        if q == 0:
            l.sweep(x[0], b, True)
            l.sweep(x[0], b, True)
        else:
            x[q] = jacobi(l, rhs[q], jacobi(l, rhs[q], x[q]))
    return x[0]


def device_vcycle(units, m, lev, b, inverse, fp32, blocks):  # noqa: F811
    ints, places, vals, value_at, rds = [], [], [], [], []
    at = [0, 0]

    def put(a):
        ints.append(np.asarray(a, np.int32))
        at[0] += len(ints[-1])
        return at[0] - len(ints[-1])

    for l in lev:
        q = [l.n, len(l.off) - 1, put(l.a.indptr), put(l.a.indices)]
        q += [put(l.agg), put(l.agg_off), put(l.agg_mem)] if l.agg is not None else [0, 0, 0]
        places += q + [put(l.off), put(l.rows), at[1]]
        vals.append(l.a.data)
        at[1] += len(l.a.data)
        rds.append(l.rd)
    # level 0 as diag | upper | lower, rows by position in ascending face order
    nC, nI = m.n_cells(), m.n_internal
    o, nb = m.owner[:nI], m.neighbour[:nI]
    upper = np.asarray(lev[0].a[o, nb]).ravel()
    cell, face = np.concatenate([o, nb]), np.tile(np.arange(nI), 2)
    order = np.lexsort((face, cell))
    cell, face, own = cell[order], face[order], np.repeat([True, False], nI)[order]
    count = np.bincount(cell, minlength=nC)
    pos = np.arange(2 * nI) - np.repeat(np.cumsum(count) - count, count)
    width = int(count.max())
    ent, col = np.zeros((width, nC), np.int32), np.full((width, nC), -1, np.int32)
    ent[pos, cell] = np.where(own, nC + face, nC + nI + face)
    col[pos, cell] = np.where(own, nb[face], o[face])
    sizes = np.array([len(lev), inverse is not None, nC, width] + places + [put(ent.ravel()), put(col.ravel())], np.int64)
    ints, vals, rds = np.concatenate(ints), np.concatenate(vals), np.concatenate(rds)
    matrix = np.concatenate([lev[0].a.diagonal(), upper, upper])
    inv = np.ascontiguousarray(inverse if inverse is not None else np.zeros((1, 1)))
    x = np.empty(nC)
    i64, f64 = (lambda a: a.ctypes.data_as(C.POINTER(C.c_int64))), C.c_int64
    assert units.unit_vcycle(fp32, blocks, i64(sizes), ints.ctypes.data_as(C.POINTER(C.c_int32)), f64(len(ints)),
                             _d(vals), f64(len(vals)), _d(matrix), f64(len(matrix)), _d(rds), _d(inv), f64(inv.size),
                             _d(b), _d(x)) == 0
    return x


def _step():
    m, b, _, _ = cases.bfs_case(24, 144, 72, 36)
    return m, b, levels(m, b, 1), True


def _duct():
    m = Mesh.make_square_duct_periodic_3d(20, 30, 30, 10.0, 2.0, 1.1)
    m = m.permuted(np.random.default_rng(17).permutation(m.n_cells()))
    b = FlowBoundaryConditions.channel_defaults(m, 0.0, 0.0, 0.0)
    return m, b, levels(m, b, 1), True


def _pieces():
    m, b, _ = separate_steps_case()
    return m, b, levels(m, b, 1), False


def _small_coarsest():
    m, b, _, _ = cases.bfs_case()
    return m, b, levels(m, b, 0), True


def _one_level():
    m, b, _, _ = cases.bfs_case()
    lev = levels(m, b, 0)[:1]
    lev[0].agg = None
    return m, b, lev, False


MESHES = {"step, inverted by the grid": _step, "duct, wide rows": _duct, "pieces, swept": _pieces,
          "small, inverted by one thread a row": _small_coarsest, "one level, swept": _one_level}


@pytest.fixture(scope="module", params=sorted(MESHES))
def hier(request):
    m, b, lev, direct = MESHES[request.param]()
    return request.param, m, lev, np.linalg.inv(lev[-1].a.toarray()) if direct else None


def test_hierarchies_reach_the_branches(hier):
    name, m, lev, inverse = hier
    n = lev[-1].n
    if name.startswith("duct"):
        assert max(np.diff(l.a.indptr).max() for l in lev[1:]) > 8
        assert max(np.bincount(l.agg).max() for l in lev[:-1]) > 4
    assert {"step, inverted by the grid": 32 < n <= 1024, "duct, wide rows": 32 < n <= 1024, "pieces, swept": n > 1024,
            "small, inverted by one thread a row": 1 < n <= 32, "one level, swept": len(lev) == 1}[name]


@pytest.mark.gpu
@pytest.mark.parametrize("fp32", [0, 1])
def test_vcycle(units, hier, fp32):  # noqa: F811
    """The order of a row's terms is the library's, the rest rounds alike up to a
    few hundred operations a value: 1e-12 in FP64, 1e-4 in FP32.  The same bits for
    any number of CTAs."""
    _, m, lev, inverse = hier
    rhs = np.random.default_rng(4).normal(size=lev[0].n)
    want = vcycle(lev, rhs, inverse)
    first = device_vcycle(units, m, lev, rhs, inverse, fp32, 100)
    assert cases.rel_l2(first, want) < (1e-4 if fp32 else 1e-12)
    for blocks in (100, 37, 152):
        assert np.array_equal(device_vcycle(units, m, lev, rhs, inverse, fp32, blocks), first), blocks
