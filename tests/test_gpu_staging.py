"""Staging of a batch's start states and results (64 MiB a part): several parts,
states and observation outputs that do not fit a part.

With no outer iterations a solve returns the state that it was given, so what
comes back is compared bit for bit with what went up."""
import ctypes as C

import numpy as np
import pytest

import cases
from rans_sst_py import Case, FlowBoundaryConditions, Mesh, solve_batch
from rans_sst_py._lib import (BND_FIELDS, CELL_FIELDS, STATE_ORDER, BtmHistory, BtmInit, BtmObservable, BtmState, check,
                              dptr, lib, mesh_struct, new_state, state_struct)

pytestmark = pytest.mark.gpu

COEFF = np.array(cases.COEFF_DEFAULTS)
PART_WORDS = (64 << 20) // 8


def _random_state(n_cells, n_bnd, rng):
    st = new_state(n_cells, n_bnd)
    for f in ("U", "Ub", "p", "pb", "CDkw"):
        st[f] = rng.normal(size=st[f].shape)
    for f in CELL_FIELDS[1:7] + BND_FIELDS[1:]:
        st[f] = rng.uniform(0.1, 1.0, st[f].shape)
    st["turb_established"] = int(rng.integers(0, 2))
    return st


def _words(n_cells, n_bnd):
    return 11 * n_cells + 6 * n_bnd


def _assert_same(out, st, tag):
    for f in STATE_ORDER:
        assert np.array_equal(out[f], st[f]), (tag, f)
    assert out["turb_established"] == st["turb_established"], tag


def test_several_parts():
    """Two meshes in turn, more than two parts of start states and of results;
    some instances share a state."""
    rng = np.random.default_rng(1)
    made = []
    for ny in (512, 24):
        m, b, nu, _ = cases.periodic_channel(ny, 180.0)
        made.append(Case(m, b, nu, cases.channel_settings(0, 0.0)))
    one = _words(made[0].n_cells, made[0].n_bnd)
    n = 2 * (int(2.2 * PART_WORDS / one) + 1)
    which = [made[i % 2] for i in range(n)]
    states = [_random_state(c.n_cells, c.n_bnd, rng) for c in which]
    for i in range(10, n, 50):   # the state of an instance in the same part, or one long past
        states[i] = states[i - 2] if i % 100 == 10 else states[0]
    outs = solve_batch(which, np.tile(COEFF, (n, 1)), inits=states)
    for i, o in enumerate(outs):
        assert o.iterations_run == 0
        _assert_same(o.state, states[i], i)


def test_state_larger_than_a_part():
    """A state that goes array by array, beside one that is staged."""
    rng = np.random.default_rng(2)
    m = Mesh.make_channel_periodic_geometric(200, 3850, 10.0, 1.0, 1.001)
    m.wall_dist = rng.uniform(0.1, 1.0, m.n_cells())
    assert _words(m.n_cells(), m.n_boundary_faces()) > PART_WORDS
    big = Case(m, FlowBoundaryConditions.channel_defaults(m, 0.0, 0.0, 0.0), 1.0 / 300.0,
               cases.channel_settings(0, 0.0))
    m, b, nu, _ = cases.periodic_channel(24, 180.0)
    small = Case(m, b, nu, cases.channel_settings(0, 0.0))
    for order in ([big, small], [small, big]):
        states = [_random_state(c.n_cells, c.n_bnd, rng) for c in order]
        outs = solve_batch(order, np.tile(COEFF, (2, 1)), inits=states)
        for q in range(2):
            _assert_same(outs[q].state, states[q], q)


def test_observation_outputs_larger_than_a_part():
    """8.4 million velocity observables on 64 cells: the outputs alone are larger
    than a part; an instance beside it is staged."""
    rng = np.random.default_rng(3)
    m, b, nu, _ = cases.periodic_channel(16, 180.0)
    many, few = (Case(m, b, nu, cases.channel_settings(0, 0.0)) for _ in range(2))
    for case, n in ((many, PART_WORDS + 40), (few, 5)):
        obs = np.zeros(n, np.dtype(BtmObservable))
        obs["type"], obs["component"], obs["sigma_obs"] = 2, np.arange(n) % 2, 1.0
        obs["location"] = m.cell_center[np.arange(n) % m.n_cells()]
        ms, keep = mesh_struct(m)
        check(lib().btm_case_set_observations(case.h, C.byref(ms), n, obs.ctypes.data_as(C.POINTER(BtmObservable))))
        case.n_obs = n
        del obs
    for order in ([many, few], [few, many]):
        states = [_random_state(c.n_cells, c.n_bnd, rng) for c in order]
        outs = solve_batch(order, np.tile(COEFF, (2, 1)), inits=states)
        for c, o, st in zip(order, outs, states):
            k = np.arange(c.n_obs)
            want = st["U"][k % m.n_cells(), k % 2]
            assert np.array_equal(o.predictions, want)
            _assert_same(o.state, st, c.n_obs)
            # the device adds the terms one after the other: off by n rounding errors at most
            assert abs(o.log_lik - (-0.5 * want * want).sum()) <= c.n_obs * 1.2e-16 * abs(o.log_lik)
