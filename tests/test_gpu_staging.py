"""Staging of a batch's start states and results (64 MiB a part):
observation outputs that do not fit a part.

With no outer iterations a solve returns the state that it was given, so what
comes back is compared bit for bit with what went up."""
import ctypes as C

import numpy as np
import pytest

import cases
from rans_sst_py import Case, solve_batch
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


def _assert_same(out, st, tag):
    for f in STATE_ORDER:
        assert np.array_equal(out[f], st[f]), (tag, f)
    assert out["turb_established"] == st["turb_established"], tag


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
