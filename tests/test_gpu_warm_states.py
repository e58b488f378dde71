"""Warm start states through the C interface: what a state must hold, and one
state for meshes of different sizes in one call."""
import ctypes as C

import numpy as np
import pytest

import cases
from rans_sst_py import Case, solve
from rans_sst_py._lib import BtmHistory, BtmInit, BtmState, check, dptr, lib, new_state, state_struct

pytestmark = pytest.mark.gpu

COEFF = np.array(cases.COEFF_DEFAULTS)
ERR_ARG = -1


def _channel(ny):
    m, b, nu, ini = cases.periodic_channel(ny, 120.0)
    s = cases.channel_settings(5, 0.0)
    s.turb_start_iter = 0
    return Case(m, b, nu, s), ini


def _solve(cs, warm):
    """One call for the cases `cs`, all started from the struct `warm`."""
    n = len(cs)
    inits = (BtmInit * n)()
    for q in range(n):
        inits[q].mode, inits[q].warm = 1, C.pointer(warm)
    outs = [new_state(c.n_cells, c.n_bnd) for c in cs]
    arr = (BtmState * n)(*[state_struct(o) for o in outs])
    handles = (C.c_void_p * n)(*[c.h.value for c in cs])
    th = np.tile(COEFF, (n, 1))
    status = lib().btm_solve_batch(n, handles, dptr(th), None, inits, arr, (BtmHistory * n)())
    return status, outs


def test_incomplete_warm_state_is_refused():
    case, ini = _channel(16)
    state = solve(case, COEFF, 0, ini).state
    want = _solve([case], state_struct(state))[1][0]
    for f in ("U", "p", "k", "omega", "Ub", "pb", "kb", "omegab"):
        warm = state_struct(state)
        setattr(warm, f, None)
        assert _solve([case], warm)[0] == ERR_ARG, f
    assert _solve([case], state_struct(state))[0] == 0
    # the closure fields are optional: each solve forms them anew, and this one
    # does so in its first iteration
    warm = state_struct(state)
    for f in ("nuT", "F1", "F2", "Pk", "CDkw"):
        setattr(warm, f, None)
    status, (out,) = _solve([case], warm)
    assert status == 0
    for f in ("U", "p", "k", "omega", "nuT"):
        assert np.array_equal(out[f], want[f]), f


def test_one_state_for_meshes_of_two_sizes():
    """The first cells and faces of a state of the larger mesh start the smaller one."""
    (small, _), (large, ini) = _channel(16), _channel(24)
    state = solve(large, COEFF, 0, ini).state
    for order in ([small, large], [large, small], [small, large, small]):
        status, outs = _solve(order, state_struct(state))
        assert status == 0
        for c, o in zip(order, outs):
            alone = _solve([c], state_struct(state))[1][0]
            for f in ("U", "p", "k", "omega", "Ub"):
                assert np.array_equal(o[f], alone[f]), f
