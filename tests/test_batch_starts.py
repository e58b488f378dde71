"""The start of every instance of solve_batch is its own, whatever kind of
sequence the starts come in (no GPU: the library call is replaced by a recorder)."""
import ctypes as C

import numpy as np
import pytest

import rans_sst_py._forward as fwd
from rans_sst_py._lib import STATE_ORDER, new_state

N_CELLS, N_BND = 6, 4


class _Case:
    n_cells, n_bnd, n_obs = N_CELLS, N_BND, 0
    h = C.c_void_p(1)


class _Lazy:
    """A sequence that makes its items on access."""

    def __init__(self, n, make):
        self._n, self._make = n, make

    def __len__(self):
        return self._n

    def __getitem__(self, i):
        return self._make(i)


def _state(i):
    st = new_state(N_CELLS, N_BND)
    for q, f in enumerate(STATE_ORDER):
        st[f][:] = 100.0 * i + q
    st["turb_established"] = i % 2
    return st


def _value(ini):
    """What the library would start from: (mode, first entries, flag)."""
    if ini.mode != 1:
        return ini.mode, (ini.u[0], ini.p, ini.k, ini.omega), 0
    w = ini.warm.contents
    return ini.mode, tuple(getattr(w, f)[0] for f in STATE_ORDER), w.turb_established


def _starts(monkeypatch, n, inits):
    seen = {}

    class Library:
        @staticmethod
        def btm_solve_batch(n, handles, coeffs, variants, ini, outs, hists):
            seen["values"] = [_value(ini[q]) for q in range(n)]
            seen["warm"] = [C.addressof(ini[q].warm.contents) if ini[q].mode == 1 else 0 for q in range(n)]
            return 0

    monkeypatch.setattr(fwd, "lib", lambda: Library)
    fwd.solve_batch([_Case()] * n, np.ones((n, 11)), inits=inits)
    return seen


def _cold(i):
    return dict(u=(1.0 + i, 0.0, 0.0), p=2.0 * i, k=3.0 + i, omega=4.0 + i)


class _Dict(dict):   # instances can be freed and their addresses used again, like any object's
    pass


KINDS = {
    "cold made on access": lambda n: _Lazy(n, lambda i: _Dict(_cold(i))),
    "states made on access": lambda n: _Lazy(n, lambda i: _Dict(_state(i))),
    "both made on access": lambda n: _Lazy(n, lambda i: _state(i) if i % 3 else _cold(i)),
    "a list of both": lambda n: [_state(i) if i % 3 else _cold(i) for i in range(n)],
}


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_every_instance_gets_its_own_start(monkeypatch, kind):
    n = 60
    inits = KINDS[kind](n)
    got = _starts(monkeypatch, n, inits)["values"]
    for i in range(n):
        start = inits[i]
        if "U" in start:
            want = (1, tuple(100.0 * i + q for q in range(len(STATE_ORDER))), i % 2)
        else:
            want = (0, (1.0 + i, 2.0 * i, 3.0 + i, 4.0 + i), 0)
        assert got[i] == want, i


def test_one_object_filled_anew(monkeypatch):
    """The same dict for every instance, with other contents at each access."""
    one = {}

    def fill(i):
        one.clear()
        one.update(_state(i) if i % 2 else _cold(i))
        return one

    got = _starts(monkeypatch, 20, _Lazy(20, fill))["values"]
    for i in range(20):
        assert got[i][0] == i % 2 and got[i][1][0] == (100.0 * i if i % 2 else 1.0 + i), i


def test_instances_of_one_state_share_it(monkeypatch):
    """The library moves a state to the device once for all its instances."""
    a, b = _state(1), _state(2)
    seen = _starts(monkeypatch, 5, [a, b, a, dict(a), dict(a, turb_established=0)])
    w = seen["warm"]
    assert w[0] == w[2] == w[3] and len({w[0], w[1], w[4]}) == 3
    assert [v[2] for v in seen["values"]] == [1, 0, 1, 1, 0]
    assert _starts(monkeypatch, 2, ["device", None])["values"] == [(2, (0.0, 0.0, 0.0, 0.0), 0),
                                                                  (0, (1.0, 0.0, 1e-4, 1.0), 0)]
