"""A case with an injection target and observations, attached in either order."""
import numpy as np
import pytest

import cases
from rans_sst_py import Case, solve

pytestmark = pytest.mark.gpu

COEFF = np.array(cases.COEFF_DEFAULTS)


def test_observations_leave_the_injection_target():
    """Attaching and detaching observations does not touch the target: the same
    bits as with the observations attached first, also after other cases have
    taken device memory."""
    m, b, nu, ini = cases.periodic_channel(32, 180.0)
    s = cases.channel_settings(30, 0.0)
    target = cases.injection_target(m)
    first = Case(m, b, nu, s)
    first.set_observations(cases.channel_operator())
    first.set_target_anisotropy(target)
    want = solve(first, COEFF, 0, ini)
    case = Case(m, b, nu, s)
    case.set_target_anisotropy(target)
    for _ in range(2):
        case.set_observations(cases.channel_operator())
        others = [Case(m, b, nu, s) for _ in range(3)]
        for o in others:
            o.set_target_anisotropy(-target)
        got = solve(case, COEFF, 0, ini)
        for f in ("U", "p", "k", "omega", "nuT"):
            assert np.array_equal(got.state[f], want.state[f]), f
        assert np.array_equal(got.predictions, want.predictions) and got.log_lik == want.log_lik
        case.set_observations(None)
        got = solve(case, COEFF, 0, ini)
        assert np.array_equal(got.state["U"], want.state["U"])
        for o in others:
            o.close()
    plain = Case(m, b, nu, s)
    assert not np.array_equal(solve(plain, COEFF, 0, ini).state["U"], want.state["U"])
    # taken away and set again
    case.set_target_anisotropy(None)
    case.set_target_anisotropy(target)
    assert np.array_equal(solve(case, COEFF, 0, ini).state["U"], want.state["U"])
    case.close()
