"""The per-order tables behind plane-wave sources are shared between calls: a caller cannot
change them for the next one."""

import numpy as np
import pytest

from miepy_gb300.special import pi_tau_emn


@pytest.mark.parametrize("theta", [0.0, 0.7, np.pi])
def test_results_of_one_call_do_not_reach_the_next(theta):
    want = [a.copy() for a in pi_tau_emn(4, theta)]
    for a in pi_tau_emn(4, theta):
        try:
            a *= 2.0
        except ValueError:   # read-only
            pass
    for a, w in zip(pi_tau_emn(4, theta), want):
        np.testing.assert_array_equal(a, w)
