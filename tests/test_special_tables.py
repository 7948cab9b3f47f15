"""pi_tau_emn gives the per-mode functions' values, bit for bit."""

import numpy as np
import pytest

from miepy_gb300.modes import mode_indices
from miepy_gb300.special import Emn, pi_func, pi_tau_emn, tau_func


@pytest.mark.parametrize("theta", [0, np.pi, np.pi / 2, 0.3, 2.9, 1e-9, -0.4, 4.0])
@pytest.mark.parametrize("lmax", [1, 2, 5, 10])
def test_mode_tables(lmax, theta):
    pi, tau, emn = pi_tau_emn(lmax, theta)
    for r, n, m in mode_indices(lmax):
        assert pi[r] == pi_func(n, m, theta) and tau[r] == tau_func(n, m, theta) and emn[r] == abs(Emn(m, n))
