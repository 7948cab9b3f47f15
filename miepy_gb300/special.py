"""Host-side angular functions for source decompositions (numpy, vectorised).

Conventions of the reference's C++ module: associated Legendre functions without
the Condon-Shortley phase (GSL_SF_LEGENDRE_NONE, cpp/src/special.cpp:148-204),
pi_func / tau_func with their exact limits at theta = 0 and pi
(cpp/src/special.cpp:209-270), E_mn (cpp/src/vsh_functions.cpp:56-58).
"""

from __future__ import annotations

from functools import lru_cache
from math import factorial

import numpy as np


def _legendre_table(nmax, x):
    """P[n][m] for 0 <= m <= n <= nmax (m >= 0, no Condon-Shortley phase)."""
    x = np.asarray(x, dtype=float)
    u = np.sqrt(np.maximum(0.0, (1.0 - x) * (1.0 + x)))
    P = np.zeros((nmax + 1, nmax + 1) + x.shape)
    P[0, 0] = 1.0
    for m in range(1, nmax + 1):
        P[m, m] = (2 * m - 1) * u * P[m - 1, m - 1]
    for m in range(0, nmax):
        P[m + 1, m] = x * (2 * m + 1) * P[m, m]
    for m in range(0, nmax + 1):
        for n in range(m + 2, nmax + 1):
            P[n, m] = ((2 * n - 1) * x * P[n - 1, m] - (n + m - 1) * P[n - 2, m]) / (n - m)
    return P


def _neg_factor(n, m):
    am = abs(m)
    return (-1) ** am * factorial(n - am) / factorial(n + am)


def associated_legendre(n, m, x):
    if abs(m) > n:
        return np.zeros_like(np.asarray(x, dtype=float))
    P = _legendre_table(n, x)[n, abs(m)]
    return P * _neg_factor(n, m) if m < 0 else P


def pi_func(n, m, theta):
    theta = np.asarray(theta, dtype=float)
    out = np.empty_like(theta)
    at0, atpi = theta == 0, theta == np.pi
    gen = ~(at0 | atpi)
    if np.any(gen):
        t = theta[gen]
        out[gen] = m / np.sin(t) * associated_legendre(n, m, np.cos(t))
    lim0 = n * (n + 1) / 2.0 if m == 1 else (0.5 if m == -1 else 0.0)
    limpi = (-1) ** (n + 1) * (n * (n + 1) / 2.0 if m == 1 else (0.5 if m == -1 else 0.0))
    out[at0] = lim0
    out[atpi] = limpi
    return out if out.shape else float(out)


def tau_func(n, m, theta):
    theta = np.asarray(theta, dtype=float)
    out = np.empty_like(theta)
    at0, atpi = theta == 0, theta == np.pi
    gen = ~(at0 | atpi)
    if np.any(gen):
        t = theta[gen]
        am = abs(m)
        P = _legendre_table(n + 1, np.cos(t))
        pp1 = P[n, am + 1] if am + 1 <= n else 0.0
        pm1 = P[n, am - 1] if am >= 1 else -P[n, 1] / (n * (n + 1))
        d = 0.5 * ((n + am) * (n - am + 1) * pm1 - pp1)
        out[gen] = d * _neg_factor(n, m) if m < 0 else d
    lim0 = n * (n + 1) / 2.0 if m == 1 else (-0.5 if m == -1 else 0.0)
    limpi = (-1) ** n * (n * (n + 1) / 2.0 if m == 1 else (-0.5 if m == -1 else 0.0))
    out[at0] = lim0
    out[atpi] = limpi
    return out if out.shape else float(out)


def Emn(m, n):
    return (1j) ** n * np.sqrt((2 * n + 1) * factorial(n - m) / (n * (n + 1) * factorial(n + m)))


@lru_cache(maxsize=16)
def _mode_constants(lmax):
    """n, |m|, m, the negative-order Legendre factor and |E_mn| of every mode."""
    nm = [(n, m) for n in range(1, lmax + 1) for m in range(-n, n + 1)]
    n, m = (np.array(v) for v in zip(*nm))
    neg = np.array([_neg_factor(*v) if v[1] < 0 else 1.0 for v in nm])
    emn = np.array([np.sqrt((2 * a + 1) * factorial(a - b) / (a * (a + 1) * factorial(a + b))) for a, b in nm])
    tables = n, np.abs(m), m, neg, emn
    for t in tables:   # shared by every caller
        t.setflags(write=False)
    return tables


def pi_tau_emn(lmax, theta):
    """pi_func, tau_func and |Emn| of every mode (in mode order) at one angle, from one
    Legendre table: the values of the functions above, in the same arithmetic.  |Emn| is a
    shared, read-only table."""
    n, am, m, neg, emn = _mode_constants(int(lmax))
    theta = float(theta)
    if theta == 0 or theta == np.pi:
        half = n * (n + 1) / 2.0   # the exact limits, of |m| = 1 only
        pi = np.where(m == 1, half, np.where(m == -1, 0.5, 0.0))
        tau = np.where(m == 1, half, np.where(m == -1, -0.5, 0.0))
        return (pi, tau, emn) if theta == 0 else ((-1.0) ** (n + 1) * pi, (-1.0) ** n * tau, emn)
    x = float(np.cos(theta))
    u = float(np.sqrt(max(0.0, (1.0 - x) * (1.0 + x))))
    top = int(lmax) + 1
    P = [[0.0] * (top + 1) for _ in range(top + 1)]
    P[0][0] = 1.0
    for k in range(1, top + 1):
        P[k][k] = (2 * k - 1) * u * P[k - 1][k - 1]
    for k in range(top):
        P[k + 1][k] = x * (2 * k + 1) * P[k][k]
    for k in range(top + 1):
        for a in range(k + 2, top + 1):
            P[a][k] = ((2 * a - 1) * x * P[a - 1][k] - (a + k - 1) * P[a - 2][k]) / (a - k)
    P = np.array(P)
    pp1 = np.where(am + 1 <= n, P[n, am + 1], 0.0)
    pm1 = np.where(am >= 1, P[n, np.maximum(am - 1, 0)], -P[n, 1] / (n * (n + 1)))
    d = 0.5 * ((n + am) * (n - am + 1) * pm1 - pp1)
    return m / np.sin(theta) * (P[n, am] * neg), d * neg, emn
