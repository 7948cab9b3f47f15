"""Field kernels at the edges of their splits: point counts around a warp and a CTA,
particle counts around the splits and tiles, every order, points on a particle's axis
and inside spheres."""

import ctypes

import numpy as np
import pytest

from miepy_gb300.modes import lmax_to_rmax, mode_indices
from miepy_gb300.special import Emn, pi_func, tau_func

K = 2 * np.pi / 600e-9


def _case(N, L, P, seed=0):
    rng = np.random.default_rng([seed, N, L, P])
    pos = rng.uniform(-1e-6, 1e-6, (N, 3))
    c = rng.normal(size=(N, 2, lmax_to_rmax(L))) + 1j * rng.normal(size=(N, 2, lmax_to_rmax(L)))
    pts = rng.uniform(-2e-6, 2e-6, (P, 3))
    pts[0] = pos[0] + [0, 0, 0.7e-6]            # on the axis of a particle, above ...
    pts[-1] = pos[-1] - [0, 0, 0.9e-6]          # ... and below it
    return pos, c, pts


def _exterior(pos, c, pts, L, swap=False):
    """Direct sum of the outgoing expansions (vsh/expansion.py:13-42): the radial functions
    by scipy, the angular ones by the host's Legendre tables."""
    from scipy.special import spherical_jn, spherical_yn
    E = np.zeros((len(pts), 3), complex)
    for x0, cc in zip(pos, c[:, ::-1] if swap else c):
        d = pts - x0
        rho = np.hypot(d[:, 0], d[:, 1])
        r = np.sqrt(rho ** 2 + d[:, 2] ** 2)
        ct, st = d[:, 2] / r, rho / r
        th = np.where(rho == 0, np.where(ct > 0, 0.0, np.pi), np.arctan2(rho, d[:, 2]))
        ph = np.arctan2(d[:, 1], d[:, 0])
        S = np.zeros((3, len(pts)), complex)
        x = K * r
        for q, n, m in mode_indices(L):
            z = spherical_jn(n, x) + 1j * spherical_yn(n, x)
            zm = spherical_jn(n - 1, x) + 1j * spherical_yn(n - 1, x)
            dz = zm - n * z / x
            pi, tau = pi_func(n, m, th), tau_func(n, m, th)
            w = 1j * Emn(m, n) * np.exp(1j * m * ph)
            P = pi * st / m if m else _p0(n, ct)
            S[0] += w * cc[0, q] * n * (n + 1) * P * z / x
            S[1] += w * (cc[0, q] * tau * dz + cc[1, q] * 1j * pi * z)
            S[2] += w * (cc[0, q] * 1j * pi * dz - cc[1, q] * tau * z)
        cp, sp = np.cos(ph), np.sin(ph)
        E += np.stack([S[0] * st * cp + S[1] * ct * cp - S[2] * sp, S[0] * st * sp + S[1] * ct * sp + S[2] * cp,
                       S[0] * ct - S[1] * st], axis=1)
    return E


def _p0(n, ct):
    from scipy.special import eval_legendre
    return eval_legendre(n, ct)


def _near(fp32, pos, c, pts, L, magnetic=0, radius=None, p_int=None, k_int=None):
    import torch

    from miepy_gb300 import _native as nat
    from miepy_gb300.engine import current_stream
    dev = torch.device("cuda", 0)
    d = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to(dev, dtype=t)
    N = len(pos)
    args = [d(pos, torch.float64), d(radius if radius is not None else np.zeros(N), torch.float64),
            d(c, torch.complex128), d(p_int if p_int is not None else c, torch.complex128)]
    ki = d(k_int if k_int is not None else np.full(N, K, complex), torch.complex128)
    hi = torch.full((N,), -1j, dtype=torch.complex128, device=dev)
    P = d(pts, torch.float64)
    out = torch.full((len(pts), 3), 7.0, dtype=torch.complex128, device=dev)
    fn = nat.lib().gb_near_field32 if fp32 else nat.lib().gb_near_field
    nat.check(fn(N, L, *[nat.ptr(a) for a in args], K, nat.ptr(ki), len(pts), nat.ptr(P), int(radius is not None), magnetic,
                 0.0, -1.0, nat.ptr(hi), nat.ptr(out), current_stream(dev)))
    return out.cpu().numpy()


SIZES = [(1, 1, 1), (1, 3, 2), (2, 2, 31), (3, 4, 33), (9, 8, 64), (17, 5, 257), (40, 6, 65), (33, 7, 129)]


@pytest.mark.gpu
@pytest.mark.parametrize("N,L,P", SIZES)
def test_near_field_sizes(N, L, P):
    pos, c, pts = _case(N, L, P)
    for magnetic in (0, 1):
        ref = _exterior(pos, c, pts, L, swap=bool(magnetic)) * (-1j if magnetic else 1.0)
        got = _near(False, pos, c, pts, L, magnetic)
        # angles through arctan2 and products of ~2 L roundings per term in the reference
        np.testing.assert_allclose(got, ref, rtol=0, atol=2e-12 * np.max(np.abs(ref)))
        got32 = _near(True, pos, c, pts, L, magnetic)
        # FP32 phases k r < 50 and recurrences of L steps: 2e-5 of the largest field
        np.testing.assert_allclose(got32, ref, rtol=0, atol=2e-5 * np.max(np.abs(ref)))


@pytest.mark.gpu
@pytest.mark.parametrize("L", [1, 4, 8])
def test_interior_points_are_the_last_sphere_that_holds_them(L):
    """Points inside two overlapping spheres take the later one, in FP64 and FP32, with the
    particles of one point split over several warps."""
    pos, c, pts = _case(19, L, 70, seed=1)
    pts[5:60] = pos[np.arange(55) % 19] + np.random.default_rng(2).uniform(-5e-8, 5e-8, (55, 3))
    pos[11] = pos[3] + 3e-8
    rad = np.full(19, 1e-7)
    p_int = c[::-1].copy()
    k_int = K * (1.5 + 0.1j + 0.05 * np.arange(19))
    out = _near(False, pos, c, pts, L, 0, rad, p_int, k_int)
    out32 = _near(True, pos, c, pts, L, 0, rad, p_int, k_int)
    inside = np.full(70, -1)
    for i in range(19):
        inside[np.sum((pts - pos[i]) ** 2, axis=1) < rad[i] ** 2] = i
    assert np.sum(inside >= 0) > 40
    # one sphere at a time: only it holds the point
    for i in np.unique(inside[inside >= 0]):
        sel = inside == i
        one = _near(False, pos[i:i + 1], c[i:i + 1], pts[sel], L, 0, np.full(1, 1.0), p_int[i:i + 1], k_int[i:i + 1])
        np.testing.assert_array_equal(out[sel], one)
        np.testing.assert_array_equal(out32[sel], one)


@pytest.mark.gpu
@pytest.mark.parametrize("N,L,n", [(1, 1, 1), (2, 10, 33), (5, 9, 64), (23, 4, 130)])
def test_far_field_sizes(N, L, n):
    """E_angular's kernel against the far-field formula (expand_E_far) summed directly."""
    import torch

    from miepy_gb300 import _native as nat
    from miepy_gb300.engine import current_stream
    pos, c, _ = _case(N, L, 2)
    rng = np.random.default_rng(5)
    th, ph, R = rng.uniform(0.05, 3.0, n), rng.uniform(0, 6, n), rng.uniform(1e-4, 2e-4, n)
    u = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], axis=1)
    E = np.zeros((n, 3), complex)
    for x0, cc in zip(pos, c):
        d = R[:, None] * u - x0
        r = np.linalg.norm(d, axis=1)
        t, p = np.arctan2(np.hypot(d[:, 0], d[:, 1]), d[:, 2]), np.arctan2(d[:, 1], d[:, 0])
        f = np.exp(1j * K * r) / (K * r)
        Et = Ep = 0
        for q, nn, m in mode_indices(L):
            w = f * Emn(m, nn) * (-1j) ** nn * np.exp(1j * m * p)
            pi, tau = pi_func(nn, m, t), tau_func(nn, m, t)
            Et = Et + 1j * w * (cc[0, q] * tau + cc[1, q] * pi)
            Ep = Ep - w * (cc[0, q] * pi + cc[1, q] * tau)
        E += np.stack([Et * np.cos(t) * np.cos(p) - Ep * np.sin(p), Et * np.cos(t) * np.sin(p) + Ep * np.cos(p),
                       -Et * np.sin(t)], axis=1)
    ref = np.stack([np.sum(E * np.stack([np.cos(th) * np.cos(ph), np.cos(th) * np.sin(ph), -np.sin(th)], 1), 1),
                    np.sum(E * np.stack([-np.sin(ph), np.cos(ph), 0 * ph], 1), 1)], axis=1)
    dev = torch.device("cuda", 0)
    d = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a)).to(dev, dtype=dt)
    a = [d(pos, torch.float64), d(c, torch.complex128)]
    pt = [d(v, torch.float64) for v in (R, th, ph)]
    out = torch.empty((n, 2), dtype=torch.complex128, device=dev)
    origin = (ctypes.c_double * 3)(0.0, 0.0, 0.0)
    nat.check(nat.lib().gb_far_field(N, L, nat.ptr(a[0]), nat.ptr(a[1]), K, ctypes.cast(origin, ctypes.c_void_p), n,
                                     *[nat.ptr(v) for v in pt], 0, 1.0, 0.0, nat.ptr(out), current_stream(dev)))
    # k R ~ 2000: the phases carry 1e-12
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=0, atol=2e-11 * np.max(np.abs(ref)))
