"""Field maps whose coordinates lie far from the origin: the kernels' separations are those of
the coordinates as given, so the fields match the direct sum over them."""

import numpy as np
import pytest

from tests.test_fields import K, _case, _exterior, _near

pytestmark = pytest.mark.gpu

OFFSET = np.array([1e4, -2e4, 5e3]) + 1 / 3   # double precision keeps 4e-12 there: geometry of 1e-6 stays itself


@pytest.mark.parametrize("N,L,P", [(1, 3, 5), (17, 1, 257), (40, 4, 65)])
def test_exterior_fields(N, L, P):
    pos, c, pts = _case(N, L, P)
    pts[:, 2] = np.abs(pts[:, 2]) + 2e-6   # no point next to a sphere: every field counts
    pos, pts = pos + OFFSET, pts + OFFSET
    ref = _exterior(pos, c, pts, L)
    top = np.max(np.abs(ref))
    # the bars of the same maps about the origin
    np.testing.assert_allclose(_near(False, pos, c, pts, L), ref, rtol=0, atol=2e-12 * top)
    np.testing.assert_allclose(_near(True, pos, c, pts, L), ref, rtol=0, atol=2e-5 * top)


@pytest.mark.parametrize("L", [2, 6])
def test_points_inside_spheres(L):
    pos, c, pts = _case(19, L, 300, seed=3)
    pts[5:290] = pos[np.arange(285) % 19] + np.random.default_rng(4).uniform(-8e-8, 8e-8, (285, 3))
    pos, pts = pos + OFFSET, pts + OFFSET
    rad = np.full(19, 1e-7)
    k_int = K * (1.5 + 0.1j + 0.05 * np.arange(19))
    out = _near(False, pos, c, pts, L, 0, rad, c[::-1].copy(), k_int)
    out32 = _near(True, pos, c, pts, L, 0, rad, c[::-1].copy(), k_int)
    inside = (np.sum((pts[:, None] - pos[None]) ** 2, axis=2) < rad ** 2).any(axis=1)
    assert inside.sum() > 50 and (~inside).sum() > 50
    # inside: the same FP64 expansion in both; outside: FP32 phases
    np.testing.assert_array_equal(out32[inside], out[inside])
    top = np.max(np.abs(out[~inside]))
    np.testing.assert_allclose(out32[~inside], out[~inside], rtol=0, atol=2e-5 * top)
