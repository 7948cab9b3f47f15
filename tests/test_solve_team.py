"""The single-launch BiCGSTAB of small FP64 systems: system sizes around its row tiles,
teams and limits, restarts, ragged batches, and the ends a solve can come to."""

import numpy as np
import pytest

from miepy_gb300 import _native as nat

pytestmark = pytest.mark.gpu


def _solve(T, b, tol=1e-12, maxiter=1000, noalloc=False):
    import torch

    from miepy_gb300.engine import current_stream
    L, dev = nat.lib(), torch.device("cuda", 0)
    D, R = b.shape
    Td = torch.as_tensor(T, device=dev)
    bd = torch.as_tensor(b, device=dev)
    x = torch.full_like(bd, complex(np.nan, np.nan))
    ws = torch.empty(L.gb_solve_dense_workspace_size(D, R), dtype=torch.uint8, device=dev)
    st, it, rs = np.zeros(R, np.int32), np.zeros(R, np.int32), np.zeros(R)
    args = (D, R, nat.ptr(Td), nat.ptr(bd), nat.ptr(x), tol, maxiter)
    tail = (st.ctypes.data, it.ctypes.data, rs.ctypes.data, current_stream(dev))
    rc = L.gb_solve_dense_noalloc(*args, *tail) if noalloc else L.gb_solve_dense(*args, nat.ptr(ws), ws.numel(), *tail)
    return rc, x, st, it, rs, Td, bd


@pytest.mark.parametrize("R", [1, 2])
@pytest.mark.parametrize("D", [1, 2, 3, 5, 15, 16, 17, 33, 64, 65, 97, 130, 257, 600, 611, 1215, 1301, 2433, 4000, 4001])
def test_dense_sizes(D, R):
    import torch
    g = torch.Generator(device="cuda").manual_seed(D * 2 + R)
    T = torch.randn(D, D, dtype=torch.complex128, device="cuda", generator=g) * (0.4 / D ** 0.5)
    b = torch.randn(D, R, dtype=torch.complex128, device="cuda", generator=g)
    for noalloc in (False, True):
        if noalloc and D * R > 2000:
            continue
        rc, x, st, it, rs, Td, bd = _solve(T, b, noalloc=noalloc)
        assert rc == nat.GB_OK and np.all(st == 0) and np.all(it >= 1)
        res = ((bd - x - Td @ x).norm(dim=0) / bd.norm(dim=0)).cpu().numpy()
        # the recurrence's residual meets 1e-12; the true one differs by rounding (~30 products of 1e-16)
        assert np.all(res < 2e-12), res
        assert np.all(rs < 1e-12)


@pytest.mark.parametrize("R", [1, 2])
def test_restart_on_a_vanishing_rho(R):
    """r0 = e1 and <r0, r1> = 0 exactly after one iteration: the solve restarts from
    r = b - A x and goes on."""
    A = np.array([[1, 0, 0.5], [0.5, 1, 0.25], [0, 1, 1]], complex)
    b = np.zeros((3, R), complex)
    b[0] = 1.0
    if R == 2:
        b[:, 1] = [0.3, -0.2j, 1.0]      # an ordinary one beside it
    rc, x, st, it, rs, _, _ = _solve(A - np.eye(3), b, tol=1e-13)
    assert rc == nat.GB_OK and np.all(st == 0)
    np.testing.assert_allclose(x.cpu().numpy(), np.linalg.solve(A, b), rtol=0, atol=1e-12)


def test_ends_of_a_solve():
    rng = np.random.default_rng(1)
    T = (rng.normal(size=(40, 40)) + 1j * rng.normal(size=(40, 40))) * 0.05
    b = rng.normal(size=(40, 2)) + 0j
    zero = b.copy()
    zero[:, 0] = 0
    rc, x, st, it, _, _, _ = _solve(T, zero)
    assert rc == nat.GB_OK and list(st) == [0, 0] and it[0] == 0
    assert np.all(x.cpu().numpy()[:, 0] == 0)
    bad = b.copy()
    bad[7, 1] = np.nan
    rc, x, st, _, _, _, _ = _solve(T, bad)
    assert list(st) == [nat.GB_OK, nat.GB_NAN]
    np.testing.assert_allclose(x.cpu().numpy()[:, 0], np.linalg.solve(np.eye(40) + T, b[:, 0]), rtol=0, atol=1e-10)
    rc, _, st, it, rs, _, _ = _solve(T, b, maxiter=2)
    assert list(st) == [nat.GB_NOT_CONVERGED] * 2 and list(it) == [2, 2] and np.all(rs > 1e-12)


@pytest.mark.parametrize("R", [1, 2])
def test_packed_ragged_batches(R):
    """Small clusters of different sizes and orders in one batch, and single clusters up to
    the largest system of the packed single-launch solve and beyond, against the packed
    operator product."""
    from miepy_gb300.engine import ClusterBatch
    rng = np.random.default_rng(3)

    def spec(N, L):
        g = np.array([(i % 7, i // 7 % 7, i // 49) for i in range(N)], float) * 2.3e-7
        pos = g + rng.uniform(-2e-8, 2e-8, (N, 3))
        mie = (rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))) * 0.1 ** np.arange(1, L + 1)
        p = rng.normal(size=(N, 2, L * (L + 2), R)) + 1j * rng.normal(size=(N, 2, L * (L + 2), R))
        return dict(position=pos, mie_scat=mie, k=1.05e7, p_src=p)

    for shapes in ([(1, 1), (2, 3), (5, 2), (9, 1), (3, 4)], [(7, 2)] * 40, [(13, 3)], [(60, 2)], [(26, 4)], [(40, 4)],
                   [(12, 3), (20, 3)]):
        b = ClusterBatch([spec(*s) for s in shapes], R=R, precision="fp64").assemble()
        b.solve(tol=1e-11)
        assert np.all(b.status == 0) and np.all(b.resid < 1e-11)
        y = b.apply(b.x)
        for s in range(len(shapes)):
            want, got = b.cluster_view(s, b.b), b.cluster_view(s, y)
            for q in range(R):
                d = (want - got)[..., q].norm() / want[..., q].norm()
                assert d < 2e-11, (shapes[s], q, float(d))


@pytest.mark.parametrize("R", [1, 2])
@pytest.mark.parametrize("shapes", [[(2, 1)], [(5, 2)], [(3, 7)], [(26, 3)], [(14, 6)], [(15, 6)], [(5, 2), (7, 1), (2, 4)],
                                    [(5, 2)] * 152, [(5, 2)] * 153])
def test_small_mixed_solves(shapes, R):
    """The mixed method's small systems and batches: the true residual (double-float
    product) meets the tolerance."""
    from miepy_gb300.engine import ClusterBatch
    rng = np.random.default_rng(11)
    specs = []
    for N, L in shapes:
        pos = np.array([(i % 4, i // 4 % 4, i // 16) for i in range(N)], float) * 3e-7 + rng.uniform(-2e-8, 2e-8, (N, 3))
        mie = (rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))) * 0.1 ** np.arange(1, L + 1)
        p = rng.normal(size=(N, 2, L * (L + 2), R)) + 1j * rng.normal(size=(N, 2, L * (L + 2), R))
        specs.append(dict(position=pos, mie_scat=mie, k=1.05e7, p_src=p))
    b = ClusterBatch(specs, R=R, precision="mixed").assemble()
    b.solve(tol=1e-10, inner_tol=1e-4)
    assert np.all(b.status == 0) and np.all(b.resid <= 1e-10) and np.all(b.iters >= 1)
    d = b.b - b.apply(b.x, "mixed")
    for s in range(len(shapes)):
        for q in range(R):
            rel = b.cluster_view(s, d)[..., q].norm() / b.cluster_view(s, b.b)[..., q].norm()
            assert float(rel) < 2e-10
    # a right-hand side that cannot be solved ends as the refinement reports it
    specs[0]["p_src"] = specs[0]["p_src"].copy()
    specs[0]["p_src"][0, 0, 0, 0] = np.inf
    b.load(specs).assemble()
    b.solve(tol=1e-10, inner_tol=1e-4)
    assert b.status[0] == nat.GB_NAN and np.all(b.status[R:] == 0)
