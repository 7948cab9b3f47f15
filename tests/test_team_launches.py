"""Which solver ran: the single-launch BiCGSTAB is one launch, the launch-per-step one many.
Both team forms at sizes whose last CTA and last warp are partly filled (stores by some of
a warp's lanes directly before the team's barrier), and the limits of the plan."""

import numpy as np
import pytest

from miepy_gb300 import _native as nat

pytestmark = pytest.mark.gpu


class _Dense:
    """A random dense system; solve() returns the launches it took."""

    def __init__(self, D, R):
        import torch
        dev = torch.device("cuda", 0)
        g = torch.Generator(device="cuda").manual_seed(D * 2 + R)
        self.T = torch.randn(D, D, dtype=torch.complex128, device=dev, generator=g) * (0.4 / D ** 0.5)
        self.b = torch.randn(D, R, dtype=torch.complex128, device=dev, generator=g)
        self.x = torch.empty_like(self.b)
        self.ws = torch.empty(nat.lib().gb_solve_dense_workspace_size(D, R), dtype=torch.uint8, device=dev)
        torch.cuda.synchronize()

    def solve(self):
        from miepy_gb300.engine import current_stream
        L, (D, R) = nat.lib(), self.b.shape
        st, it, rs = np.zeros(R, np.int32), np.zeros(R, np.int32), np.zeros(R)
        n0 = L.gb_launch_count()
        rc = L.gb_solve_dense(D, R, nat.ptr(self.T), nat.ptr(self.b), nat.ptr(self.x), 1e-12, 1000, nat.ptr(self.ws),
                              self.ws.numel(), st.ctypes.data, it.ctypes.data, rs.ctypes.data, current_stream(self.b.device))
        assert rc == nat.GB_OK and np.all(st == 0)
        return L.gb_launch_count() - n0


def _dense(D, R):
    d = _Dense(D, R)
    n = d.solve()
    res = ((d.b - d.x - d.T @ d.x).norm(dim=0) / d.b.norm(dim=0)).cpu().numpy()
    assert np.all(res < 2e-12), res   # the recurrence's 1e-12 and the rounding of ~30 products
    return n


@pytest.mark.parametrize("D,R", [(D, R) for D in (1, 3, 7, 62, 130, 501, 999, 1301, 2999, 3450) for R in (1, 2)] + [(4000, 1)])
def test_dense_systems_take_one_launch(D, R):
    assert _dense(D, R) == 1


@pytest.mark.parametrize("D,R", [(4001, 1), (3600, 2)])
def test_larger_dense_systems_take_the_launch_per_step_solver(D, R):
    assert _dense(D, R) > 1


@pytest.mark.parametrize("n,single", [(1, True), (19, True), (150, True), (152, True), (304, True), (305, False)])
def test_fp64_batches(n, single):
    """Batches of one-launch systems up to two CTAs per SM (152 SMs; N = 5, lmax 2: two CTAs
    per system up to 152 of them) and beyond, against the packed operator's product."""
    from miepy_gb300.engine import ClusterBatch
    if nat.lib().gb_device_sm_count() != 152:
        pytest.skip("batch limits of 152 SMs")
    rng = np.random.default_rng(5)
    N, L = (5, 2) if n <= 152 else (2, 1)
    specs = []
    for _ in range(n):
        pos = np.array([(i % 2, i // 2 % 2, i // 4) for i in range(N)], float) * 3e-7 + rng.uniform(-2e-8, 2e-8, (N, 3))
        mie = (rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))) * 0.1 ** np.arange(1, L + 1)
        p = rng.normal(size=(N, 2, L * (L + 2))) + 1j * rng.normal(size=(N, 2, L * (L + 2)))
        specs.append(dict(position=pos, mie_scat=mie, k=1.05e7, p_src=p))
    b = ClusterBatch(specs, R=1, precision="fp64").assemble()
    n0 = nat.lib().gb_launch_count()
    b.solve(tol=1e-11)
    launches = nat.lib().gb_launch_count() - n0
    assert (launches == 1) == single, launches
    d = b.b - b.apply(b.x)
    for s in range(n):
        assert float(b.cluster_view(s, d).norm() / b.cluster_view(s, b.b).norm()) < 2e-11


@pytest.mark.parametrize("N,L,R,single", [(31, 3, 1, True), (32, 3, 1, True), (25, 4, 1, True), (43, 3, 1, True),
                                          (44, 3, 1, False), (30, 3, 2, True), (42, 3, 2, True), (43, 3, 2, False),
                                          (200, 1, 1, True), (9, 7, 1, True)])
def test_fp64_clusters_beyond_half_of_every_sm(N, L, R, single):
    """Packed systems whose rows take whole SMs, up to the limits (152 SMs), against the
    packed operator's product."""
    from miepy_gb300.engine import ClusterBatch
    if nat.lib().gb_device_sm_count() != 152:
        pytest.skip("limits of 152 SMs")
    rng = np.random.default_rng([N, L])
    pos = np.array([(i % 6, i // 6 % 6, i // 36) for i in range(N)], float) * 4e-7 + rng.uniform(-2e-8, 2e-8, (N, 3))
    mie = (rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))) * 0.1 ** np.arange(1, L + 1)
    p = rng.normal(size=(N, 2, L * (L + 2), R)) + 1j * rng.normal(size=(N, 2, L * (L + 2), R))
    b = ClusterBatch([dict(position=pos, mie_scat=mie, k=1.05e7, p_src=p)], R=R, precision="fp64").assemble()
    n0 = nat.lib().gb_launch_count()
    b.solve(tol=1e-11)
    launches = nat.lib().gb_launch_count() - n0
    assert (launches == 1) == single, launches
    d = (b.b - b.apply(b.x)).view(-1, R)
    assert np.all((d.norm(dim=0) / b.b.view(-1, R).norm(dim=0)).cpu().numpy() < 2e-11)


@pytest.mark.parametrize("R", [1, 2])
def test_expired_team_wait_falls_back(R):
    """A cooperative team whose barrier runs out of its limit is no error: the
    launch-per-step solver takes the system, and the next call is one launch again."""
    L = nat.lib()
    nat.check(L.gb_set_gemv_wait_limit(0, None))
    try:
        assert _dense(1301, R) > 1
    finally:
        nat.check(L.gb_set_gemv_wait_limit(-1, None))
    assert _dense(1301, R) == 1


def test_other_streams_run_beside_a_single_launch_solve():
    """A mixed solve (many small launches) on one stream beside single-launch dense solves of
    some 5 ms each on another: it shares the SMs with them rather than waiting for their
    end at every step.  Shared SMs cost it 1.2 times its time alone; five times are allowed
    (ten waits of 5 ms each would be some fifty times)."""
    import threading
    import time

    import torch

    from miepy_gb300.engine import ClusterBatch
    rng = np.random.default_rng(2)
    N, L = 12, 3
    pos = np.array([(i % 3, i // 3 % 3, i // 9) for i in range(N)], float) * 3e-7
    mie = (rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))) * 0.1 ** np.arange(1, L + 1)
    p = rng.normal(size=(N, 2, L * (L + 2))) + 1j * rng.normal(size=(N, 2, L * (L + 2)))
    stop, started = threading.Event(), threading.Event()

    def dense():
        with torch.cuda.stream(torch.cuda.Stream()):
            while not stop.is_set():
                system.solve()
                started.set()

    system = _Dense(2880, 2)
    assert system.solve() == 1
    with torch.cuda.stream(torch.cuda.Stream()):
        b = ClusterBatch([dict(position=pos, mie_scat=mie, k=1.05e7, p_src=p)], R=1, precision="mixed").assemble()

        def median(n):
            t = []
            for _ in range(n):
                t0 = time.perf_counter()
                b.solve(tol=1e-10, inner_tol=1e-4)
                t.append(time.perf_counter() - t0)
            return sorted(t)[n // 2]

        median(5)
        alone = median(25)
        th = threading.Thread(target=dense)
        th.start()
        try:
            assert started.wait(60)
            beside = median(25)
        finally:
            stop.set()
            th.join()
    assert beside < 5 * alone, (beside, alone)
