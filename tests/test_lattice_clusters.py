"""Lattice sums whose chunks are shared by clusters of 2 to 16 CTAs (small blocks, few
pairs): cell counts at the limits of each, CTAs with no cells left, against the oracle's
periodic aggregate; the same bits on every call."""

import numpy as np
import pytest

from miepy_gb300 import _native as nat
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# N = 1, lmax 1: 2, 4 CTAs per chunk from 31, 63 cells on; of two chunks 4, 8, 16 from 128, 255, 511
CASES = [(1, 1, n) for n in (30, 31, 62, 63, 65, 127, 128, 130, 254, 255, 257, 510, 511, 513, 1031, 5039)] + \
        [(1, 2, 447), (1, 2, 900), (2, 1, 511), (6, 1, 300), (6, 1, 520), (1, 3, 901), (1, 5, 200), (1, 8, 97), (3, 9, 70)]


@pytest.mark.parametrize("N,L,ncell", CASES)
def test_periodic_aggregate(N, L, ncell):
    import torch

    from miepy_gb300.engine import current_stream
    rng = np.random.default_rng([N, L, ncell])
    k = 1.05e7
    pos = np.array([(i, i % 2, 0.3 * i) for i in range(N)], float) * 3e-7 + rng.uniform(-2e-8, 2e-8, (N, 3))
    mie = rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))
    side = int(np.ceil(np.sqrt(ncell + 1))) | 1
    xy = np.array([(a, b, 0) for a in range(-(side // 2), side // 2 + 1) for b in range(-(side // 2), side // 2 + 1)
                   if a or b], float)
    cells = np.ascontiguousarray(xy[:ncell] * 1.9e-6)
    kh = np.array([0.3, -0.2, np.sqrt(1 - 0.13)])
    dev = torch.device("cuda", 0)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    D = 2 * L * (L + 2) * N
    dp, dm, dc = d(pos), d(mie), d(cells)

    def aggregate():
        out = torch.full((D, D), complex(np.nan, np.nan), dtype=torch.complex128, device=dev)
        nat.check(nat.lib().gb_aggregate_periodic_dense(N, L, nat.ptr(dp), nat.ptr(dm), k, nat.ptr(dc), ncell, *kh,
                                                        nat.ptr(out), current_stream(dev)))
        return out
    out = aggregate()
    assert torch.equal(out, aggregate())
    ref = O.sphere_aggregate_tmatrix_periodic(pos, mie.reshape(N, -1), k, cells.reshape(-1, 3), kh).reshape(D, D)
    err = np.max(np.abs(out.cpu().numpy() - ref)) / np.max(np.abs(ref))
    assert err < (1e-12 if L <= 8 else 1e-10)   # the aggregate's bars


@pytest.mark.parametrize("N,L", [(1, 1), (1, 9), (7, 3)])
def test_no_cells(N, L):
    """Without cells the aggregate is the plain one: the same bits from the same launches."""
    import torch

    from miepy_gb300.engine import current_stream
    lib = nat.lib()
    rng = np.random.default_rng([N, L])
    dev = torch.device("cuda", 0)
    pos = torch.from_numpy(np.array([(i, i % 2, 0.3 * i) for i in range(N)], float) * 3e-7).to(dev)
    mie = torch.from_numpy(rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))).to(dev)
    D = 2 * L * (L + 2) * N
    out = [torch.full((D, D), complex(np.nan, np.nan), dtype=torch.complex128, device=dev) for _ in range(2)]
    n0 = lib.gb_launch_count()
    nat.check(lib.gb_assemble_sphere_dense(N, L, nat.ptr(pos), nat.ptr(mie), 1.05e7, nat.ptr(out[0]), current_stream(dev)))
    n1 = lib.gb_launch_count()
    nat.check(lib.gb_aggregate_periodic_dense(N, L, nat.ptr(pos), nat.ptr(mie), 1.05e7, None, 0, 0.0, 0.0, 1.0,
                                              nat.ptr(out[1]), current_stream(dev)))
    assert lib.gb_launch_count() - n1 == n1 - n0
    assert torch.equal(out[0], out[1])
