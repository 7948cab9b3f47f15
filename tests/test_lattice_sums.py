"""The lattice-sum kernel at the edges of its chunks and stages: cell counts around them,
every order it takes, one particle and several, against the oracle's periodic aggregate."""

import numpy as np
import pytest

from miepy_gb300 import _native as nat
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 1), (1, 3, 128), (2, 1, 0), (2, 2, 1), (3, 1, 511), (3, 2, 512), (2, 3, 513), (2, 4, 1300), (4, 3, 127),
         (2, 5, 257), (2, 6, 100), (1, 7, 255), (2, 8, 129), (2, 9, 40)]


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
    dp, dm, dc = d(pos), d(mie), d(cells if ncell else np.zeros((1, 3)))
    out = torch.full((D, D), complex(np.nan, np.nan), dtype=torch.complex128, device=dev)
    nat.check(nat.lib().gb_aggregate_periodic_dense(N, L, nat.ptr(dp), nat.ptr(dm), k, nat.ptr(dc), ncell, *kh,
                                                    nat.ptr(out), current_stream(dev)))
    ref = O.sphere_aggregate_tmatrix_periodic(pos, mie.reshape(N, -1), k, cells.reshape(-1, 3), kh).reshape(D, D)
    err = np.max(np.abs(out.cpu().numpy() - ref)) / max(np.max(np.abs(ref)), 1e-300)
    assert err < (1e-12 if L <= 8 else 1e-10)   # the aggregate's bars
