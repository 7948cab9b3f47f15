"""complex128 passes whose CTAs' warps share a strip (few strips per SM), at 2, 3 and 4
warps, one and two right-hand sides, with uneven shares: against the double-float product,
which carries sums of ~1e3 terms to 2e-12."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L,R", [(2, 8, 1), (5, 4, 2), (20, 6, 1), (25, 8, 2), (42, 6, 1), (50, 6, 2), (61, 5, 1),
                                   (61, 5, 2), (33, 5, 4)])
def test_products_match_double_float(N, L, R):
    from miepy_gb300.engine import ClusterBatch
    rng = np.random.default_rng(N + L)
    pos = np.array([(i % 5, i // 5 % 5, i // 25) for i in range(N)], float) * 2.5e-7 + rng.uniform(-3e-8, 3e-8, (N, 3))
    mie = (rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))) * 0.2 ** np.arange(1, L + 1)
    p = rng.normal(size=(N, 2, L * (L + 2), R)) + 1j * rng.normal(size=(N, 2, L * (L + 2), R))
    spec = dict(position=pos, mie_scat=mie, k=1.05e7, p_src=p)
    b = ClusterBatch([spec], R=R, precision="fp64").assemble()
    m = ClusterBatch([spec], R=R, precision="mixed").assemble()
    got, want = b.apply(b.b, "fp64"), m.apply(m.b, "mixed")
    assert float((got - want).abs().max() / want.abs().max()) < 2e-12
    assert torch.equal(got, b.apply(b.b, "fp64"))
