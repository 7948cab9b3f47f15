"""Tensor-core pass on half blocks: the tiles hold the sum and the difference of a
block's quadrants, the vectors' operands are prepared once per product.

Bar 2e-5 of the largest entry: per term the split drops lo x lo (2^-9 of hi each, so
2^-18) and rounds the two lo parts to bf16 (2^-9 of 2^-9 each): 3 * 2^-18 = 1.2e-5 of
the sum of |terms| at worst, and FP32 accumulation.
"""

import numpy as np
import pytest
import torch

from miepy_gb300._native import GBError
from miepy_gb300.engine import ClusterBatch

pytestmark = pytest.mark.gpu


def batch(cases, R, seed=0):
    rng = np.random.default_rng(seed)
    specs = []
    for N, lmax in cases:
        side = int(np.ceil(N ** (1 / 3)))
        grid = np.array([(a, b, c) for a in range(side) for b in range(side) for c in range(side)][:N], float)
        pos = (grid * 250 + rng.uniform(-20, 20, size=(N, 3))) * 1e-9
        mie = (rng.normal(size=(N, 2, lmax)) + 1j * rng.normal(size=(N, 2, lmax))) * 0.3
        rmax = lmax * (lmax + 2)
        x = rng.normal(size=(N, 2, rmax, R)) + 1j * rng.normal(size=(N, 2, rmax, R))
        specs.append(dict(position=pos, mie_scat=mie, k=2 * np.pi / 650e-9, p_src=x))
    return ClusterBatch(specs, R=R, precision="mixed", tensor=True).assemble()


# one pair; padded columns (lmax 1, 3, 5); rows past a warp's 32 (lmax 5); strips of
# several blocks and of several per CTA; block sizes side by side
@pytest.mark.parametrize("cases,R", [([(2, 1)], 8), ([(2, 4)], 8), ([(3, 2)], 4), ([(2, 5)], 4), ([(150, 1)], 8),
                                     ([(150, 3)], 4), ([(120, 4)], 8), ([(70, 5)], 4),
                                     ([(1, 4), (40, 1), (33, 4), (2, 3), (2, 2)], 8), ([(33, 5), (2, 1), (9, 4)], 4)])
def test_products_match_double_float(cases, R):
    b = batch(cases, R, seed=len(cases) + R)
    x = b.b.clone()
    y, want = b.apply_tc(x), b.apply(x, "mixed")
    for s in range(len(cases)):
        d = b.cluster_view(s, y) - b.cluster_view(s, want)
        assert float(d.abs().max() / b.cluster_view(s, want).abs().max()) < 2e-5
    assert torch.equal(y, b.apply_tc(x))


def test_blocks_past_lmax_5_are_refused():
    b = batch([(4, 6)], 4)
    with pytest.raises(GBError):
        b.apply_tc(b.b.clone())
