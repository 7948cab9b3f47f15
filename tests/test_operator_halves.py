"""The packed operator reads the upper half of every block: products at every order and
right-hand-side count, and a ragged batch whose clusters take both summations, against the
dense aggregate of the assembler."""

import numpy as np
import pytest
import torch

from miepy_gb300 import _native as nat

pytestmark = pytest.mark.gpu


def _spec(rng, N, L, R):
    pos = np.array([(i % 5, i // 5 % 5, i // 25) for i in range(N)], float) * 2.5e-7 + rng.uniform(-3e-8, 3e-8, (N, 3))
    mie = (rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))) * 0.2 ** np.arange(1, L + 1)
    p = rng.normal(size=(N, 2, L * (L + 2), R)) + 1j * rng.normal(size=(N, 2, L * (L + 2), R))
    return dict(position=pos, mie_scat=mie, k=1.05e7, p_src=p)


def _dense(sp):
    from miepy_gb300.engine import current_stream
    dev = torch.device("cuda", 0)
    N, _, L = sp["mie_scat"].shape
    D = 2 * L * (L + 2) * N
    pos = torch.from_numpy(sp["position"]).to(dev)
    mie = torch.from_numpy(np.ascontiguousarray(sp["mie_scat"])).to(dev)
    T = torch.empty((D, D), dtype=torch.complex128, device=dev)
    nat.check(nat.lib().gb_assemble_sphere_dense(N, L, nat.ptr(pos), nat.ptr(mie), sp["k"], nat.ptr(T),
                                                 current_stream(dev)))
    return T + torch.eye(D, dtype=torch.complex128, device=dev)


CASES = [([(3 + 4 * (L % 3), L)], R) for L in range(1, 9) for R in (1, 2, 4) if 2 * L * (L + 2) * R <= 384]
CASES += [([(2, 3), (7, 4), (5, 1), (3, 6), (4, 3)], R) for R in (1, 2)] + [([(33, 3)], 8), ([(33, 4)], 8)]


@pytest.mark.parametrize("shapes,R", CASES)
def test_products_match_the_dense_aggregate(shapes, R):
    from miepy_gb300.engine import ClusterBatch
    rng = np.random.default_rng(len(shapes) * 10 + R)
    specs = [_spec(rng, N, L, R) for N, L in shapes]
    ops = [_dense(s) for s in specs]
    # FP64 and double-float carry sums of ~1e3 terms; complex64's bar is the solver's
    for batch_prec, prec, bar in (("fp64", "fp64", 2e-14), ("mixed", "mixed", 2e-12), ("mixed", "fp32", 2e-6)):
        b = ClusterBatch(specs, R=R, precision=batch_prec).assemble()
        y = b.apply(b.b, prec)
        for s, A in enumerate(ops):
            x = b.cluster_view(s, b.b).reshape(A.shape[0], R)
            want, got = A @ x, b.cluster_view(s, y).reshape(A.shape[0], R)
            assert float((got - want).abs().max() / want.abs().max()) < bar, (shapes[s], prec)
