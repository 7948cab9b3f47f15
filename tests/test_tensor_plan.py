"""Workspaces of four right-hand sides: room for the tensor-core pass's units only where the
pass serves the clusters (up to lmax 5)."""

import ctypes

import numpy as np
import pytest

from miepy_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax", [4, 6])
def test_workspace_holds_units_only_for_the_pass(lmax):
    import torch
    torch.zeros(1, device="cuda")
    N, R, D = 60, 4, 60 * 2 * lmax * (lmax + 2)
    sys = nat.gb_system(N=N, lmax=lmax, k=1.05e7, pos_off=0, mat_off=0, vec_off=0, t_off=0)
    size = {p: nat.lib().gb_solve_workspace_size(1, ctypes.byref(sys), R, p) for p in (nat.PREC_FP64, nat.PREC_FP32)}
    # beside the units, FP32's eight vectors take 8 bytes an element less; regions are rounded to 256 bytes
    extra = size[nat.PREC_FP32] + 8 * 8 * D * R - size[nat.PREC_FP64]
    assert extra > 512 if lmax <= 5 else abs(extra) <= 512


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
def test_solves_with_and_without_tiles_share_a_workspace(precision):
    """One workspace serves both: with tiles (units in the plan) and without."""
    from miepy_gb300.engine import ClusterBatch
    rng = np.random.default_rng(4)
    N, L, R = 20, 3, 4
    pos = np.array([(i % 3, i // 3 % 3, i // 9) for i in range(N)], float) * 3e-7 + rng.uniform(-2e-8, 2e-8, (N, 3))
    mie = (rng.normal(size=(N, 2, L)) + 1j * rng.normal(size=(N, 2, L))) * 0.1 ** np.arange(1, L + 1)
    p = rng.normal(size=(N, 2, L * (L + 2), R)) + 1j * rng.normal(size=(N, 2, L * (L + 2), R))
    tol = 1e-5 if precision == "fp32" else 1e-10
    x = []
    for tensor in (True, False, True):
        b = ClusterBatch([dict(position=pos, mie_scat=mie, k=1.05e7, p_src=p)], R=R, precision=precision,
                         tensor=tensor).assemble()
        b.solve(tol=tol, inner_tol=1e-4)
        assert np.all(b.status == 0)
        x.append(b.x.clone())
    # each solves to tol; well conditioned, so the errors are a few times that
    assert float((x[0] - x[1]).norm() / x[1].norm()) < 20 * tol
    assert bool((x[0] == x[2]).all())
