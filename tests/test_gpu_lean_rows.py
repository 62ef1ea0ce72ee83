"""Rows whose cells and neighbours are all open take a straight line without fractions or divisions in the one-cell
column kernels of FP32 levels that are not whole quads (their FP64 sweeps, and variant 6 of whole quads, take the general
line): cycles of levels where such rows meet walls, cut rows and the ends of chunks, against the FP64 oracle."""
import numpy as np
import pytest
import torch

from test_gpu_cycle_cluster import T, _close, _problem

pytestmark = pytest.mark.gpu


def balanced(f, act):
    """f in steps of 1/256 with the sum 0 exactly: the solves take f's mean off, the oracle's cycles do not."""
    g = np.where(act, np.round(f * 256), 0.0)
    at = np.flatnonzero(act)
    k = int(g.sum())
    step = -(-abs(k) // at.size)
    while k:
        m = min(abs(k) // step, at.size)
        g.reshape(-1)[at[:m]] -= np.sign(k) * step
        k, step = int(g.sum()), 1
    return g / 256


@pytest.mark.parametrize("n", [(16, 32, 4), (17, 64, 5), (33, 36, 12), (9, 67, 7), (8, 128, 16), (23, 133, 9), (40, 198, 11),
                               (12, 256, 10), (5, 6, 7)])
@pytest.mark.parametrize("zc", [1, 3, 64])
def test_cycles_match_oracle(wp, oracle, n, zc):
    """Three cycles with the finest level's kernels pinned to their own launches.  Bound: as for the small levels'
    cycles, 100 eps32 of the iterate, and for the FP64 iterate of FP64 cycles 200 eps64 (the oracle rounds as often)."""
    h, a, act, f = _problem(oracle, n, seed=sum(n), steps=16)
    f = balanced(f, act)
    ref = oracle.mgfrac3d_solve(f, *a, n, (h,) * 3, 3, 2, 2, 2 / 3, prolong=1)[0]
    mg = wp.CuMultigridFrac3D(*[T(v) for v in a], n, h)
    out = torch.full(f.shape, float("nan"), device="cuda")
    for var in (0, 1, 2, 6):
        mg.SetTile(0, 0, zc, var)
        mg.SetTile(0, 1, zc, min(var, 4))
        mg.SetTile(0, 2, zc, 0)
        for precision in (wp.PREC_FP32, wp.PREC_MIXED, wp.PREC_FP64):
            rep = mg.SolveTol(out, None, T(f), rel_tol=0.0, max_cycles=3, precision=precision)
            assert rep["status"] == "WP_OK" and rep["cycles"] == 3
            _close(ref, out.double().cpu().numpy(), act, 1.2e-5)
            if precision == wp.PREC_FP64:
                _close(ref, mg.Iterate64(), act, 200 * 1.1e-16)
            assert not out.cpu().numpy()[~act].any()
