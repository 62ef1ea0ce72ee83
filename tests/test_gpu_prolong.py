"""Prolongation by pairs of planes (quads) and by four planes (any extents): V(1, 1) cycles of levels with odd and even
numbers of planes, against the FP64 oracle."""
import pytest
import torch

from test_gpu_cycle_cluster import T, _close, _problem
from test_gpu_lean_rows import balanced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 32, 2), (17, 64, 3), (12, 36, 5), (33, 40, 8), (9, 67, 2), (23, 35, 3), (14, 21, 6), (31, 33, 9)])
def test_cycles_match_oracle(wp, oracle, n):
    """Three V(1, 1) cycles with the levels' own kernels.  Bound: as for the small levels' cycles, 100 eps32 of the
    iterate, and for the FP64 iterate of FP64 cycles 200 eps64 (the oracle rounds as often)."""
    h, a, act, f = _problem(oracle, n, seed=sum(n), steps=16)
    f = balanced(f, act)
    ref = oracle.mgfrac3d_solve(f, *a, n, (h,) * 3, 3, 1, 1, 2 / 3, prolong=1)[0]
    mg = wp.CuMultigridFrac3D(*[T(v) for v in a], n, h)
    mg.SetTile(0, 0, 0, 0)
    out = torch.full(f.shape, float("nan"), device="cuda")
    for precision in (wp.PREC_FP32, wp.PREC_FP64):
        rep = mg.SolveTol(out, None, T(f), rel_tol=0.0, max_cycles=3, nu1=1, nu2=1, precision=precision)
        assert rep["status"] == "WP_OK" and rep["cycles"] == 3
        _close(ref, out.double().cpu().numpy(), act, 1.2e-5)
        if precision == wp.PREC_FP64:
            _close(ref, mg.Iterate64(), act, 200 * 1.1e-16)
