"""What must not show in the bits of a solve: the kernel variant and tile of a level (the tuner picks them by the clock)
and the alignment of an argument."""
import numpy as np
import pytest
import torch

from test_gpu_cycle_cluster import T, _problem

pytestmark = pytest.mark.gpu


def _quantised(oracle, n, seed):
    """_problem with right-hand sides of few bits: their sums are exact in FP64 in any order."""
    h, a, act, f = _problem(oracle, n, seed=seed)
    return h, a, act, np.where(act, np.round(f * 256) / 256, 0.0)


def _solve(wp, mg, f, precision):
    out = torch.full(f.shape, float("nan"), device="cuda")
    rep = mg.SolveTol(out, None, f, rel_tol=0.0, max_cycles=3, precision=precision)
    assert rep["cycles"] == 3
    return out if precision == wp.PREC_FP32 else torch.as_tensor(mg.Iterate64())


@pytest.mark.parametrize("n", [(64, 64, 64), (40, 48, 36), (33, 68, 20)])
def test_variants_give_the_same_bits(wp, oracle, n):
    h, a, act, f = _quantised(oracle, n, seed=sum(n))
    mg = wp.CuMultigridFrac3D(*[T(v) for v in a], n, h)
    tf = T(f)
    mg.SetTile(0, 4, 0, 0)  # (the two fused kernels of level 0 agree to rounding only)
    levels = (0, 1) if n[1] % 8 == 0 else (0,)
    for level in levels:
        for kind in (0, 1):
            mg.SetTile(level, kind, 0, 0)
    for precision in (wp.PREC_FP32, wp.PREC_MIXED):
        ref = _solve(wp, mg, tf, precision)
        for level in levels:
            for kind, variants in ((0, 7), (1, 5), (2, 2)):
                if kind == 2 and level:
                    continue
                for var in range(variants):
                    for zc in (0, 5):
                        mg.SetTile(level, kind, zc, var)
                        assert torch.equal(_solve(wp, mg, tf, precision), ref), (precision, level, kind, var, zc)
                mg.SetTile(level, kind, 0, 0)


@pytest.mark.parametrize("n", [(64, 64, 64), (24, 40, 36)])
def test_alignment_gives_the_same_bits(wp, oracle, n):
    """A right-hand side off a 16-byte boundary takes the one-cell kernels of level 0."""
    h, a, act, f = _quantised(oracle, n, seed=7)
    mg = wp.CuMultigridFrac3D(*[T(v) for v in a], n, h)
    mg.SetTile(0, 4, 0, 0)
    buf = torch.empty(f.size + 4, device="cuda")
    off = buf[1:1 + f.size].view(f.shape)
    off.copy_(T(f))
    assert off.data_ptr() % 16
    for precision in (wp.PREC_FP32, wp.PREC_MIXED):
        assert torch.equal(_solve(wp, mg, off, precision), _solve(wp, mg, T(f), precision)), precision
