"""Sub-sampled face fractions of an arbitrary level set (the static CuSolidLevelSet3D::GetFrac)
against the reference's golden fixtures and the FP64 oracle.  The fraction of a cut face is a count
of 128 x 128 sub-face samples; a sample whose interpolated level set lies within rounding of zero
may fall on either side, so two results may differ by a few samples (1/16384 each)."""
import numpy as np
import pytest
import torch

from conftest import load_golden
from test_gpu_parity import N, T

pytestmark = pytest.mark.gpu

SAMPLE = 1.0 / 16384


def _frac(wp, ls, n, h):
    s = wp.mac_shapes3d(*n)
    out = [torch.full(s[k], -1.0, device="cuda") for k in ("xv", "yv", "zv")]
    lso = wp.CuSolidLevelSet3D(n, h)
    lso.GetFrac(*out, ls=T(ls), dim=n, dx=h)
    torch.cuda.synchronize()
    return [N(t) for t in out]


def test_subsampled_fractions_match_reference(wp):
    g = load_golden("frac3d_sub")
    for key in [k for k in g.files if k.startswith("n_")]:
        tag = key[2:]
        n = tuple(int(v) for v in g[key])
        got = _frac(wp, g[f"ls_{tag}"], n, 1.0 / n[0])
        for k, o in zip(("ax", "ay", "az"), got):
            ref = g[f"{k}_{tag}"]
            d = np.abs(o - ref)
            assert d.max() <= 3 * SAMPLE and np.count_nonzero(d) <= max(3, ref.size // 10000), (tag, k, d.max())
            assert np.any((ref > 0) & (ref < 1))


def test_subsampled_fractions_match_oracle_at_64(wp, oracle):
    n = (64, 48, 40)
    h = 1.0 / 64
    rng = np.random.default_rng(3)
    sdf = oracle.sdf_spheres3d(n, h, rng.uniform(0.2, 0.6, (5, 3)), rng.uniform(0.08, 0.2, 5))
    ls = (-sdf).astype(np.float32).astype(np.float64)  # fluid inside the balls
    ref = oracle.fractions3d_subsampled(ls, n, h)
    got = _frac(wp, ls, n, h)
    for r, o in zip(ref, got):
        d = np.abs(o - r)
        assert d.max() <= 3 * SAMPLE and np.count_nonzero(d) <= max(3, r.size // 10000), d.max()
        assert np.all((o >= 0) & (o <= 1))


@pytest.mark.parametrize("slope", [(1.0, 0.0, 0.0), (0.0, -0.5, 0.0), (0.0, 0.0, 1.0), (1.0, 0.25, -0.5), (0.5, 0.5, 0.5)])
@pytest.mark.parametrize("n", [(5, 9, 7), (8, 33, 6)])
@pytest.mark.parametrize("offset", [0.0, 1.0 / 1024, 5.0 / 32])
def test_plane_fractions_are_exact_counts(wp, oracle, n, offset, slope):
    """Planes with dyadic coefficients, the zero set on sample positions and cell centres.  Every product of
    the interpolation is a dyadic number of fewer than 53 bits, so the sample values are exact and the counts
    must be equal (bound 0).  In the first half cell the position is clamped to a number that is not dyadic: a
    plane through its samples (offset 0) is left out there."""
    h = 1.0 / 16
    z, x, y = np.meshgrid(*[np.arange(k) + 0.5 for k in (n[2], n[0], n[1])], indexing="ij")
    ls = (slope[0] * (x - n[0] / 2) + slope[1] * (y - n[1] / 2) + slope[2] * (z - n[2] / 2) + offset) * h
    assert np.array_equal(ls, ls.astype(np.float32))
    got = _frac(wp, ls.astype(np.float32), n, h)
    at = (slice(1, None),) * 3 if offset == 0 else ()
    for r, o in zip(oracle.fractions3d_subsampled(ls, n, h), got):
        assert np.array_equal(o[at], r[at])


def test_non_finite_level_sets_match_oracle(wp, oracle):
    """A value that is not finite makes every face whose 27 taps hold it compare false (closed), taps of
    weight 0 included.  No bound: comparisons only."""
    n, h = (6, 40, 5), 1.0 / 16
    ls = np.full((n[2], n[0], n[1]), 3 * h, dtype=np.float32)
    ls[2, 3, 7] = np.nan
    ls[2, 3, 20] = np.inf
    ls[2, 3, 33] = -np.inf
    for r, o in zip(oracle.fractions3d_subsampled(ls.astype(np.float64), n, h), _frac(wp, ls, n, h)):
        assert np.array_equal(o, r)
        assert (r == 0).any() and (r == 1).any()


@pytest.mark.parametrize("far", [1e8, 1e30, 3e38])
@pytest.mark.parametrize("h", [0.3, 1e-20])
def test_huge_values_classify_as_in_fp64(wp, far, h):
    """Cells marked by a huge value: where positions round, taps of nominal weight 0 count.  The same cells beside one that is
    not a number, which makes every face take FP64, give the same fractions (bound 0) away from it."""
    n = (24, 17, 16)
    rng = np.random.default_rng(8)
    ls = (rng.standard_normal((n[2], n[0], n[1])) * 4 * h).astype(np.float32)
    ls.reshape(-1)[::503] = far
    fp64 = ls.copy()
    fp64[:, -1] = np.nan
    for a, b in zip(_frac(wp, ls, n, h), _frac(wp, fp64, n, h)):
        assert np.array_equal(a[:, :20], b[:, :20])
        assert 0.1 < (a[:, :20] > 0).mean() < 0.9
