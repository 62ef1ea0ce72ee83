"""The small levels' V-cycle as one launch of one thread-block cluster (csrc/wp_mg_cluster.cuh) against
the FP64 oracle's cycles: slab splits of every kind (whole cubes, odd and thin extents, more planes
than CTAs, replicated levels, a coarsest level above and below one warp), sweep counts and both
prolongations, from zero and from an iterate, stored and added into the FP64 iterate."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def T(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda")


def _problem(oracle, n, seed, steps=0):
    """steps: fractions in 1 / steps (a power of two), which every level's averages of them hold exactly"""
    rng = np.random.default_rng(seed)
    dims = len(n)
    h = 1.0 / max(n)
    if dims == 3:
        sdf = oracle.sdf_spheres3d(n, h, [[0.4 * n[0] * h, 0.5 * n[1] * h, 0.6 * n[2] * h]], [0.22 * min(n) * h])
        a = oracle.fractions3d(sdf, n, h)
        cells, ax = (n[2], n[0], n[1]), (1, 2, 0)
    else:
        x, y = np.meshgrid((np.arange(n[0]) + 0.5) * h, (np.arange(n[1]) + 0.5) * h, indexing="ij")
        a = oracle.fractions2d(np.hypot(x - 0.4 * n[0] * h, y - 0.5 * n[1] * h) - 0.2 * min(n) * h, n, h)
        cells, ax = tuple(n), (0, 1)
    a = [np.round(v * steps) / steps if steps else v.astype(np.float32).astype(np.float64) for v in a]
    diag = np.zeros(cells)
    for v, d in zip(a, ax):
        m = v.shape[d] - 1
        w = v.copy()
        w[tuple(slice(0, 1) if k == d else slice(None) for k in range(dims))] = 0.0
        w[tuple(slice(m, m + 1) if k == d else slice(None) for k in range(dims))] = 0.0
        diag += np.take(w, range(m), axis=d) + np.take(w, range(1, m + 1), axis=d)
    act = diag > 0
    f = np.where(act, rng.standard_normal(cells), 0.0)
    f[act] -= f[act].mean()
    return h, a, act, f.astype(np.float32).astype(np.float64)


def _close(ref, got, act, bound):
    d = got - ref
    d = d - d[act].mean()
    err = np.sqrt(np.sum(d[act] ** 2) / np.sum((ref[act] - ref[act].mean()) ** 2))
    assert err < bound, err


CASES = [((32, 32, 32), 2, 2, 1), ((16, 16, 16), 2, 2, 1), ((8, 8, 8), 1, 2, 1), ((4, 4, 4), 2, 2, 1), ((2, 2, 2), 2, 2, 1),
         ((33, 17, 9), 2, 2, 1), ((5, 40, 23), 2, 1, 0), ((20, 30, 50), 3, 2, 1), ((16, 8, 100), 2, 2, 1), ((7, 3, 65), 1, 1, 1),
         ((64, 64, 4), 2, 2, 1), ((31, 31, 17), 2, 3, 0), ((6, 5, 16), 2, 0, 1), ((50, 12, 15), 2, 2, 1),
         ((256, 256), 2, 2, 1), ((64, 33), 2, 2, 1), ((3, 200), 1, 2, 1), ((301, 7), 2, 2, 0), ((17, 129), 3, 1, 1), ((2, 5), 2, 2, 1)]


@pytest.mark.parametrize("n,nu1,nu2,prolong", CASES)
def test_cluster_cycles_match_oracle(wp, oracle, n, nu1, nu2, prolong):
    """Four FP32 cycles from zero, and two refinement steps of two cycles into the FP64 iterate.  Bound: a
    cycle's FP32 sums (at most ten terms per cell and sweep, cycles contract) stay within 100 eps32 =
    1.2e-5 of the iterate; the oracle's cycles are the same operations in FP64."""
    h, a, act, f = _problem(oracle, n, seed=sum(n))
    solve = oracle.mgfrac3d_solve if len(n) == 3 else oracle.mgfrac2d_solve
    mg = (wp.CuMultigridFrac3D if len(n) == 3 else wp.CuMultigridFrac2D)(*[T(v) for v in a], n, h)
    kw = dict(nu1=nu1, nu2=nu2, weight=2 / 3, prolongation=prolong, rel_tol=0.0, max_cycles=4)
    ref = solve(f, *a, n, (h,) * len(n), 4, nu1, nu2, 2 / 3, prolong=prolong)[0]
    out = torch.full(f.shape, float("nan"), device="cuda")
    rep = mg.SolveTol(out, None, T(f), precision=wp.PREC_FP32, **kw)
    assert rep["status"] == "WP_OK" and rep["cycles"] == 4
    _close(ref, out.double().cpu().numpy(), act, 1.2e-5)
    if nu2:  # a sweep clears what the prolongation left in closed cells
        assert not out.cpu().numpy()[~act].any()
    rep = mg.SolveTol(out, None, T(f), precision=wp.PREC_MIXED, inner_cycles=2, **kw)
    assert rep["cycles"] == 4
    _close(ref, out.double().cpu().numpy(), act, 1.2e-5)


def test_pinned_level_keeps_its_own_kernels(wp, oracle):
    """A level pinned with SetTile is not part of the single launch, until it is given back; the cycles stay the same."""
    n = (32, 32, 32)
    h, a, act, f = _problem(oracle, n, seed=3)
    ref = oracle.mgfrac3d_solve(f, *a, n, (h,) * 3, 3, 2, 2, 2 / 3, prolong=1)[0]
    mg = wp.CuMultigridFrac3D(*[T(v) for v in a], n, h)
    tf = T(f)

    def solve():
        out = torch.zeros(f.shape, device="cuda")
        c0 = wp.lib().wp_launch_count()
        mg.SolveTol(out, None, tf, rel_tol=0.0, max_cycles=3, precision=wp.PREC_FP32)
        _close(ref, out.double().cpu().numpy(), act, 1.2e-5)
        return out, wp.lib().wp_launch_count() - c0

    whole, launches = solve()
    for pin, back in (((0, 0, 0, 0), (0, 0, -1, 0)), ((1, 0, 4, 0), (1, 0, -1, 0)), ((2, 1, 0, 1), (2, 1, -1, 0)),
                      ((0, 4, 0, 0), (0, 4, -1, 1)), ((0, 4, 8, 1), (0, 4, -1, 1))):
        mg.SetTile(*pin)
        assert solve()[1] > launches, pin
        mg.SetTile(*back)
        out, again = solve()
        assert again == launches and torch.equal(out, whole), back
    mg.SetTile(1, 0, 4, 0)  # every pin counts
    mg.SetTile(2, 1, 4, 0)
    for back in ((2, 1, -1, 0), (1, 0, -1, 0)):
        assert solve()[1] > launches
        mg.SetTile(*back)
    assert solve()[1] == launches


@pytest.mark.parametrize("ctas", [8, 4, 2, 1, 0])
@pytest.mark.parametrize("n", [(32, 32, 32), (33, 17, 9), (7, 3, 65), (256, 256)])
def test_smaller_clusters_match_oracle(wp, oracle, n, ctas):
    """A device that places smaller clusters only, or none: fewer levels in the launch, the same cycles.  Bound as above,
    or that of a finest level with kernels of its own: they round f - sum(c v) by eps v / h^2, white noise whose smoothest
    mode (1 / N of it) the cycle divides by an eigenvalue 8 N^2 / pi^2 below the coefficients: 0.8 N eps32, twice that
    for its neighbours."""
    bound = max(1.2e-5, 1.6 * max(n) * 6e-8)
    h, a, act, f = _problem(oracle, n, seed=sum(n) + ctas)
    solve = oracle.mgfrac3d_solve if len(n) == 3 else oracle.mgfrac2d_solve
    ref = solve(f, *a, n, (h,) * len(n), 4, 2, 2, 2 / 3, prolong=1)[0]
    results = []
    for limit in (ctas, -1):
        wp.debug_cluster_limit(limit)
        mg = (wp.CuMultigridFrac3D if len(n) == 3 else wp.CuMultigridFrac2D)(*[T(v) for v in a], n, h)
        out = torch.full(f.shape, float("nan"), device="cuda")
        c0 = wp.lib().wp_launch_count()
        rep = mg.SolveTol(out, None, T(f), rel_tol=0.0, max_cycles=4, precision=wp.PREC_FP32)
        results.append((out, wp.lib().wp_launch_count() - c0))
        assert rep["status"] == "WP_OK" and rep["cycles"] == 4
        _close(ref, out.double().cpu().numpy(), act, bound)
    (less, launches), (whole, launches16) = results
    if ctas >= 4 and n == (33, 17, 9) or ctas and n == (7, 3, 65):  # still the whole grid: the same bits
        assert launches == launches16 and torch.equal(less, whole)
    else:
        assert launches > launches16
