"""What must not show in the bits of a solve: the kernel variant and tile of a level (the tuner picks them by the clock)
and the alignment of an argument."""
import numpy as np
import pytest
import torch

from test_gpu_cycle_cluster import T, _problem
from test_gpu_failure_paths import _kernel_names

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
            mg.SetTile(level, kind, 3, 0)
    for precision in (wp.PREC_FP32, wp.PREC_MIXED):
        ref = _solve(wp, mg, tf, precision)
        for level in levels:
            for kind, variants in ((0, 7), (1, 5), (2, 2)):
                if kind == 2 and level:
                    continue
                for var in range(variants):
                    for zc in (2, 5):
                        mg.SetTile(level, kind, zc, var)
                        assert torch.equal(_solve(wp, mg, tf, precision), ref), (precision, level, kind, var, zc)
                mg.SetTile(level, kind, 3, 0)


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


@pytest.mark.parametrize("n", [(64, 64, 64), (96, 64, 48), (40, 48, 36), (72, 88, 132), (64, 64, 24)])
def test_persistent_cycle_gives_the_same_bits(wp, oracle, n):
    """The levels below the finest as one cooperative launch: the pack's larger levels from global memory (extents down to
    9 x 11 x 17) and the rest in one CTA, against the cluster of up to 16."""
    h, a, act, f = _quantised(oracle, n, seed=sum(n))
    mg = wp.CuMultigridFrac3D(*[T(v) for v in a], n, h)
    mg.SetTile(0, 4, 0, 0)
    tf = T(f)
    for precision in (wp.PREC_FP32, wp.PREC_MIXED):
        mg.SetTile(0, 3, 0, 0)
        ref = _solve(wp, mg, tf, precision)
        mg.SetTile(0, 3, 0, 1)
        box = {}
        names = _kernel_names(lambda: box.update(out=_solve(wp, mg, tf, precision)))
        assert "mid_cycle" in names, names
        assert torch.equal(box["out"], ref), precision


def _batch(wp, oracle, specs, **kw):
    """Grids of quantised fractions and velocities on power-of-two spacings: divergences whose FP64 sums are exact in
    any order, so the mean that every way of solving removes is the same."""
    rng = np.random.default_rng(5)
    grids, u = [], []
    for n in specs:
        h, a, act, f = _problem(oracle, n, seed=sum(n))
        h = 1.0 / 64
        a = [T(np.round(v * 16) / 16) for v in a]
        grids.append({"dim": n, "dx": h, **dict(zip(("ax", "ay", "az"), a))})
        u.append([T(np.round(rng.standard_normal(v.shape) * 64) / 64) for v in a])
    return grids, u, wp.BatchProjector(grids, rel_tol=0.0, max_cycles=3, nstreams=2, **kw)


def _potentials(wp, n):
    s = wp.mac_shapes3d(*n) if len(n) == 3 else wp.mac_shapes2d(*n)
    return [torch.full(tuple(s[k]), 7.0, device="cuda") for k in ("qx", "qy", "qz")[0 if len(n) == 3 else 2:]]


def _run(wp, grids, u, bp):
    fu = [[x.clone() for x in v] for v in u]
    outs = [_potentials(wp, g["dim"]) for g in grids]
    bp.run(fu, outs)
    assert bp.results()["cycles"] == [3] * len(grids)
    return fu, outs


# (16 x ...: the finest level is not one of the fused kernels'; 4 x 4 x 256 and 8 x 8 x 256: the pack's last level is divided
# among the CTAs; 16 x 256 x 8: no level fits one CTA)
SPECS = [(32, 32, 32), (16, 32, 64), (16, 256, 8), (16, 64, 64), (8, 8, 256), (4, 4, 256), (8, 16, 128), (256, 128), (64, 64), (32, 256),
         (16, 16, 16), (512, 128)]


def _same(specs, a, b):
    for i, n in enumerate(specs):
        for x, y in zip(a[0][i] + a[1][i], b[0][i] + b[1][i]):
            assert torch.equal(x, y), n


@pytest.mark.parametrize("nu1,nu2,prolong", [(2, 2, 1), (1, 3, 0), (0, 2, 1)])
def test_batch_graph_gives_the_bits_of_one_grid_solves(wp, oracle, nu1, nu2, prolong):
    """A batch divides the pack between the global-memory kernels and one CTA, a grid of its own runs it in a cluster."""
    grids, u, bp = _batch(wp, oracle, SPECS, nu1=nu1, nu2=nu2, prolongation=prolong)
    got = _run(wp, grids, u, bp)
    ref = ([], [])
    for g, v in zip(grids, u):
        n = g["dim"]
        kw = dict(rel_tol=0.0, max_cycles=3, nu1=nu1, nu2=nu2, prolongation=prolong)
        fu = [x.clone() for x in v]
        if len(n) == 3:
            pr = wp.Projector3D(g["ax"], g["ay"], g["az"], n, g["dx"], autotune=False, **kw)
        else:
            pr = wp.Projector2D(g["ax"], g["ay"], n, g["dx"], **kw)
        q = _potentials(wp, n)
        pr.run(*fu, *q)
        ref[0].append(fu)
        ref[1].append(q)
    _same(SPECS, ref, got)


@pytest.mark.parametrize("nu1,nu2,inner,tile", [(2, 2, 1, 0), (1, 2, 3, 4096)])
def test_batch_modes_give_the_same_bits(wp, oracle, nu1, nu2, inner, tile):
    specs = [n for n in SPECS if n != (4, 4, 256)]  # (has no level for the coarse cycle: refused)
    kw = dict(nu1=nu1, nu2=nu2, inner_cycles=inner)
    grids, u, bp = _batch(wp, oracle, specs, **kw)
    ref = _run(wp, grids, u, bp)
    bp.set_mode(wp.BATCH_PERSISTENT, tile)
    got = _run(wp, grids, u, bp)
    _same(specs, ref, got)
