"""The calls that programs built on this framework make, with their inputs, their results in 64 bits
and the tolerances between two correct implementations.

A case is a dict of plain values with a "kind":

  project3d   Projector3D.run: divergence, multigrid solve to a tolerance, gradient update, max|div|,
              wavelet potential recovery of a 3D MAC velocity around spheres
  project2d   Projector2D.run, the same in 2D around circles
  pressure3d  the pressure step alone on a grid of any extents (no recovery): divergence,
              CuMultigridFrac3D.SolveTol, gradient update
  recover3d   CuWaveletPotentialRecover3D.Solve of a divergence-free velocity on a box
  dwt         CuWHHDForward.Solve1D along one axis of an array whose other extents are arbitrary
  sweep3d     CuParallelSweep3D.Solve and Project (sweep + DST-I recovery)
  levelset    CuFastSweeping.ReinitLevelSet and the sub-sampled CuSolidLevelSet3D.GetFrac
  porous3d    CuMultigridFrac3D.Solve_index on a mostly solid domain
  batch       BatchProjector.run on many uneven 2D and 3D grids
  unet        UNetWarmStart.predict and the gradient step of train_step (BF16 network)

Arrays are in the framework's layout: 3D (z, x, y), 2D (x, y), y fastest.  Inputs are made in FP64
from the seed with torch and rounded to the type of the call.
"""
import math

import numpy as np
import torch

from waveletpotentials_b200 import api

DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the headline use: one large projection in mixed precision, five FP32 cycles per FP64 step
        {"name": "project3d 256 mixed", "kind": "project3d", "nx": 256, "ny": 256, "nz": 256, "precision": "mixed",
         "tol": 1e-10, "inner": 5, "solids": 4},
        # an ordinary simulation step in plain single precision
        {"name": "project3d 128 fp32", "kind": "project3d", "nx": 128, "ny": 128, "nz": 128, "precision": "fp32",
         "tol": 1e-6, "inner": 1, "solids": 1},
        # the smallest 3D call: launches and host latency
        {"name": "project3d 32 mixed", "kind": "project3d", "nx": 32, "ny": 32, "nz": 32, "precision": "mixed",
         "tol": 1e-6, "inner": 1, "solids": 1},
        # a 2D flow without solids
        {"name": "project2d 256 fp32", "kind": "project2d", "nx": 256, "ny": 256, "precision": "fp32", "tol": 1e-6,
         "inner": 1, "solids": 0},
        # a pressure solver's grid: no extent a power of two, two of them odd
        {"name": "pressure3d 201x150x101", "kind": "pressure3d", "nx": 201, "ny": 150, "nz": 101, "precision": "mixed",
         "tol": 1e-8, "inner": 2, "solids": 3},
        # recovery of a channel-shaped box from a solver's divergence-free field
        {"name": "recover3d 256x128x64", "kind": "recover3d", "nx": 256, "ny": 128, "nz": 64},
        # analysis of double-precision data along lines of 2^L + 1, the other extents odd
        {"name": "dwt f64 257 lines", "kind": "dwt", "nx": 100, "ny": 257, "nz": 83, "axis": "y", "wavelet": "cdf46",
         "bc": "d", "forward": True, "double": True},
        # the sweep + DST-I recovery at the size of the headline projection
        {"name": "sweep3d 256", "kind": "sweep3d", "nx": 256, "ny": 256, "nz": 256},
        # a moving solid: redistance its level set, then the face fractions of the new position
        {"name": "levelset 160x128x97", "kind": "levelset", "nx": 160, "ny": 128, "nz": 97, "iters": 24, "solids": 3},
        # flow through a porous block, 15% fluid
        {"name": "porous3d 256", "kind": "porous3d", "nx": 256, "ny": 256, "nz": 256, "cycles": 4, "fluid": 0.15},
        # many independent grids of uneven sizes in one launch
        {"name": "batch 64 grids", "kind": "batch", "count3": 32, "count2": 32, "sizes3": "32,64,128",
         "sizes2": "256,512,1024", "tol": 1e-6, "mix": 1},
        # training the warm-start network: forward, loss, backward
        {"name": "unet 64 step", "kind": "unet", "nx": 64, "ny": 64, "nz": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2(rng, lo, hi):
    return 1 << rng.randint(lo.bit_length() - 1, hi.bit_length() - 1)


def draw(rng):
    kind = rng.choice(["project3d", "project3d", "project2d", "pressure3d", "pressure3d", "recover3d", "dwt", "sweep3d",
                       "levelset", "porous3d", "batch", "unet"])
    c = {"kind": kind}
    if kind == "project3d":
        # cubes and boxes; a box keeps its extents within a factor of four
        n = _pow2(rng, 16, 256)
        lo = max(16, n // 4)
        ext = [n, _pow2(rng, lo, n), _pow2(rng, lo, n)]
        rng.shuffle(ext)
        precision = rng.choice(["mixed", "mixed", "fp32", "fp64"])
        # what single precision reaches is 1e-6 on small grids; its rounding floor grows with the extent
        tol = rng.choice([1e-8, 1e-10]) if precision != "fp32" and rng.random() < 0.5 else (1e-6 if precision != "fp32" else 1e-5)
        c.update(nx=ext[0], ny=ext[1], nz=ext[2], precision=precision, tol=tol,
                 inner=rng.choice([1, 2, 5]) if precision == "mixed" else 1, solids=rng.randint(0, 6))
    elif kind == "project2d":
        n = _pow2(rng, 64, 2048)
        precision = rng.choice(["mixed", "fp32"])
        c.update(nx=n, ny=_pow2(rng, max(32, n // 4), n), precision=precision, tol=1e-5 if precision == "fp32" else 1e-6,
                 inner=rng.choice([1, 2]) if precision == "mixed" else 1, solids=rng.randint(0, 4))
    elif kind == "pressure3d":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        n = _log(rng, 20, 240)
        c.update(nx=n, ny=_log(rng, max(16, n // 2), n), nz=_log(rng, max(16, n // 2), n), precision=precision,
                 tol=rng.choice([1e-6, 1e-8]), inner=rng.choice([1, 2, 3]) if precision == "mixed" else 1,
                 solids=rng.randint(0, 5))
    elif kind == "recover3d":
        c.update(nx=_pow2(rng, 16, 256), ny=_pow2(rng, 16, 256), nz=_pow2(rng, 16, 256))
    elif kind == "dwt":
        axis, wavelet = rng.choice("xyz"), rng.choice(["cdf37", "cdf46"])
        n = _pow2(rng, 16, 512) + (1 if wavelet == "cdf46" else 0)
        a = _log(rng, 8, 200)
        b = max(1, min(_log(rng, 8, 200), (1 << 24) // (n * a)))
        ext = {"x": (n, a, b), "y": (a, n, b), "z": (a, b, n)}[axis]
        c.update(nx=ext[0], ny=ext[1], nz=ext[2], axis=axis, wavelet=wavelet, bc=rng.choice("nd"),
                 forward=rng.random() < 0.5, double=rng.random() < 0.4)
    elif kind == "sweep3d":
        if rng.random() < 0.5:
            c.update(nx=_pow2(rng, 16, 256), ny=_pow2(rng, 16, 256), nz=_pow2(rng, 16, 256))
        else:
            c.update(nx=_log(rng, 12, 256), ny=_log(rng, 12, 256), nz=_log(rng, 12, 256))
    elif kind == "levelset":
        n = _log(rng, 24, 160)
        c.update(nx=n, ny=_log(rng, max(16, n // 2), n), nz=_log(rng, max(16, n // 2), n), iters=rng.randint(4, 40),
                 solids=rng.randint(1, 4))
    elif kind == "porous3d":
        n = _log(rng, 32, 256)
        c.update(nx=n, ny=_log(rng, max(24, n // 2), n), nz=_log(rng, max(24, n // 2), n), cycles=rng.randint(1, 4),
                 fluid=round(rng.uniform(0.05, 0.4), 3))
    elif kind == "batch":
        small = rng.random() < 0.5
        c.update(count3=rng.randint(1, 32 if small else 16), count2=rng.randint(1, 32 if small else 16),
                 sizes3="16,32" if small else "32,64,128", sizes2="64,128" if small else "256,512,1024", tol=1e-6,
                 mix=rng.randint(2, 1 << 20))
    else:
        c.update(nx=_pow2(rng, 16, 64), ny=_pow2(rng, 16, 64), nz=4 * rng.randint(4, 16))
    return c


def _dim(case):
    return (case["nx"], case["ny"]) if case["kind"] == "project2d" else (case["nx"], case["ny"], case["nz"])


# ------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * (salt + 1) + seed)
    return g


def _spectral(shape, slope, rms, g):
    """Gaussian random field with power spectrum k^slope and the given RMS (FP64)."""
    spec = torch.fft.rfftn(torch.randn(shape, generator=g, device=DEV, dtype=F64))
    k2 = torch.zeros((), device=DEV, dtype=F64)
    for a, s in enumerate(shape):
        k = (torch.fft.rfftfreq(s, device=DEV, dtype=F64) if a == len(shape) - 1 else torch.fft.fftfreq(s, device=DEV, dtype=F64)) * s
        k2 = k2 + (k * k).reshape([-1 if b == a else 1 for b in range(len(shape))])
    k2.view(-1)[0] = 1.0
    amp = k2.pow_(slope / 4.0)
    amp.view(-1)[0] = 0.0
    f = torch.fft.irfftn(spec * amp, s=shape)
    return f * (rms / f.std(correction=0))


def _axes(nd):
    """Array dimension of the x, y(, z) axes."""
    return (0, 1) if nd == 2 else (1, 2, 0)


def _diff(t, d):
    return t.narrow(d, 1, t.shape[d] - 1) - t.narrow(d, 0, t.shape[d] - 1)


def _spacing(dim):
    return [1.0 / max(dim)] * len(dim)


def _curl3(q, d):
    qx, qy, qz = q
    return [_diff(qz, 2) / d[1] - _diff(qy, 0) / d[2], _diff(qx, 0) / d[2] - _diff(qz, 1) / d[0],
            _diff(qy, 1) / d[0] - _diff(qx, 2) / d[1]]


def _velocity(dim, d, g, phi=True):
    """curl of a random potential (spectra k^-11/3, in 2D k^-3) plus, with phi, the gradient of a random
    scalar (k^-2), no flux through the walls."""
    nd = len(dim)
    ax = _axes(nd)
    if nd == 3:
        nx, ny, nz = dim
        big = (nz + 1, nx + 1, ny + 1)
        q = [_spectral(big, -11.0 / 3.0, 1.0, g)[:, :nx, :], _spectral(big, -11.0 / 3.0, 1.0, g)[:, :, :ny],
             _spectral(big, -11.0 / 3.0, 1.0, g)[:nz]]
        if not phi:  # tangential potential zero on the walls: divergence-free with no wall flux
            for a, c in ((0, q[0]), (2, q[0]), (0, q[1]), (1, q[1]), (1, q[2]), (2, q[2])):
                c.narrow(a, 0, 1).zero_()
                c.narrow(a, c.shape[a] - 1, 1).zero_()
        u = _curl3(q, d)
    else:
        psi = _spectral((dim[0] + 1, dim[1] + 1), -3.0, 1.0, g)
        u = [_diff(psi, 1) / d[1], -_diff(psi, 0) / d[0]]
    if phi:
        cells = [0] * nd
        for a in range(nd):
            cells[ax[a]] = dim[a]
        s = _spectral(tuple(cells), -2.0, 1.0 if nd == 3 else 0.5, g)
        for a in range(nd):
            u[a].narrow(ax[a], 1, dim[a] - 1).add_(_diff(s, ax[a]) / d[a])
            u[a].narrow(ax[a], 0, 1).zero_()
            u[a].narrow(ax[a], dim[a], 1).zero_()
    return u


def _solids(dim, h, count, rng):
    """Signed distance (positive in the fluid) of `count` random spheres or circles."""
    nd = len(dim)
    ax = _axes(nd)
    pos = [((torch.arange(dim[a], device=DEV, dtype=F64) + 0.5) * h).reshape([-1 if b == ax[a] else 1 for b in range(nd)]) for a in range(nd)]
    small = min(dim) * h
    out = None
    for _ in range(count):
        r = rng.uniform(0.05, 0.15) * small
        d2 = sum((p - rng.uniform(r + 0.02 * small, n * h - r - 0.02 * small)) ** 2 for p, n in zip(pos, dim))
        s = torch.sqrt(d2) - r
        out = s if out is None else torch.minimum(out, s)
    if out is None:
        out = torch.full([dim[ax.index(b)] for b in range(nd)], 10.0, device=DEV, dtype=F64)
    return out


def _fractions(sdf, h):
    """Open share of each face from the level set in the two cells beside it."""
    nd = sdf.dim()
    out = []
    for d in _axes(nd):
        n = sdf.shape[d]
        lo = torch.cat([sdf.narrow(d, 0, 1), sdf], d)
        hi = torch.cat([sdf, sdf.narrow(d, n - 1, 1)], d)
        t = (1.0 - (hi + lo) / torch.sqrt(torch.clamp(h * h - (hi - lo) ** 2, min=1e-14))) * 0.5
        out.append((1.0 - t.clamp(0.0, 1.0)).float())
    return out


def _flow(dim, seed, solids, salt=0):
    """(velocity, face fractions, level set, spacing) of a projection, rounded to FP32."""
    import random
    d = _spacing(dim)
    sdf = _solids(dim, d[0], solids, random.Random(7919 * seed + salt))
    u = [t.float().contiguous() for t in _velocity(dim, d, _gen(seed, salt))]
    return u, [a.contiguous() for a in _fractions(sdf, d[0])], sdf, d[0]


def _porous(case, seed):
    """Balls of fluid in a solid block: face fractions (cut faces of random area) and a right-hand
    side that sums to zero over each level's cells with open faces."""
    import random
    dim = _dim(case)
    nx, ny, nz = dim
    g, r = _gen(seed, 5), random.Random(31 * seed + 5)
    z, x, y = [torch.arange(n, device=DEV, dtype=torch.float32).add_(0.5).reshape([-1 if b == a else 1 for b in range(3)]) for a, n in enumerate((nz, nx, ny))]
    fluid = torch.zeros((nz, nx, ny), device=DEV, dtype=torch.bool)
    for _ in range(4000):
        for _ in range(16):
            rad = r.uniform(0.04, 0.1) * min(dim)
            fluid |= (x - r.uniform(0, nx)) ** 2 + (y - r.uniform(0, ny)) ** 2 + (z - r.uniform(0, nz)) ** 2 < rad * rad
        if float(fluid.float().mean()) >= case["fluid"]:
            break
    m, faces = fluid.float(), []
    for d in _axes(3):
        n = m.shape[d]
        lo, hi = torch.cat([m.narrow(d, 0, 1), m], d), torch.cat([m, m.narrow(d, n - 1, 1)], d)
        part = torch.rand(lo.shape, generator=g, device=DEV) * 0.7 + 0.2
        faces.append(torch.where(lo * hi > 0, torch.ones_like(lo), torch.where(lo + hi > 0, part, torch.zeros_like(lo))).contiguous())
    f = torch.randn((nz, nx, ny), generator=g, device=DEV) * m
    f = torch.where(fluid, f - f.sum() / m.sum(), torch.zeros_like(f))
    return fluid, faces, f.contiguous()


def _batch_grids(case, seed):
    import random
    r = random.Random(case["mix"])
    s3, s2 = [int(v) for v in case["sizes3"].split(",")], [int(v) for v in case["sizes2"].split(",")]
    grids = []
    for i in range(case["count3"] + case["count2"]):
        n = r.choice(s3 if i < case["count3"] else s2)
        grids.append((((n,) * (3 if i < case["count3"] else 2)), r.randint(0, 4)))
    return [(dim,) + _flow(dim, seed, k, 100 + i)[:2] + (1.0 / dim[0],) for i, (dim, k) in enumerate(grids)]


def _unet_data(case, seed):
    import random
    dim = _dim(case)
    h = 1.0 / case["nx"]
    g = _gen(seed, 9)
    cells = (dim[2], dim[0], dim[1])
    sdf = _solids(dim, h, 3, random.Random(seed)).float().contiguous()
    b = _spectral(cells, -2.0, 30.0, g).float()
    p = _spectral(cells, -4.0, 0.5, g).float()
    return b.contiguous(), sdf, p.contiguous(), h


def _dwt_data(case, seed):
    t = torch.randn((case["nz"], case["nx"], case["ny"]), generator=_gen(seed, 3), device=DEV, dtype=F64)
    return t if case["double"] else t.float()


def _levelset_data(case, seed):
    """A level set that has lost its unit slope, as advection leaves it."""
    import random
    dim, h = _dim(case), 1.0 / case["nx"]
    sdf = _solids(dim, h, case["solids"], random.Random(seed))
    wave = _spectral(tuple(sdf.shape), -4.0, 0.2, _gen(seed, 4))
    return (sdf * (1.0 + wave.clamp(-0.6, 0.6))).float().contiguous(), h


# ------------------------------------------------------------------ the calls
_PREC = {"fp32": api.PREC_FP32, "mixed": api.PREC_MIXED, "fp64": api.PREC_FP64}
_WAV = {"cdf37": api.CDF3_7, "cdf46": api.CDF4_6}


def _packed(shapes):
    """One zeroed allocation and a view of each shape in it, every view on a 256-byte boundary."""
    size = [(math.prod(v) + 63) // 64 * 64 for v in shapes]
    flat = torch.zeros(sum(size), device=DEV)
    return flat, [t[:math.prod(v)].view(v) for t, v in zip(flat.split(size), shapes)]


def _empty(shapes, names):
    return [torch.zeros(shapes[k], device=DEV) for k in names]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("project3d", "project2d", "pressure3d"):
        dim = _dim(case)
        u0, a, _, h = _flow(dim, seed, case["solids"])
        s = {"u0": u0, "u": [torch.empty_like(t) for t in u0], "a": a, "h": h, "dim": dim}
        opts = dict(rel_tol=case["tol"], max_cycles=100, precision=_PREC[case["precision"]], inner_cycles=case["inner"])
        if kind == "project3d":
            s["pr"] = api.Projector3D(*a, dim, h, **opts)
            s["q"] = _empty(api.mac_shapes3d(*dim), ("qx", "qy", "qz"))
        elif kind == "project2d":
            s["pr"] = api.Projector2D(*a, dim, h, **opts)
            s["q"] = _empty(api.mac_shapes2d(*dim), ("qz",))
        else:
            s["mg"], s["opts"] = api.CuMultigridFrac3D(*a, dim, h), opts
            s["mg"].Autotune()
            s["b"], s["p"] = _empty(api.mac_shapes3d(*dim), ("p", "p"))
        return s
    if kind == "recover3d":
        dim = _dim(case)
        d = [1.0 / n for n in dim]
        return {"rec": api.CuWaveletPotentialRecover3D(dim, d),
                "u": [t.float().contiguous() for t in _velocity(dim, d, _gen(seed), phi=False)],
                "q": _empty(api.mac_shapes3d(*dim), ("qx", "qy", "qz"))}
    if kind == "dwt":
        src = _dwt_data(case, seed)
        n = {"x": case["nx"], "y": case["ny"], "z": case["nz"]}[case["axis"]]
        return {"src": src, "dst": torch.empty_like(src), "dim": _dim(case), "level": n.bit_length() - 1, "axis": case["axis"],
                "bc": case["bc"], "wavelet": _WAV[case["wavelet"]], "forward": case["forward"]}
    if kind == "sweep3d":
        dim = _dim(case)
        h = 1.0 / case["nx"]
        return {"sw": api.CuParallelSweep3D(dim, h),
                "u": [t.float().contiguous() for t in _velocity(dim, [h] * 3, _gen(seed), phi=False)],
                "q": _empty(api.mac_shapes3d(*dim), ("qx", "qy", "qz"))}
    if kind == "levelset":
        dim = _dim(case)
        ls, h = _levelset_data(case, seed)
        return {"ls0": ls, "ls": torch.empty_like(ls), "h": h, "sls": api.CuSolidLevelSet3D(dim, h), "dim": dim, "iters": case["iters"],
                "a": _empty(api.mac_shapes3d(*dim), ("xv", "yv", "zv"))}
    if kind == "porous3d":
        dim = _dim(case)
        _, a, f = _porous(case, seed)
        return {"mg": api.CuMultigridFrac3D(*a, dim, 1.0), "f": f, "p": torch.zeros_like(f), "cycles": case["cycles"]}
    if kind == "batch":
        made = _batch_grids(case, seed)
        grids = [dict(zip(("ax", "ay", "az"), a), dim=dim, dx=h) for dim, _, a, h in made]
        # the program keeps each quantity of all its grids in one allocation
        names = [(api.mac_shapes3d(*dim), ("qx", "qy", "qz")) if len(dim) == 3 else (api.mac_shapes2d(*dim), ("qz",)) for dim, _, _, _ in made]
        src, u0 = _packed([t.shape for _, v, _, _ in made for t in v])
        for t, v in zip(u0, [t for _, v, _, _ in made for t in v]):
            t.copy_(v)
        dst, u = _packed([t.shape for t in u0])
        out, q = _packed([sh[k] for sh, keys in names for k in keys])
        take = lambda ts, counts: [[ts.pop(0) for _ in range(n)] for n in counts]
        u0, u, q = take(u0, [len(g[0]) for g in made]), take(u, [len(g[0]) for g in made]), take(q, [len(n[1]) for n in names])
        bp = api.BatchProjector(grids, rel_tol=case["tol"])
        bp.plan(u0)
        return {"bp": bp, "grids": grids, "u": u, "q": q, "src": src, "dst": dst, "out": out}
    b, sdf, p, h = _unet_data(case, seed)
    net = api.UNetWarmStart(_dim(case), seed=seed % 1000)
    return {"net": net, "b": b, "sdf": sdf, "p": p, "h": h, "guess": torch.zeros_like(b)}


def run(state):
    s = state
    if "bp" in s:
        s["dst"].copy_(s["src"])  # the projection works in place; the program keeps its input
        s["bp"].run(s["u"], s["q"])
        s["bp"].results()
        return [s["dst"], s["out"]]
    if "pr" in s:
        torch._foreach_copy_(s["u"], s["u0"])
        s["pr"].run(*s["u"], *s["q"])
        return s["u"] + s["q"]
    if "rec" in s:
        s["rec"].Solve(*s["q"], *s["u"])
        return s["q"]
    if "sw" in s:
        s["sw"].Solve(*s["q"], *s["u"])
        s["sw"].Project(*s["q"])
        return s["q"]
    if "sls" in s:
        s["ls"].copy_(s["ls0"])
        api.CuFastSweeping.ReinitLevelSet(s["ls"], s["dim"], s["h"], s["iters"])
        s["sls"].GetFrac(*s["a"], s["ls"], s["dim"], s["h"])
        return [s["ls"]] + s["a"]
    if "net" in s:
        s["net"].predict(s["guess"], s["b"], s["sdf"], s["h"])
        loss = s["net"].train_step(s["b"], s["sdf"], s["p"], s["h"], 0.0)
        return [s["guess"], loss, s["net"].params(1)]
    if "opts" in s:
        torch._foreach_copy_(s["u"], s["u0"])
        api.CuConvergence.GetB_3d_frac_vel(s["b"], *s["u"], *s["a"], s["dim"], s["h"])
        s["mg"].SolveTol(s["p"], None, s["b"], raise_on_fail=False, **s["opts"])
        api.CuGradient.SubtractGradient3D_Frac_P64(*s["u"], s["mg"].Iterate64Ptr(), *s["a"], s["dim"], s["h"])
        return s["u"]
    if "mg" in s:
        s["mg"].Solve_index(s["p"], None, s["f"], s["cycles"], 2, 2, 2.0 / 3.0)
        return s["p"]
    api.CuWHHDForward.Solve1D(s["dst"], s["src"], s["dim"], s["level"], s["axis"], s["bc"], s["wavelet"], s["forward"])
    return s["dst"]


# ------------------------------------------------------------------ results in 64 bits
# One level of the lifting on pairs a[k] = x[2k], d[k] = x[2k+1]; the base level is a small matrix.
_U37 = [-0.003797743055556, 0.032552083333333, -0.137044270833333, 0.444444444444444, 0.137044270833333,
        -0.032552083333333, 0.003797743055556]
_U46 = [0.008544921875, -0.064697265625, 0.24365234375, 0.24365234375, -0.064697265625, 0.008544921875]
_H3 = [[-0.353553390593274, 0.530330085889911, -0.176776695296637, 0], [0, 0.176776695296637, -0.530330085889911, 0.353553390593274]]
_BASE = {
    ("cdf37", "n"): [[0.5] * 4, [-0.39990234375, -0.2001953125, 0.2001953125, 0.39990234375]] + _H3,
    ("cdf37", "d"): [[0.80078125, 1.599609375, 1.599609375, 0.80078125], [-1, -1, 1, 1],
                     [-0.707106781186548] + _H3[0][1:], _H3[1][:3] + [0.707106781186548]],
    ("cdf46", "n"): [[1.8515625, 2.09765625, 0.5, -1.09765625, -1.3515625], [-1.3515625, -1.09765625, 0.5, 2.09765625, 1.8515625],
                     [1, 0, -2, 0, 1], [0.353553390593274, -0.618718433538229, 0.353553390593274, -0.088388347648318, 0],
                     [0, -0.088388347648318, 0.353553390593274, -0.618718433538229, 0.353553390593274]],
    ("cdf46", "d"): [[2.102851867675782, 0, 0, 0, 0], [0, 0, 0, 0, 2.102851867675782],
                     [0.68310546875, -0.19970703125, -0.400390625, -0.19970703125, 0.68310546875],
                     [0.353553390593274, -0.441941738241592, 0.353553390593274, -0.088388347648318, 0],
                     [0, -0.088388347648318, 0.353553390593274, -0.441941738241592, 0.353553390593274]],
}
_MATRICES = {}


def _analysis(n, wavelet, bc):
    """The n x n matrix of the full-depth analysis (numpy FP64): CDF3.7 on lines of 2^L, reflected about
    the half samples, CDF4.6 on lines of 2^L + 1, about the end samples."""
    if (n, wavelet, bc) in _MATRICES:
        return _MATRICES[n, wavelet, bc]
    ext = n & 1
    x, length, details = np.eye(n), n - ext, []
    while length > 4:
        k = np.arange(-8, length // 2 + ext + 8)
        idx = np.stack([2 * k, 2 * k + 1])
        sign = np.ones(idx.shape)
        if wavelet == "cdf37":
            out = (idx < 0) | (idx >= length)
            idx = np.where(idx < 0, -1 - idx, np.where(idx >= length, 2 * length - 1 - idx, idx))
        else:
            out = (idx < 0) | (idx > length)
            idx = np.where(idx < 0, -idx, np.where(idx > length, 2 * length - idx, idx))
        if bc == "d":
            sign[out] = -1.0
        ok = (idx >= 0) & (idx < x.shape[0])
        a, d = [np.where(ok[i], sign[i], 0.0)[:, None] * x[np.clip(idx[i], 0, x.shape[0] - 1)] for i in (0, 1)]
        a1, d1 = a.copy(), d.copy()
        if wavelet == "cdf37":
            a1[1:] -= d[:-1] / 3.0
            d1[:-1] += -0.375 * a1[1:] - 1.125 * a1[:-1]
            taps = [(t, _U37[3 - t]) for t in range(-3, 4)]
            sa, sd = 3.0 / math.sqrt(2.0), math.sqrt(2.0) / 3.0
        else:
            a1[1:] -= 0.25 * (d[:-1] + d[1:])
            d1[:-1] -= a1[:-1] + a1[1:]
            taps = [(t, _U46[2 - t]) for t in range(-3, 3)]
            sa, sd = 2.0 * math.sqrt(2.0), -0.5 / math.sqrt(2.0)
        na, nd = length // 2 + ext, length // 2
        s = a1[8:8 + na].copy()
        for t, c in taps:
            s += c * d1[8 + t:8 + t + na]
        details.insert(0, d1[8:8 + nd] * sd)
        x, length = s * sa, length // 2
    x = np.concatenate([np.array(_BASE[wavelet, bc]) @ x] + details)
    _MATRICES[n, wavelet, bc] = x
    return x


def _apply(m, t, d):
    m = torch.as_tensor(m, device=t.device)
    return torch.movedim(torch.tensordot(m, t, dims=([1], [d])), 0, d)


def _norms(n, wavelet, bc):
    return torch.as_tensor((np.linalg.inv(_analysis(n, wavelet, bc)) ** 2).sum(0), device=DEV)


def _wav(n, cells):
    """Along an axis, cells + 1 samples are a div (CDF4.6, 'd') line and cells samples a curl one."""
    return ("cdf46", "d") if n == cells + 1 else ("cdf37", "n")


def _lwt(t, dim, inverse):
    for a, d in enumerate(_axes(len(dim))):
        m = _analysis(t.shape[d], *_wav(t.shape[d], dim[a]))
        t = _apply(np.linalg.inv(m) if inverse else m, t, d)
    return t


def _level_scale(n, h, sh):
    """s = 4 / (h 2^j) of each coefficient index, j = L + 1 - bitlength(index)."""
    lev = n.bit_length() - 1
    return torch.tensor([4.0 / h / (2.0 ** (lev + 1 - i.bit_length()) + 1e-12) for i in range(n)], device=DEV, dtype=F64).reshape(sh)


def _recover(u, dim, d):
    """The vector (3D) or scalar (2D) potential of a velocity by local projection in coefficient space."""
    nd = len(dim)
    ax = _axes(nd)
    v = [_lwt(t.double(), dim, False) for t in u]
    sh = [[-1 if b == ax[a] else 1 for b in range(nd)] for a in range(nd)]
    s = [_level_scale(dim[a], d[a], sh[a]) for a in range(nd)]
    ipc = [_norms(dim[a], "cdf37", "n").reshape(sh[a]) for a in range(nd)]
    ipd = [_norms(dim[a] + 1, "cdf46", "d")[1:].reshape(sh[a]) for a in range(nd)]
    v = [v[a].narrow(ax[a], 1, dim[a]) for a in range(nd)]
    if nd == 2:
        wx, wy = s[0] * ipc[0] * ipd[1], s[1] * ipd[0] * ipc[1]
        p = (v[0] * wy - v[1] * wx) / (s[0] * wx + s[1] * wy + 1e-12)
        p[0] = 0.0
        p[:, 0] = 0.0
        return [_lwt(torch.nn.functional.pad(p, (1, 0, 1, 0)), dim, True)]
    (x, y, z), (sx, sy, sz) = v, s
    inv = 1.0 / (sx * sx + sy * sy + sz * sz)
    qx, qy, qz = (sz * y - sy * z) * inv, (sx * z - sz * x) * inv, (sy * x - sx * y) * inv

    def ratio(a, b, c):
        """One component on the plane where the index along c is 0: the other two weighted by the norms."""
        wa = s[a] * ipc[a] * ipd[b] * ipc[c]
        wb = s[b] * ipd[a] * ipc[b] * ipc[c]
        return ((v[a] * wb - v[b] * wa) / (s[a] * wa + s[b] * wb + 1e-12)).narrow(ax[c], 0, 1)
    for q, (a, b, c) in ((qx, (1, 2, 0)), (qy, (2, 0, 1)), (qz, (0, 1, 2))):
        for e in range(3):
            q.narrow(ax[e], 0, 1).zero_()
        w = ratio(a, b, c)
        for e in (a, b):
            w.narrow(ax[e], 0, 1).zero_()
        q.narrow(ax[c], 0, 1).copy_(w)
    pad = lambda t, dims: torch.nn.functional.pad(t, [v for b in (2, 1, 0) for v in (1 if b in dims else 0, 0)])
    return [_lwt(pad(q, [ax[e] for e in range(3) if e != c]), dim, True) for c, q in enumerate((qx, qy, qz))]


def _divergence(flux, d):
    return sum(_diff(f, ax) / h for f, ax, h in zip(flux, _axes(len(flux)), d))


def _project(u, a, dim, d):
    """u - grad p times the face fractions, p from conjugate gradients in FP64 (preconditioned by the
    cosine-transform solve of the open domain plus the diagonal)."""
    nd = len(dim)
    ax = _axes(nd)
    u, a = [t.double() for t in u], [t.double() for t in a]
    w = []
    for t, x in zip(a, ax):
        t = t.clone()
        t.narrow(x, 0, 1).zero_()
        t.narrow(x, t.shape[x] - 1, 1).zero_()
        w.append(t)
    grad = lambda p: [torch.nn.functional.pad(_diff(p, x) / h, [v for b in range(nd - 1, -1, -1) for v in ((1, 1) if b == x else (0, 0))]) for x, h in zip(ax, d)]
    op = lambda p: -_divergence([t * g for t, g in zip(w, grad(p))], d)
    diag = sum((t.narrow(x, 1, t.shape[x] - 1) + t.narrow(x, 0, t.shape[x] - 1)) / (h * h) for t, x, h in zip(w, ax, d))
    act = diag > 1e-12
    inv_diag = torch.where(act, 1.0 / diag.clamp(min=1e-300), torch.zeros_like(diag))
    basis, lam = [], 0.0
    for n, x, h in zip(dim, ax, d):
        k = torch.arange(n, device=DEV, dtype=F64)
        c = torch.cos(math.pi * k[:, None] * (k[None, :] + 0.5) / n) * math.sqrt(2.0 / n)
        c[0] /= math.sqrt(2.0)
        basis.append(c)
        lam = lam + ((2.0 - 2.0 * torch.cos(math.pi * k / n)) / (h * h)).reshape([-1 if b == x else 1 for b in range(nd)])
    lam[(0,) * nd] = 1.0

    def precond(r):
        t = r
        for c, x in zip(basis, ax):
            t = _apply(c, t, x)
        t = t / lam
        t[(0,) * nd] = 0.0
        for c, x in zip(basis, ax):
            t = _apply(c.T, t, x)
        return torch.where(act, t + 0.25 * r * inv_diag, torch.zeros_like(t))
    b = torch.where(act, -_divergence([t * v for t, v in zip(a, u)], d), torch.zeros_like(diag))
    b = torch.where(act, b - b.sum() / act.sum(), b)
    p, r = torch.zeros_like(b), b.clone()
    z = precond(r)
    q, rz, stop = z.clone(), float((r * z).sum()), 1e-13 * float(b.norm())
    for _ in range(400):
        aq = op(q)
        al = rz / float((q * aq).sum())
        p += al * q
        r -= al * aq
        if float(r.norm()) <= stop:
            break
        r = torch.where(act, r - r.sum() / act.sum(), r)
        z = precond(r)
        new = float((r * z).sum())
        q, rz = z + (new / rz) * q, new
    return [(v - torch.where(t > 1e-12, g, torch.zeros_like(g))) * f for v, g, t, f in zip(u, grad(p), w, a)]


def _sweep(u, dim, h):
    nx, ny, nz = dim
    u = [t.double() for t in u]
    pad0 = lambda t, d: torch.nn.functional.pad(t, [v for b in (2, 1, 0) for v in (1 if b == d else 0, 0)])
    qx, qy = pad0(torch.cumsum(u[1], 0) * h, 0), pad0(-torch.cumsum(u[0], 0) * h, 0)
    qz = torch.zeros((nz, nx + 1, ny + 1), device=DEV, dtype=F64)
    qz[-1, 1:] = -torch.cumsum(qx[-1], 0)
    qx[-1] = 0.0
    qy[-1] = 0.0
    phi = -(_diff(qx[1:-1, :, 1:-1], 1) + _diff(qy[1:-1, 1:-1], 2) + _diff(qz[:, 1:-1, 1:-1], 0)) / h
    lam = 0.0
    for n, d in zip(dim, _axes(3)):
        k = torch.arange(1, n, device=DEV, dtype=F64)
        phi = _apply(torch.sin(math.pi * k[:, None] * k[None, :] / n) * (2.0 / n), phi, d)
        lam = lam + (2.0 - 2.0 * torch.cos(math.pi * k / n)).reshape([-1 if b == d else 1 for b in range(3)])
    phi = phi * (h * h) / lam
    for n, d in zip(dim, _axes(3)):
        k = torch.arange(1, n, device=DEV, dtype=F64)
        phi = _apply(torch.sin(math.pi * k[:, None] * k[None, :] / n), phi, d)
    phi = torch.nn.functional.pad(phi, (1, 1, 1, 1, 1, 1))
    return [qx - _diff(phi, 1) / h, qy - _diff(phi, 2) / h, qz - _diff(phi, 0) / h]


def _eikonal(ls, iters, h):
    for _ in range(iters):
        m = []
        for d in (1, 2, 0):
            n = ls.shape[d]
            big = torch.full_like(ls.narrow(d, 0, 1), 1e8)
            m.append(torch.minimum(torch.cat([big, ls.narrow(d, 0, n - 1)], d), torch.cat([ls.narrow(d, 1, n - 1), big], d)))
        m = torch.sort(torch.stack(m), 0).values
        r = m[0] + h
        two = 0.5 * (m[0] + m[1] + torch.sqrt((2 * h * h - (m[0] - m[1]) ** 2).clamp(min=0)))
        r = torch.where(r > m[1], two, r)
        s, ss = m.sum(0), (m * m).sum(0)
        three = (s + torch.sqrt((s * s - 3.0 * (ss - h * h)).clamp(min=0))) / 3.0
        r = torch.where((m[0] + h > m[1]) & (two > m[2]), three, r)
        ls = torch.where(ls > -1e-12, r, ls)
    return ls


def _corners(ls, pos, quadratic):
    """ls interpolated at cell-index positions pos (three (N,) tensors in x, y, z order)."""
    nx, ny, nz = ls.shape[1], ls.shape[2], ls.shape[0]
    base, wt = [], []
    for p, n in zip(pos, (nx, ny, nz)):
        if quadratic:
            i = torch.floor(p - 0.5)
            f = p - i
            wt.append([0.5 * (1.5 - f) ** 2, 0.75 - (f - 1.0) ** 2, 0.5 * (f - 0.5) ** 2])
            base.append([(i.long() + k).clamp(0, n - 1) for k in range(3)])
        else:
            p = p.clamp(min=1e-10)
            i = p.long().clamp(max=n - 2)
            f = torch.where(p.long() >= n - 1, torch.ones_like(p), p - i)
            wt.append([1 - f, f])
            base.append([i, i + 1])
    out, flat = 0.0, ls.reshape(-1)
    for k, wz in enumerate(wt[2]):
        for j, wx in enumerate(wt[0]):
            for i, wy in enumerate(wt[1]):
                out = out + wx * wy * wz * flat[base[1][i] + base[0][j] * ny + base[2][k] * (nx * ny)]
    return out


def _subsampled(ls, dim, h):
    ls, out = ls.double(), []
    for a in range(3):
        ext = [dim[e] + (1 if e == a else 0) for e in range(3)]
        res = torch.zeros((ext[2], ext[0], ext[1]), device=DEV, dtype=F64).reshape(-1)
        cut = []
        for part in torch.arange(res.numel(), device=DEV).split(1 << 22):
            y, x, z = part % ext[1], (part // ext[1]) % ext[0], part // (ext[0] * ext[1])
            c = [i.double() + (0.0 if e == a else 0.5) - 0.5 for e, i in enumerate((x, y, z))]
            v = _corners(ls, c, True)
            res[part] = (v > h).double()
            cut.append(part[(v <= h) & (v > -h)])
        k = (torch.arange(128, device=DEV, dtype=F64) + 0.5) / 128.0
        for part in torch.cat(cut).split(1024):
            y, x, z = part % ext[1], (part // ext[1]) % ext[0], part // (ext[0] * ext[1])
            c = [i.double() for i in (x, y, z)]
            others = [e for e in range(3) if e != a]
            sub = {others[0]: k.repeat(128), others[1]: k.repeat_interleave(128)}
            pos = [((c[e][:, None] + sub[e][None, :]) if e != a else c[e][:, None].expand(-1, 16384)).reshape(-1) - 0.5 for e in range(3)]
            res[part] = (_corners(ls, pos, False) > 0).reshape(-1, 16384).double().mean(1)
        out.append(res.reshape(ext[2], ext[0], ext[1]))
    return out


def _coarse_faces(t, cells, main):
    for a, d in enumerate(_axes(3)):
        n = t.shape[d]
        if a == main:
            idx = [min(2 * i, n - 1) if n & 1 or 2 * i < n else 2 * i - 1 for i in range((n >> 1) + 1)]
            t = t.index_select(d, torch.tensor(idx, device=DEV))
        else:
            lo, hi = torch.arange(0, n, 2, device=DEV), torch.arange(0, n, 2, device=DEV)
            hi = torch.clamp(hi + 1, max=n - 1)
            t = 0.5 * (t.index_select(d, lo) + t.index_select(d, hi))
    return t


def _porous_cycles(faces, f, dim, cycles, om=2.0 / 3.0, nu=2):
    """Index-sparse V-cycles: sweeps, residuals and corrections on the cells with an open face; the
    residual workspace is one array that the levels share; 50 sweeps on the coarsest level."""
    ax = _axes(3)
    levels, n, a = [], list(dim), [t.double() for t in faces]
    d = [torch.ones(v, device=DEV, dtype=F64) for v in dim]
    while min(n) > 1:
        col = lambda t, e: t.reshape([-1 if b == ax[e] else 1 for b in range(3)])
        c = []
        act = torch.zeros([n[2], n[0], n[1]], device=DEV, dtype=torch.bool)
        for e in range(3):
            t, x = a[e], ax[e]
            act |= (t.narrow(x, 0, n[e]) >= 1e-12) | (t.narrow(x, 1, n[e]) >= 1e-12)
            lo, hi = torch.zeros(n[e], device=DEV, dtype=F64), torch.zeros(n[e], device=DEV, dtype=F64)
            lo[1:] = 2.0 / (d[e][:-1] + d[e][1:]) / d[e][1:]
            hi[:-1] = 2.0 / (d[e][:-1] + d[e][1:]) / d[e][:-1]
            c += [t.narrow(x, 0, n[e]) * col(lo, e), t.narrow(x, 1, n[e]) * col(hi, e)]
        levels.append({"c": c, "diag": sum(c), "act": act, "d": [col(t, e) for e, t in enumerate(d)], "n": list(n), "any": bool(act.any())})
        a = [_coarse_faces(a[e], n, e) for e in range(3)]
        d = [torch.nn.functional.pad(t, (0, t.numel() & 1)).reshape(-1, 2).sum(1) for t in d]
        n = [(v + 1) // 2 for v in n]

    def off(L, v):
        out = 0.0
        for e in range(3):
            x, m = ax[e], v.shape[ax[e]]
            z = torch.zeros_like(v.narrow(x, 0, 1))
            out = out + L["c"][2 * e] * torch.cat([z, v.narrow(x, 0, m - 1)], x) + L["c"][2 * e + 1] * torch.cat([v.narrow(x, 1, m - 1), z], x)
        return out

    def sweep(L, v, f, where):
        new = torch.where(L["diag"] > 1e-12, (1.0 - om) * v + om * (f + off(L, v)) / L["diag"].clamp(min=1e-300), torch.zeros_like(v))
        return torch.where(where, new, v)
    work = torch.zeros(f.numel(), device=DEV, dtype=F64)

    def cycle(l, v, f):
        L = levels[l]
        if l + 1 >= len(levels) or not levels[l + 1]["any"]:
            for _ in range(50):
                v = sweep(L, v, f, torch.ones_like(L["act"]))
            return v
        for _ in range(nu):
            v = sweep(L, v, f, L["act"])
        r = torch.where(L["diag"] > 1e-12, f - (L["diag"] * v - off(L, v)), torch.zeros_like(v))
        own = work[:v.numel()].view(v.shape)
        own.copy_(torch.where(L["act"], r, own))
        r = own
        K = levels[l + 1]
        for e in (1, 0, 2):
            x, m = ax[e], r.shape[ax[e]]
            w = L["d"][e]
            num, den = r * w, w
            if m & 1:
                num = torch.cat([num, torch.zeros_like(num.narrow(x, 0, 1))], x)
                den = torch.cat([den, torch.zeros_like(den.narrow(x, 0, 1))], x)
            ev = torch.arange(0, num.shape[x], 2, device=DEV)
            r = (num.index_select(x, ev) + num.index_select(x, ev + 1)) / (den.index_select(x, ev) + den.index_select(x, ev + 1))
        fc = torch.where(K["act"], r, torch.zeros_like(r))
        vc = cycle(l + 1, torch.zeros_like(fc), fc)
        for e in range(3):
            vc = vc.index_select(ax[e], torch.arange(L["n"][e], device=DEV) // 2)
        v = torch.where(L["act"], v + vc, v)
        for _ in range(nu):
            v = sweep(L, v, f, L["act"])
        return v
    v = torch.zeros_like(f, dtype=F64)
    for _ in range(cycles):
        v = cycle(0, v, f.double())
    return v


_UNET = [(16, 0, 16), (16, 0, 16), (16, 0, 32), (32, 0, 32), (32, 0, 64), (64, 0, 64), (32, 64, 32), (32, 0, 32), (16, 32, 16), (16, 0, 16)]


def _unet_exact(vec, b, sdf, p, h):
    import torch.nn.functional as F
    vec = torch.as_tensor(vec, device=DEV, dtype=F64).requires_grad_()
    off, convs = 0, []
    for c0, c1, co in _UNET:
        ws = []
        for c in (c0, c1):
            if c:  # [27][cout][cin], taps in (z, x, y) order
                ws.append(vec[off:off + 27 * co * c].reshape(3, 3, 3, co, c).permute(3, 4, 0, 1, 2))
                off += 27 * co * c
        convs.append((torch.cat(ws, 1), vec[off:off + co]))
        off += co
    head = vec[off:]
    b, sdf, p = b.double(), sdf.double(), p.double()
    rms = b.square().mean().sqrt()
    x = torch.zeros((1, 16) + tuple(b.shape), device=DEV, dtype=F64)
    x[0, 0], x[0, 1] = b / rms, (sdf / (4.0 * h)).clamp(-1.0, 1.0)

    def conv(i, t):
        w, bias = convs[i]
        out = bias.reshape(1, -1, 1, 1, 1)
        t = F.pad(t, (1, 1, 1, 1, 1, 1))
        n = b.shape
        ext = [t.shape[k + 2] - 2 for k in range(3)]
        for k in range(27):  # one tap at a time: a plain matrix product in FP64
            dz, dx, dy = k // 9, (k // 3) % 3, k % 3
            out = out + torch.einsum("oc,bczxy->bozxy", w[:, :, dz, dx, dy], t[:, :, dz:dz + ext[0], dx:dx + ext[1], dy:dy + ext[2]])
        return torch.relu(out)
    up = lambda t: t.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
    s1 = conv(1, conv(0, x))
    s2 = conv(3, conv(2, F.avg_pool3d(s1, 2)))
    e3 = conv(5, conv(4, F.avg_pool3d(s2, 2)))
    e2 = conv(7, conv(6, torch.cat([s2, up(e3)], 1)))
    e1 = conv(9, conv(8, torch.cat([s1, up(e2)], 1)))
    pred = torch.einsum("c,czxy->zxy", head[:16], e1[0]) + head[16]
    scale = 4.0 * math.pi ** 2 / (b.shape[1] * h) ** 2
    fluid = sdf > 0
    r = (pred - p * scale / rms)[fluid]
    loss = (r - r.mean()).square().mean()
    (grad,) = torch.autograd.grad(loss, vec)
    return [(pred * rms / scale).detach(), float(loss.detach()), grad.cpu().numpy()]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("project3d", "project2d", "pressure3d"):
        dim = _dim(case)
        u, a, _, h = _flow(dim, seed, case["solids"])
        u = _project(u, a, dim, [h] * len(dim))
        return u if kind == "pressure3d" else u + _recover(u, dim, [h] * len(dim))
    if kind == "recover3d":
        dim = _dim(case)
        d = [1.0 / n for n in dim]
        return _recover([t.float() for t in _velocity(dim, d, _gen(seed), phi=False)], dim, d)
    if kind == "dwt":
        t = _dwt_data(case, seed)
        d = {"x": 1, "y": 2, "z": 0}[case["axis"]]
        m = _analysis(t.shape[d], case["wavelet"], case["bc"])
        return _apply(m if case["forward"] else np.linalg.inv(m), t.double(), d)
    if kind == "sweep3d":
        dim = _dim(case)
        h = 1.0 / case["nx"]
        return _sweep([t.float() for t in _velocity(dim, [h] * 3, _gen(seed), phi=False)], dim, h)
    if kind == "levelset":
        ls, h = _levelset_data(case, seed)
        ls = _eikonal(-_eikonal(-ls.double(), case["iters"], h), case["iters"], h)
        return [ls] + _subsampled(ls, _dim(case), h)
    if kind == "porous3d":
        _, a, f = _porous(case, seed)
        return _porous_cycles(a, f, _dim(case), case["cycles"])
    if kind == "batch":
        us, qs = [], []
        pack = lambda ts: torch.cat([torch.nn.functional.pad(t.reshape(-1), (0, -t.numel() % 64)) for t in ts])
        for dim, u, a, h in _batch_grids(case, seed):
            us.append(_project(u, a, dim, [h] * len(dim)))
            qs.append(_recover(us[-1], dim, [h] * len(dim)))
        return [pack([t for v in us for t in v]), pack([t for v in qs for t in v])]
    b, sdf, p, h = _unet_data(case, seed)
    net = api.UNetWarmStart(_dim(case), seed=seed % 1000)  # its seeded weights are the call's input
    vec = net.params(0)
    net.close()
    return _unet_exact(vec, b, sdf, p, h)


# ------------------------------------------------------------------ work and tolerances
def _faces(dim):
    n = math.prod(dim)
    return sum(n // m * (m + 1) for m in dim)


def _edges(dim):
    if len(dim) == 2:
        return (dim[0] + 1) * (dim[1] + 1)
    n = math.prod((m + 1) for m in dim)
    return sum(n // (m + 1) * m for m in dim)


def _one_projection(dim, tol, cycles_per_digit=2.0):
    """Velocity and fractions in, velocity and potential out; the flops are those of the V-cycles that
    the tolerance takes (five stencil passes of 16 flops a cell and the coarse levels) and of the lifting."""
    n = math.prod(dim)
    cycles = cycles_per_digit * -math.log10(tol)
    coarse = 4.0 / 3.0 if len(dim) == 2 else 8.0 / 7.0
    return {"bytes": 4.0 * (3 * _faces(dim) + _edges(dim)), "flops": n * (cycles * 5 * 16 * coarse + len(dim) * len(dim) * 2 * 17)}


def work(case):
    kind = case["kind"]
    if kind in ("project3d", "project2d", "pressure3d"):
        w = _one_projection(_dim(case), case["tol"])
        if kind == "pressure3d":
            w["bytes"] -= 4.0 * _edges(_dim(case))
        return w
    if kind == "batch":
        import random
        r = random.Random(case["mix"])
        s3, s2 = [int(v) for v in case["sizes3"].split(",")], [int(v) for v in case["sizes2"].split(",")]
        total = {"bytes": 0.0, "flops": 0.0}
        for i in range(case["count3"] + case["count2"]):
            d3 = i < case["count3"]
            n = r.choice(s3 if d3 else s2)
            r.randint(0, 4)
            for k, v in _one_projection((n,) * (3 if d3 else 2), case["tol"]).items():
                total[k] += v
        return total
    dim = _dim(case)
    n = math.prod(dim)
    if kind == "recover3d":
        return {"bytes": 4.0 * (_faces(dim) + _edges(dim)), "flops": 18.0 * 17 * n}
    if kind == "dwt":
        return {"bytes": (16.0 if case["double"] else 8.0) * n, "flops": 17.0 * n}
    if kind == "sweep3d":
        return {"bytes": 4.0 * (_faces(dim) + _edges(dim)), "flops": n * (6 * 2.5 * math.log2(n) / 3 + 20.0)}
    if kind == "levelset":
        return {"bytes": 4.0 * (2 * n + _faces(dim)), "flops": 2.0 * case["iters"] * 20 * n}
    if kind == "porous3d":
        return {"bytes": n * (4.0 * 2 + 4.0 * 3 * case["fluid"]), "flops": case["cycles"] * case["fluid"] * n * 5 * 16 * 8 / 7}
    macs = sum(27 * (c0 + c1) * co * s for (c0, c1, co), s in zip(_UNET, (1, 1, 1 / 8, 1 / 8, 1 / 64, 1 / 64, 1 / 8, 1 / 8, 1, 1)))
    return {"bytes": 16.0 * n + 4.0 * 4 * 300000, "flops": 8.0 * macs * n}


def tolerance(case):
    """About four times the distance between the calls and exact(), measured over the ranges."""
    kind = case["kind"]
    if kind in ("project3d", "project2d", "pressure3d", "batch"):
        # FP32 fields, and what a residual at the stopping tolerance leaves in them
        return {"rel": 5e-6 + 300 * case["tol"]}
    if kind == "recover3d":
        return {"rel": 4e-6}
    if kind == "dwt":
        return {"rel": 1e-14 if case["double"] else 4e-6}
    if kind == "sweep3d":
        return {"rel": 1.5e-5}
    if kind == "levelset":
        return {"rel": 2e-6, "max": 2e-4}  # three samples of a cut face's 16384
    if kind == "porous3d":
        return {"rel": 3e-3}  # the constant of each closed pore drifts with the rounding of the residuals
    return {"rel": 2e-2}  # BF16 activations and gradients through ten layers
