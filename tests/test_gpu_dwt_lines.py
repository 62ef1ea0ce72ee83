"""Lines of every length that the in-place line kernel takes, and the next longer ones of the tile kernel, against
the FP64 oracle: line counts around a tile of 32, three axes, both wall rules, both directions."""
import numpy as np
import pytest
import torch

from test_gpu_parity import N, T, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [2, 3, 4, 5, 6, 7, 8, 9, 10])
@pytest.mark.parametrize("wav,ext", [(11, 0), (7, 1)])
@pytest.mark.parametrize("axis", ["x", "y", "z"])
def test_lines_match_oracle(wp, oracle, wav, ext, axis, levels):
    """Bound: a level rounds at most 12 products and sums per output, the base matrices amplify by at most 3:
    36 levels eps.  (FP64: the oracle rounds as often, twice that.)"""
    rng = np.random.default_rng(levels)
    n = (1 << levels) + ext
    for a, b in ((1, 1), (31, 1), (11, 3), (5, 13)):
        dims = {"x": (n, a, b), "y": (a, n, b), "z": (a, b, n)}[axis]
        v = rng.standard_normal((dims[2], dims[0], dims[1])).astype(np.float32).astype(np.float64)
        for bc in "nd":
            for fwd in (True, False):
                ref = oracle.dwt_axis(v, levels, axis, wav, bc, fwd)
                for dt, tol in ((torch.float32, 36 * levels * 6e-8), (torch.float64, 72 * levels * 1.1e-16)):
                    src = T(v, dt)
                    dst = torch.full_like(src, float("nan"))
                    wp.CuWHHDForward.Solve1D(dst, src, dims, levels, axis, bc, wav, fwd)
                    assert rel(ref, N(dst)) < tol, (dims, bc, fwd, dt, rel(ref, N(dst)))
                    wp.CuWHHDForward.Solve1D(src, None, dims, levels, axis, bc, wav, fwd)
                    assert torch.equal(src, dst)
