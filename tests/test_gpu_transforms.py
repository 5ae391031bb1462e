"""The folded transforms (lengths without an FFT) at the lengths where a tile, a
coefficient stage or the choice of form ends.

Tolerances: a transform of N terms and the substitutions of nr rows each add
rounding of a few eps per operation, well conditioned except for the
near-constant modes: 1e-11 of the largest value, as in the parity tests of the
Poisson solve."""
import numpy as np
import pytest

from parity_util import make_pair, prep, seed_random

pytestmark = pytest.mark.gpu

# (ntheta, nr, nz): theta 3 .. 16 and odd, even and long folded lines; z around
# the stage of 16 steps (2 x 16 positions), groups of 8 and 16 outputs, the
# longest z; column counts below and above a CTA's 32
GRIDS = [(3, 5, 6), (4, 4, 4), (5, 33, 8), (7, 9, 15), (8, 6, 16), (15, 13, 31), (16, 7, 33), (17, 5, 34), (31, 4, 35),
         (33, 5, 48), (48, 6, 180), (63, 4, 47), (100, 4, 64), (128, 4, 36), (12, 4, 511), (16, 40, 300), (380, 4, 8),
         (727, 4, 5), (1023, 4, 4)]


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_folded_lengths_match_oracle(grid):
    nth, nr, nz = grid
    orc, gpu = make_pair(nth, nr, nz)
    seed_random(orc, gpu, ["rhs"], seed=7)
    prep(orc, gpu)
    rhs = orc.field("rhs").copy()
    orc.laplace_solve()
    gpu.laplace_solve()
    g = gpu.get("dph")[:, 1:nr + 1, 1:nz + 1]
    r = orc.field("dph")[:, 1:nr + 1, 1:nz + 1]
    assert np.abs(g - r).max() <= 1e-11 * np.abs(r).max()
    assert np.array_equal(gpu.get("rhs"), rhs)  # the right-hand side is an input


def test_folded_columns_above_two_ctas_per_sm():
    # 64-column CTAs: theta 64 by FFT, z folded, nth * nr / 64 >= 2 * 148
    nth, nr, nz = 64, 300, 20
    orc, gpu = make_pair(nth, nr, nz)
    seed_random(orc, gpu, ["rhs"], seed=8)
    prep(orc, gpu)
    orc.laplace_solve()
    gpu.laplace_solve()
    g = gpu.get("dph")[:, 1:nr + 1, 1:nz + 1]
    r = orc.field("dph")[:, 1:nr + 1, 1:nz + 1]
    assert np.abs(g - r).max() <= 1e-11 * np.abs(r).max()
