"""The transforms by products (lengths without an FFT), long sweep lines and the axisymmetric direct
solve, at the lengths where a tile, a coefficient stage or the choice of form
ends.

Tolerances: a transform of N terms and the substitutions of nr rows each add
rounding of a few eps per operation, well conditioned except for the
near-constant modes: 1e-11 of the largest value, as in the parity tests of the
Poisson solve."""
import numpy as np
import pytest

from parity_util import assert_field_close, make_pair, prep, seed_random

pytestmark = pytest.mark.gpu

# (ntheta, nr, nz): theta 3 .. 16 and odd, even and long lines; z around
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


# z of 1024: tiles of 8 slots streamed (theta a multiple of 8; more tiles than
# SMs, so that the buffers rotate), else whole columns per warp; z lines of
# 1025 positions in registers (even theta) or the shared-memory sweep
@pytest.mark.parametrize("grid", [(8, 5, 1024), (24, 4, 1024), (256, 16, 1024), (12, 4, 1024), (5, 4, 1024)],
                         ids=lambda g: "x".join(map(str, g)))
def test_long_z_lines_match_oracle(grid):
    nth, nr, nz = grid
    orc, gpu = make_pair(nth, nr, nz)
    seed_random(orc, gpu, ["rhs", "q1", "q2", "q3", "ru1", "ru2", "ru3", "prg", "dq1", "dq2", "dq3"], seed=9, scale=0.1)
    prep(orc, gpu)
    orc.laplace_solve()
    gpu.laplace_solve()
    g = gpu.get("dph")[:, 1:nr + 1, 1:nz + 1]
    r = orc.field("dph")[:, 1:nr + 1, 1:nz + 1]
    assert np.abs(g - r).max() <= 1e-11 * np.abs(r).max()
    orc.step()
    gpu.step()
    for n in ("dq1", "dq2", "dq3"):
        assert_field_close(gpu, orc, n)


# r lines where the register form begins and ends (641 .. 1088 positions, q2
# has one less), where its chunks are full (1024) and where its last chunks are
# empty (673 = 30 x 22 + 13 in 32 chunks of 22)
@pytest.mark.parametrize("grid", [(4, 640, 4), (4, 641, 4), (6, 673, 4), (4, 1024, 4), (10, 1088, 4), (4, 1089, 4),
                                  (5, 700, 4), (64, 700, 40)], ids=lambda g: "x".join(map(str, g)))
def test_long_r_lines_match_oracle(grid):
    orc, gpu = make_pair(*grid)
    seed_random(orc, gpu, ["q1", "q2", "q3", "ru1", "ru2", "ru3", "prg", "dq1", "dq2", "dq3"], seed=10, scale=0.1)
    prep(orc, gpu)
    orc.step()
    gpu.step()
    for n in ("dq1", "dq2", "dq3"):
        assert_field_close(gpu, orc, n)


def test_folded_columns_above_two_ctas_per_sm():
    # 64-column CTAs: theta 64 by FFT, z by products, nth * nr / 64 >= 2 * 148
    nth, nr, nz = 64, 300, 20
    orc, gpu = make_pair(nth, nr, nz)
    seed_random(orc, gpu, ["rhs"], seed=8)
    prep(orc, gpu)
    orc.laplace_solve()
    gpu.laplace_solve()
    g = gpu.get("dph")[:, 1:nr + 1, 1:nz + 1]
    r = orc.field("dph")[:, 1:nr + 1, 1:nz + 1]
    assert np.abs(g - r).max() <= 1e-11 * np.abs(r).max()


# two columns per lane (enough output groups for every scheduler), with an odd
# number of columns, a last tile partly filled and groups beyond the line
@pytest.mark.parametrize("grid", [(63, 301, 20), (47, 121, 100), (48, 100, 180)], ids=lambda g: "x".join(map(str, g)))
def test_two_columns_per_lane(grid):
    nth, nr, nz = grid
    orc, gpu = make_pair(nth, nr, nz)
    seed_random(orc, gpu, ["rhs"], seed=11)
    prep(orc, gpu)
    orc.laplace_solve()
    gpu.laplace_solve()
    g = gpu.get("dph")[:, 1:nr + 1, 1:nz + 1]
    r = orc.field("dph")[:, 1:nr + 1, 1:nz + 1]
    assert np.abs(g - r).max() <= 1e-11 * np.abs(r).max()


def _direct(faces, nz, zmax, f):
    """The direct solve in plain numpy: z cosine products, a Thomas solve per mode."""
    nr = faces.size - 1
    dz, rm, dr = zmax / nz, 0.5 * (faces[:-1] + faces[1:]), np.diff(faces)
    c = faces[1:-1] * dz / np.diff(rm)
    vol = rm * dr * dz
    lo, up = -np.concatenate([[0.0], c]) / vol, -np.concatenate([c, [0.0]]) / vol
    q = np.arange(nz)
    C = np.cos(np.pi * ((np.outer(q, 2 * q + 1)) % (4 * nz)) / (2 * nz))
    fh = f @ C.T / nz
    d = (-(lo + up))[:, None] + 2.0 / dz ** 2 * (1.0 - np.cos(q * np.pi / nz))
    d[-1, 0] += 2.0 * faces[-1] * dz / dr[-1] / vol[-1]
    for j in range(1, nr):
        w = lo[j] / d[j - 1]
        d[j] -= w * up[j - 1]
        fh[j] -= w * fh[j - 1]
    fh[-1] /= d[-1]
    for j in range(nr - 2, -1, -1):
        fh[j] = (fh[j] - up[j] * fh[j + 1]) / d[j]
    C[1:] *= 2.0
    return fh @ C


# z: FFT (32 .. 1024), products by k_lin (other lengths up to 1453), full products above;
# r: below a lane's 16 positions, around a segment of 512
@pytest.mark.parametrize("nr,nz", [(4, 4), (5, 7), (16, 16), (17, 31), (33, 32), (100, 33), (511, 64), (512, 97),
                                   (513, 128), (64, 180), (30, 256), (40, 512), (1025, 40), (512, 1024), (20, 1000),
                                   (18, 1453), (18, 1454), (12, 2048)])
def test_axisymmetric_direct_solve(nr, nz):
    import vring_b200 as V
    from vring_b200.learned import tanh_faces
    faces = tanh_faces(nr)
    k = V.K2d(faces, nz, 15.0)
    f = np.random.default_rng(nr * 10007 + nz).standard_normal((nr, nz))
    x = k.direct(f)
    r = _direct(faces, nz, 15.0, f)
    assert np.abs(x - r).max() <= 1e-11 * np.abs(r).max()
