"""The batched Thomas solver at the edges of its tiles (16 positions, 8 or 16
systems per CTA), against the oracle's restatement of trithom.F90:6-29.

Tolerance: the systems are diagonally dominant (|beta| >= 0.5 |bb|), so each
step contracts the error of the one before it; a handful of roundings per step
stay below 1e-14 of the largest solution entry, as in the parity test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _systems(rng, n, nbatch, scale=1.0):
    a = rng.uniform(-1.0, 1.0, (nbatch, n)) * scale
    c = rng.uniform(-1.0, 1.0, (nbatch, n)) * scale
    b = (2.5 + rng.uniform(0.0, 1.0, (nbatch, n))) * scale * rng.choice([-1.0, 1.0], (nbatch, 1))
    return rng.uniform(-1.0, 1.0, (nbatch, n)), a, b, c


@pytest.mark.parametrize("n,nbatch,scale", [(1, 1, 1.0), (1, 9, 1.0), (2, 3, 1.0), (15, 8, 1.0), (16, 7, 1.0),
                                            (17, 17, 1.0), (32, 16, 1.0), (33, 1, 1.0), (100, 40, 1e60),
                                            (257, 12, 1e-60), (1024, 9, 1.0), (19, 2369, 1.0), (64, 2368, 1.0)])
def test_thomas_tile_edges(n, nbatch, scale):
    import vring_b200 as V
    from oracle import oracle as O
    r, a, b, c = _systems(np.random.default_rng(n * 7919 + nbatch), n, nbatch, scale)
    a[:, 0] = np.nan   # aa(1) and cc(n) are not used
    c[:, -1] = np.nan
    x = V.solve_lap_thom(r, a, b, c).reshape(nbatch, n)
    a[:, 0] = 0.0
    c[:, -1] = 0.0
    rows = range(nbatch) if nbatch <= 64 else list(range(20)) + list(range(nbatch - 20, nbatch))
    for k in rows:
        o = O.solve_lap_thom(r[k], a[k], b[k], c[k])
        assert np.abs(x[k] - o).max() <= 1e-14 * max(np.abs(o).max(), 1e-300), (k, np.abs(x[k] - o).max())


def test_thomas_small_pivots_follow_the_recurrence():
    """Not diagonally dominant: the elimination order is the recurrence's, so
    the residual stays at rounding for moderate growth."""
    import vring_b200 as V
    n = 48
    rng = np.random.default_rng(5)
    a, c, r = (rng.uniform(0.5, 1.0, (16, n)) for _ in range(3))
    b = rng.uniform(0.3, 0.6, (16, n))
    x = V.solve_lap_thom(r, a, b, c)
    # the recurrence in extended precision
    A, B, C, R = (v.astype(np.longdouble) for v in (a, b, c, r))
    beta, g = np.empty_like(B), np.empty_like(R)
    beta[:, 0], g[:, 0] = B[:, 0], R[:, 0] / B[:, 0]
    growth = np.ones(16)
    for k in range(1, n):
        beta[:, k] = B[:, k] - C[:, k - 1] * A[:, k] / beta[:, k - 1]
        g[:, k] = (R[:, k] - A[:, k] * g[:, k - 1]) / beta[:, k]
        growth = np.maximum(growth, np.abs(1 / beta[:, k]).astype(float))
    y = np.empty_like(g)
    y[:, -1] = g[:, -1]
    for k in range(n - 2, -1, -1):
        y[:, k] = g[:, k] - C[:, k] * y[:, k + 1] / beta[:, k]
    # elimination without pivoting is backward stable up to the growth of its
    # pivots and multipliers; the solution's condition enters once
    for s in range(16):
        M = np.diag(b[s]) + np.diag(a[s, 1:], -1) + np.diag(c[s, :-1], 1)
        bound = 64 * np.finfo(float).eps * growth[s] * max(1.0, float(np.abs(beta[s]).max())) * np.linalg.cond(M)
        assert np.abs(x[s] - y[s].astype(float)).max() <= bound * np.abs(y[s]).max().astype(float)
