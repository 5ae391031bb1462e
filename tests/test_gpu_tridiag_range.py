"""The batched Thomas solver over the range of the numbers it is given: pivots
far from 1, rows and unknowns of mixed scale, infinities, and the size of its
rounding errors.

The recurrence itself (trithom.F90:6-29) forms cc*aa/beta, (rhs - aa*gamm)/beta
and cc*sol/beta, so it solves a system whose pivots are of any size.  The
systems are diagonally dominant; a power of two on a row or on an unknown
changes no rounding, so the bound is the one of the unscaled systems, 1e-14 of
the largest entry (of the unscaled solution), against extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _systems(rng, n, nbatch, off=1.0):
    a, c = (rng.uniform(-1.0, 1.0, (nbatch, n)) * off for _ in range(2))
    b = 2.5 + rng.uniform(0.0, 1.0, (nbatch, n))
    return rng.uniform(-1.0, 1.0, (nbatch, n)), a, b, c


def _recurrence(r, a, b, c, dtype):
    r, a, b, c = (v.astype(dtype) for v in (r, a, b, c))
    beta, g = b.copy(), r.copy()
    with np.errstate(all="ignore"):
        g[:, 0] = r[:, 0] / beta[:, 0]
        for k in range(1, r.shape[1]):
            beta[:, k] = b[:, k] - c[:, k - 1] * a[:, k] / beta[:, k - 1]
            g[:, k] = (r[:, k] - a[:, k] * g[:, k - 1]) / beta[:, k]
        x = g.copy()
        for k in range(r.shape[1] - 2, -1, -1):
            x[:, k] = g[:, k] - c[:, k] * x[:, k + 1] / beta[:, k]
    return x


def _solve(r, a, b, c):
    import vring_b200 as V
    return V.solve_lap_thom(r, a, b, c).reshape(r.shape)


@pytest.mark.parametrize("off", [1.0, 1e-5])
@pytest.mark.parametrize("scale", [1e-300, 1e-165, 1e-160, 1e-156, 1e-150, 1e150, 1e154, 1e160, 1e300])
def test_pivots_of_any_size(scale, off):
    s = 2.0 ** np.round(np.log2(scale))
    r, a, b, c = _systems(np.random.default_rng(11), 67, 21, off)
    ref = _recurrence(r, a, b, c, np.longdouble)
    x = _solve(r * s, a * s, b * s, c * s).astype(np.longdouble)
    assert np.abs(x - ref).max() <= 1e-14 * np.abs(ref).max()
    # the same matrix under a right-hand side of its own scale (which loses bits at the lowest one)
    t = 2.0 ** -40
    ref = _recurrence((r * s * t).astype(np.longdouble) / s / t, a, b, c, np.longdouble)
    x = _solve(r * s * t, a * s, b * s, c * s).astype(np.longdouble) / t
    assert np.abs(x - ref).max() <= 1e-14 * np.abs(ref).max()


@pytest.mark.parametrize("rows,cols", [(0, 0), (60, 0), (300, 0), (0, 200), (250, 150)])
def test_rows_and_unknowns_of_mixed_scale(rows, cols):
    n, nbatch = 100, 19
    rng = np.random.default_rng(rows + 7 * cols)
    r, a, b, c = _systems(rng, n, nbatch)
    ref = _recurrence(r, a, b, c, np.longdouble)
    row = 2.0 ** rng.integers(-rows, rows + 1, (nbatch, n))
    col = 2.0 ** rng.integers(-cols, cols + 1, (nbatch, n))
    left, right = np.roll(col, 1, axis=1), np.roll(col, -1, axis=1)
    x = _solve(r * row, a * row * left, b * row * col, c * row * right) * col
    assert np.abs(x.astype(np.longdouble) - ref).max() <= 1e-14 * np.abs(ref).max()


def test_one_extreme_system_leaves_the_others_alone():
    n, nbatch = 45, 2375  # 16 systems to a CTA, the last one with 7
    r, a, b, c = _systems(np.random.default_rng(3), n, nbatch)
    x = _solve(r, a, b, c)
    far = [0, 9, 1600, nbatch - 1]
    s = np.ones((nbatch, 1))
    s[far] = np.array([[2.0 ** 990], [2.0 ** -990], [2.0 ** 600], [2.0 ** -600]])
    y = _solve(r * s, a * s, b * s, c * s)
    near = np.setdiff1d(np.arange(nbatch), far)
    assert np.array_equal(x[near], y[near])
    assert np.abs(y[far] - x[far]).max() <= 2e-14 * np.abs(x).max()


def test_infinities_and_zero_pivots_go_where_the_recurrence_takes_them():
    r, a, b, c = _systems(np.random.default_rng(8), 40, 6)
    b[0, 17] = np.inf                  # that unknown is 0, the rest decouples
    r[1, 20] = np.inf
    r[2, 20], a[2, 21] = -np.inf, 0.0
    b[3, 11] = np.nan
    c[4, 9] = np.inf
    b[5, 0] = 0.0
    x, ref = _solve(r, a, b, c), _recurrence(r, a, b, c, np.float64)
    assert np.array_equal(np.isnan(x), np.isnan(ref))
    same = np.isinf(ref)
    assert np.array_equal(x[same], ref[same])
    fin = np.isfinite(ref)
    assert np.abs(x[fin] - ref[fin]).max() <= 1e-14 * np.abs(ref[fin]).max()


@pytest.mark.parametrize("off", [1.0, 1e-5])
def test_rounding_is_no_larger_than_the_recurrences(off):
    r, a, b, c = _systems(np.random.default_rng(21), 257, 400, off)
    ref = _recurrence(r, a, b, c, np.longdouble)
    top = np.abs(ref).max(axis=1, keepdims=True)

    def rms(x):
        return float(np.sqrt(np.mean(((x.astype(np.longdouble) - ref) / top) ** 2)))

    assert rms(_solve(r, a, b, c)) <= rms(_recurrence(r, a, b, c, np.float64))
