"""CG and Jacobi CG at the grid shapes where the resident kernel's split
changes: segments per CTA, idle threads, a partly filled last CTA, one to
eight planes per thread, and the grids that do not fit (streaming kernels).

Tolerance: the error of an answer with relative residual tol is at most the
operator's condition number times tol; with tol 1e-12 and condition numbers
below 1e6 on these grids (bounded by 4 / h^2 over the lowest eigenvalue,
about 1e-2) it stays below 1e-6 of the largest value, and the direct solve
itself adds 1e-11."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# nr x nz: one CTA; several segments; nr one above and below a half CTA; exact
# and ragged last CTAs; C = 7 and 8; beyond C = 8 and beyond 512 columns
SHAPES = [(4, 4), (5, 9), (31, 70), (64, 148), (100, 1023), (255, 33), (256, 300), (257, 149), (511, 20), (512, 7),
          (512, 1036), (512, 1184), (512, 1185), (513, 24)]


@pytest.mark.parametrize("method", ["cg", "pcg"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda v: "%dx%d" % v)
def test_shapes_converge_to_the_direct_solve(method, shape):
    import vring_b200 as V
    nr, nz = shape
    faces = np.linspace(0.0, 5.0, nr + 1)
    k = V.K2d(faces, nz, 15.0)
    rm, zm = 0.5 * (faces[1:] + faces[:-1]), (np.arange(nz) + 0.5) * 15.0 / nz
    f = np.exp(-(rm[:, None] - 1.3) ** 2 - (zm[None, :] - 6.0) ** 2 / 4) + 0.1 * np.cos(zm)[None, :]
    x, it, rr, _ = k.solve(f, method, tol=1e-12, maxit=40000)
    ref = k.direct(f)
    assert it < 40000 and np.abs(x - ref).max() <= 1e-6 * np.abs(ref).max(), (it, rr)
    # the same answer again, from the same and from a second solver
    y, it2, _, _ = k.solve(f, method, tol=1e-12, maxit=40000)
    assert it2 == it and np.array_equal(x, y)


@pytest.mark.parametrize("method", ["cg", "pcg"])
def test_iterations_carry_over_launches_and_caps(method):
    """A solve stopped at a cap and restarted from its answer still converges,
    and a cap on either side of a launch's 512 iterations is met exactly."""
    import vring_b200 as V
    from vring_b200.learned import tanh_faces
    k = V.K2d(tanh_faces(160), 700, 15.0)
    f = np.random.default_rng(3).standard_normal((160, 700))
    for cap in (1, 511, 512, 513):
        x, it, rr, _ = k.solve(f, method, tol=1e-12, maxit=cap)
        assert it == cap and rr > 1e-12
    x, it, rr, _ = k.solve(f, method, x0=x, tol=1e-12, maxit=40000)
    ref = k.direct(f)
    assert np.abs(x - ref).max() <= 1e-6 * np.abs(ref).max()
