"""What an object is made from has arrived when its first call runs: objects
made one after the other and kept, so that each lies in memory of its own, and
used at once, give the same answers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_networks_run_with_their_weights_from_the_first_call():
    import vring_b200 as V
    x = np.random.default_rng(1).standard_normal((64, 64))
    kept, first = [], None
    for _ in range(40):
        kept.append(V.UNet(64, 64, (64, 64, 64, 64), seed=2))
        y = kept[-1].forward(x)
        first = y if first is None else first
        assert np.abs(y).max() > 0 and np.array_equal(y, first)


def test_axisymmetric_solvers_run_with_their_coefficients_from_the_first_call():
    import torch
    import vring_b200 as V
    from vring_b200.learned import tanh_faces
    faces = tanh_faces(512)
    f = torch.randn((1024, 512), dtype=torch.float64, device="cuda")
    x = torch.zeros_like(f)
    torch.cuda.synchronize()
    kept, first = [], None
    for _ in range(12):
        kept.append(V.K2d(faces, 1024, 15.0))
        kept[-1].direct_dev(f.data_ptr(), x.data_ptr())
        y = x.clone()
        torch.cuda.synchronize()
        first = y if first is None else first
        assert torch.equal(y, first) and bool(torch.isfinite(y).all())


def test_particles_are_advanced_from_the_state_they_were_given():
    import vring_b200 as V
    from vring_b200.synthetic import annulus_particles, ring_fields
    n = 20000
    u = np.zeros((n, 117), order="F")
    u[:, 0], u[:, 1], u[:, 2] = annulus_particles(n, 0.5, 1.5, 2.0, 4.0, seed=1)
    v = np.zeros((n, 3), order="F")
    v[:, 2] = np.arange(1, n + 1)
    r = V.Run(32, 24, 64, 4.0, 12.0, 1e-3, 1000.0, 1.0, 1.0)
    for name, a in zip(("q1", "q2", "q3"), ring_fields(32, 24, 64, 4.0, 12.0, noise=1e-4, seed=5)):
        r.set(name, a)
    kept, first = [], None
    for _ in range(8):
        p = V.Part(r, 8, n, 1)
        kept.append(p)
        p.set_state(u, v, None, n)
        p.iter_part(1)
        got = p.state()[0]
        first = got if first is None else first
        assert np.array_equal(got, first) and not np.array_equal(got[:, :3], u[:, :3])
    for p in kept:
        p.close()
    r.close()


@pytest.mark.parametrize("method", ["cg", "pcg"])
def test_a_second_solver_gives_the_first_ones_bits(method):
    import vring_b200 as V
    f = np.random.default_rng(9).standard_normal((100, 150))
    a, b = (V.K2d(np.linspace(0.0, 4.0, 101), 150, 12.0) for _ in range(2))
    x, its, _, _ = a.solve(f, method, tol=1e-10, maxit=5000)
    y, its2, _, _ = b.solve(f, method, tol=1e-10, maxit=5000)
    assert its == its2 and np.array_equal(x, y)
