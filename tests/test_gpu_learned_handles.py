"""The learned solve's network is a handle of its own: destroyed and replaced
networks, also at an address that the first one had."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NR, NZ, CH = 64, 128, (8, 16, 16, 16)


def _solver():
    import vring_b200 as V
    from vring_b200.learned import tanh_faces
    return V.K2d(tanh_faces(NR), NZ, 15.0)


def _net(seed):
    import vring_b200 as V
    return V.UNet(NR, NZ, ch=CH, seed=seed)


def _rhs():
    return np.random.default_rng(4).standard_normal((NR, NZ))


def _fresh(seed, f):
    k, net = _solver(), _net(seed)
    k.set_preconditioner(net)
    # few iterations: the answer then depends on the network
    return k.solve(f, "learned", tol=1e-12, maxit=12)[0]


def test_a_replaced_network_is_the_one_that_runs():
    f = _rhs()
    want = {s: _fresh(s, f) for s in (1, 2, 3)}
    assert not np.array_equal(want[1], want[2])
    k = _solver()
    for seed in (1, 2, 3, 1):
        net = _net(seed)
        k.set_preconditioner(net)
        assert np.array_equal(k.solve(f, "learned", tol=1e-12, maxit=12)[0], want[seed])
        net.close()  # the next one may be made where this one was


def test_a_closed_network_lives_on_in_its_solver():
    f = _rhs()
    want = _fresh(5, f)
    k, net = _solver(), _net(5)
    k.set_preconditioner(net)
    net.close()
    spare = [_net(s) for s in (6, 7)]  # takes memory that was freed, had it been
    for _ in range(2):
        assert np.array_equal(k.solve(f, "learned", tol=1e-12, maxit=12)[0], want)
    k.set_preconditioner(spare[0])
    k.set_preconditioner(None)
    k.close()
