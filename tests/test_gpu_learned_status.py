"""A convolution's tensor-core wait that gives up is reported by the call it
belongs to, once, and leaves the network as it was.

The failure is made without a fault: the self-test waits 10 ms on a barrier
that nothing completes and sets the word that a convolution would set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VR_ERR_TIMEOUT = 5
NR, NZ, CH = 64, 128, (8, 16, 16, 16)


def _times_out(V, call):
    with pytest.raises(V.VrError) as e:
        call()
    assert e.value.code == VR_ERR_TIMEOUT


def test_forward_backward_and_solve_report_a_wait_that_gave_up():
    import vring_b200 as V
    from vring_b200.learned import tanh_faces
    net, k = V.UNet(NR, NZ, ch=CH, seed=3), V.K2d(tanh_faces(NR), NZ, 15.0)
    k.set_preconditioner(net)
    rng = np.random.default_rng(1)
    f, g = rng.standard_normal((2, NR, NZ))
    calls = [lambda: net.forward(f), lambda: net.backward(f, g)[1],
             lambda: k.solve(f, "learned", tol=1e-12, maxit=8)[0]]
    want = [c() for c in calls]
    for c, w in zip(calls, want):
        assert net.wait_selftest(10_000_000) == VR_ERR_TIMEOUT
        _times_out(V, c)
        assert np.array_equal(c(), w)
    # a solve without the network does not report the network's word
    assert net.wait_selftest(10_000_000) == VR_ERR_TIMEOUT
    k.solve(f, "pcg", tol=1e-8, maxit=2000)
    _times_out(V, calls[0])
    assert net.wait_selftest(10) == 8 and net.wait_selftest(5_000_000_000) == 8  # VR_ERR_ARG


def test_training_step_that_gave_up_leaves_the_weights_alone():
    import torch
    import vring_b200 as V
    from vring_b200.learned import tanh_faces
    k = V.K2d(tanh_faces(NR), NZ, 15.0)
    e = torch.randn((2, NZ, NR), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    net, ref = (V.UNet(NR, NZ, ch=CH, seed=9) for _ in range(2))
    w0 = net.get_params()
    assert net.wait_selftest(10_000_000) == VR_ERR_TIMEOUT
    _times_out(V, lambda: net.train_step(k, e.data_ptr(), 2, 1e-3))
    assert np.array_equal(net.get_params(), w0)
    # the step after it is the first one; the gradients' atomic sums leave
    # FP32 rounding between two runs, which Adam's first step (lr times the
    # gradient's sign) passes on only where a gradient is near 0
    net.train_step(k, e.data_ptr(), 2, 1e-3)
    ref.train_step(k, e.data_ptr(), 2, 1e-3)
    d = np.abs(net.get_params() - ref.get_params())
    assert np.mean(d > 1e-6) < 0.01 and np.median(np.abs(net.get_params() - w0)) > 5e-4
