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
