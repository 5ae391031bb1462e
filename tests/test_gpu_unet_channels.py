"""The network at the ends of the channel counts that it takes (8 to 64 per
level, 128 into a decoder's first convolution), on grids of several patches per
SM: forward on the tensor cores against the CUDA cores, and the gradients,
which start from that forward's activations.

Both forwards round at the same points and sum in FP32 in another order, so
they differ by a few BF16 roundings, as in the tests of the usual counts: 5e-3
of the output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("nr,nz,ch,pool", [(64, 320, (64, 64, 64, 64), 2), (64, 1280, (64, 64, 64, 64), 4),
                                           (256, 512, (64, 64, 8, 8), 4), (128, 640, (8, 64, 64, 8), 2),
                                           (512, 512, (48, 64, 56, 64), 4), (320, 64, (8, 8, 64, 64), 2),
                                           (512, 1024, (8, 8, 8, 8), 4), (576, 576, (64, 8, 8, 64), 4)])
def test_forward_and_gradients_of_every_channel_count(nr, nz, ch, pool):
    import vring_b200 as V
    tc = V.UNet(nr, nz, ch, seed=2, pool=pool)
    cc = V.UNet(nr, nz, ch, seed=2, flags=V.UNet.CUDA_CORES, pool=pool)
    x, g = np.random.default_rng(7).standard_normal((2, nr, nz))
    assert _rel(tc.forward(x), cc.forward(x)) <= 5e-3
    (wt, xt), (wc, xc) = tc.backward(x, g), cc.backward(x, g)
    # dL/dx of a linear network does not depend on the activations
    assert np.array_equal(xt, xc)
    assert _rel(wt, wc) <= 5e-3
