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
