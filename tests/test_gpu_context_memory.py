"""A z length without an FFT costs a context its tables and no further field."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _taken(nth, nr, nz, precision):
    import torch
    import vring_b200 as V
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    r = V.Run(nth, nr, nz, 4.0, 12.0, 1e-3, 1000.0, 1.0, 1.0, precision=precision)
    taken = before - torch.cuda.mem_get_info()[0]
    r.close()
    return taken


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_z_lengths_with_and_without_an_fft_take_the_same_memory(precision):
    nth, nr, nz = 64, 256, 256
    _taken(nth, nr, nz, precision), _taken(nth, nr, nz - 1, precision)  # modules, driver pools
    fft, lin = _taken(nth, nr, nz, precision), _taken(nth, nr, nz - 1, precision)
    # two tables of 16 x 16 x 255 doubles, in blocks of 2 MB; a field is 32 MB
    assert lin <= fft + (6 << 20), (fft, lin)


def test_the_spectrum_in_a_work_array_leaves_the_steps_alone():
    """Extra pressure solves between steps change nothing but their own field."""
    import vring_b200 as V
    from vring_b200.synthetic import ring_fields
    nth, nr, nz = 12, 20, 45
    runs = []
    for extra in (False, True):
        r = V.Run(nth, nr, nz, 4.0, 12.0, 1e-3, 1000.0, 1.0, 1.0)
        for n, a in zip(("q1", "q2", "q3"), ring_fields(nth, nr, nz, 4.0, 12.0, noise=1e-3, seed=5)):
            r.set(n, a)
        rhs = np.random.default_rng(3).standard_normal((nth, nr, nz))
        for _ in range(3):
            if extra:
                r.set("rhs", np.asfortranarray(rhs))
                r.laplace_solve()
            r.iterate(1)
        runs.append(r)
    for n in ("q1", "q2", "q3", "pres"):
        assert np.array_equal(runs[0].get(n), runs[1].get(n)), n
