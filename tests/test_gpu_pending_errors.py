"""An error of some other CUDA call that is pending on the thread: making a
context or a solver does not fail for it, and a step does not lose it."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cudart():
    import vring_b200 as V
    V.api.lib()  # loads the runtime that the library uses
    path = next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart.so" in line)
    return ctypes.CDLL(path)


@pytest.fixture
def pending():
    """Leaves an error pending on the thread (an allocation nothing can hold), and clears it at the end."""
    rt = _cudart()
    rt.cudaFree(None)
    rt.cudaGetLastError()

    def make():
        p = ctypes.c_void_p()
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(1 << 60)) != 0
        assert rt.cudaPeekAtLastError() != 0

    yield rt, make
    rt.cudaGetLastError()


@pytest.mark.parametrize("nth,nz", [(16, 48), (15, 32), (15, 48)])
def test_contexts_of_any_length_are_made_beside_a_pending_error(pending, nth, nz):
    import vring_b200 as V
    _, make = pending
    V.Run(16, 16, 32, 4.0, 12.0, 2e-3, 1000.0, 1.0, 1.0).close()  # the library's kernels are loaded
    make()
    V.Run(nth, 16, nz, 4.0, 12.0, 2e-3, 1000.0, 1.0, 1.0).close()


def test_solvers_of_any_length_are_made_beside_a_pending_error(pending):
    import vring_b200 as V
    _, make = pending
    for nz in (64, 100):
        make()
        V.K2d(np.linspace(0.0, 4.0, 33), nz, 12.0).close()


@pytest.mark.parametrize("nth", [16, 15])
def test_a_step_does_not_lose_a_pending_error(pending, nth):
    import vring_b200 as V
    rt, make = pending
    r = V.Run(nth, 16, 32, 4.0, 12.0, 2e-3, 1000.0, 1.0, 1.0)
    r.set_clock(1, 2e-3, 1)
    for call in (r.ucoeff, r.coesys, r.hdnbc, r.hdnl1, r.hdnl2, r.hdnl3, r.step):
        call()  # the runtime clears the thread's error when it loads a kernel, so load them all
    make()
    try:
        r.step()
        reported = False
    except V.VrError as e:
        reported = e.code == 3  # VR_ERR_CUDA
    assert reported or rt.cudaPeekAtLastError() != 0
    rt.cudaGetLastError()
    r.close()
