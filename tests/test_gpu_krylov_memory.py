"""What the axisymmetric solves ask of the device's memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(nr=512, nz=1024):
    import vring_b200 as V
    from vring_b200.learned import tanh_faces
    return V.K2d(tanh_faces(nr), nz, 15.0)


def _rhs(k):
    return np.random.default_rng(2).standard_normal((k.nr, k.nz))


@pytest.mark.parametrize("method", ["cg", "pcg"])
def test_a_resident_solve_allocates_nothing(method):
    import torch
    for _ in range(2):  # the first solver loads the kernels
        k = _solver()
        f = torch.from_numpy(np.ascontiguousarray(_rhs(k).T)).cuda()
        x = torch.zeros_like(f)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        k.solve_dev(f.data_ptr(), x.data_ptr(), method, tol=1e-6, maxit=600)
        taken = before - torch.cuda.mem_get_info()[0]
    assert taken == 0
