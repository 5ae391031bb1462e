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


def test_a_flexible_cg_refused_for_memory_leaves_the_solver_whole():
    """The kept directions are two arrays of 32 MB at 512 x 1024; with about 48
    MB left the first fits and the second does not."""
    import torch
    import vring_b200 as V
    ref, k = _solver(), _solver()
    f = _rhs(k)
    want = ref.solve(f, "fcg_jacobi", tol=1e-6, maxit=40)[0]  # loads the kernels
    d = [torch.from_numpy(np.ascontiguousarray(f.T)).cuda(), torch.zeros((k.nz, k.nr), dtype=torch.float64, device="cuda")]
    torch.cuda.synchronize()
    MB = 1 << 20
    ballast = []
    while True:
        spare = torch.cuda.mem_get_info()[0] - 48 * MB
        if spare < 8 * MB:
            break
        ballast.append(torch.empty(spare // (2 * MB) * 2 * MB, dtype=torch.uint8, device="cuda"))
    assert 34 * MB < torch.cuda.mem_get_info()[0] < 64 * MB
    for _ in range(2):  # the second time it is the same answer, not an error left over or a half-made state
        with pytest.raises(V.VrError) as e:
            k.solve_dev(d[0].data_ptr(), d[1].data_ptr(), "fcg_jacobi", tol=1e-6, maxit=40)
        assert e.value.code == 2  # VR_ERR_OOM
        assert torch.cuda.mem_get_info()[0] > 34 * MB
    del ballast
    torch.cuda.empty_cache()
    assert np.array_equal(k.solve(f, "fcg_jacobi", tol=1e-6, maxit=40)[0], want)
