"""What the axisymmetric solves ask of the device's memory."""
import ctypes
import gc

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
        gc.collect()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        k.solve_dev(f.data_ptr(), x.data_ptr(), method, tol=1e-6, maxit=600)
        taken = before - torch.cuda.mem_get_info()[0]
    assert taken <= 0


def test_a_flexible_cg_refused_for_memory_leaves_the_solver_whole():
    """The kept directions are two arrays of 32 MB at 512 x 1024; with a block of
    48 MB left the first fits and the second does not."""
    import torch
    import vring_b200 as V
    rt = ctypes.CDLL(next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart.so" in line))

    def malloc(mb):
        p = ctypes.c_void_p()
        if rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(mb << 20)) != 0:
            rt.cudaGetLastError()
            return None
        return p

    ref, k = _solver(), _solver()
    f = _rhs(k)
    want = ref.solve(f, "fcg_jacobi", tol=1e-6, maxit=40)[0]  # loads the kernels
    d = [torch.from_numpy(np.ascontiguousarray(f.T)).cuda(), torch.zeros((k.nz, k.nr), dtype=torch.float64, device="cuda")]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hole, ballast, mb = malloc(48), [], 1 << 14
    try:
        while mb >= 2:  # all that is left, the driver's own reserves included
            p = malloc(mb)
            if p is None:
                mb //= 2
            else:
                ballast.append(p)
        rt.cudaFree(hole)
        hole = None
        for _ in range(2):  # the second time it is the same answer, not an error left over or a half-made state
            with pytest.raises(V.VrError) as e:
                k.solve_dev(d[0].data_ptr(), d[1].data_ptr(), "fcg_jacobi", tol=1e-6, maxit=40)
            assert e.value.code == 2  # VR_ERR_OOM
    finally:
        for p in ballast + ([hole] if hole else []):
            rt.cudaFree(p)
    assert np.array_equal(k.solve(f, "fcg_jacobi", tol=1e-6, maxit=40)[0], want)
