"""The same bits on every kind of stream: a context's own, a caller's, the
legacy and the per-thread default stream, and captured into a caller's graph.
The substep's kernels start before their predecessors end, so an order that a
stream does not keep would show here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(32, 24, 64), (12, 20, 45), (128, 12, 32), (15, 16, 33)]  # FFT, products, marching in 2 rows, odd extent


def _ring(nth, nr, nz, precision="fp64"):
    import vring_b200 as V
    from vring_b200.synthetic import ring_fields
    r = V.Run(nth, nr, nz, 4.0, 12.0, 1e-3, 1000.0, 1.0, 1.0, precision=precision, theta_wavenumber="modified")
    for n, a in zip(("q1", "q2", "q3"), ring_fields(nth, nr, nz, 4.0, 12.0, noise=1e-3, seed=5)):
        r.set(n, a)
    return r


def _state(r):
    r.sync()
    return [r.get(n) for n in ("q1", "q2", "q3")]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "%dx%dx%d" % g)
def test_steps_have_the_same_bits_on_every_stream(grid, precision):
    import torch
    ref = _ring(*grid, precision)
    ref.iterate(4)
    want = _state(ref)
    user = torch.cuda.Stream()
    for handle in (user.cuda_stream, 1, 2):  # a caller's, cudaStreamLegacy, cudaStreamPerThread
        for graphs in (True, False):
            r = _ring(*grid, precision)
            r.set_graphs(graphs)
            r.set_stream(handle)
            r.iterate(4)
            for a, b in zip(_state(r), want):
                assert np.array_equal(a, b), (handle, graphs)
            r.close()


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "%dx%dx%d" % g)
def test_substeps_captured_by_a_caller_replay_with_the_same_bits(grid):
    import torch
    ref = _ring(*grid)
    ref.iterate(3)
    want = _state(ref)
    r = _ring(*grid)
    r.iterate(1)  # loads the kernels
    r.set_graphs(False)
    s = torch.cuda.Stream()
    r.set_stream(s.cuda_stream)
    r.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        for irk in (1, 2, 3):
            r.substep(irk)
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    for a, b in zip(_state(r), want):
        assert np.array_equal(a, b)
    del g
