"""The z-marching right-hand side and pressure update at the shapes where
their rows per CTA, threads per CTA and planes per CTA change: 8 rows up to 32
theta cells, 4 up to 64, 2 up to 128 and 2 in 512 threads up to 256, with
radial extents that leave a CTA partly filled and z extents around a solve
batch of four planes.  Tolerance as in the fused substep's parity test."""
import numpy as np
import pytest

from parity_util import STATE, assert_field_close, copy_to_gpu, make_pair, prep

pytestmark = pytest.mark.gpu

GRIDS = [(4, 9, 5), (16, 8, 4), (30, 17, 21), (32, 7, 128), (34, 12, 22), (64, 5, 33), (66, 6, 20), (126, 5, 31),
         (130, 5, 18), (200, 4, 9), (256, 7, 34), (256, 4, 4)]


def _state(orc, gpu, grid, seed):
    rng = np.random.default_rng(seed)
    for n in ("q1", "q2", "q3", "ru1", "ru2", "ru3", "prg", "pres"):
        a = orc.field(n)
        a[...] = 0.1 * rng.uniform(-1.0, 1.0, size=a.shape)
    copy_to_gpu(orc, gpu, ["q1", "q2", "q3", "ru1", "ru2", "ru3", "prg", "pres"])


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
@pytest.mark.parametrize("irk", [1, 3])
def test_fused_substep(grid, irk):
    orc, gpu = make_pair(*grid, wth="modified")
    _state(orc, gpu, grid, irk)
    prep(orc, gpu, irk, 2e-3, 0)
    orc.substep(irk)
    gpu.substep(irk)
    for n in STATE + ["dph"]:
        assert_field_close(gpu, orc, n, rel=1e-11)


@pytest.mark.parametrize("grid", GRIDS + [(9, 6, 10)], ids=lambda g: "x".join(map(str, g)))
def test_step_with_given_explicit_terms(grid):
    """vr_step on arbitrary H in dq1..3: the walk that reads them (odd theta
    extents go through the separate kernels)."""
    orc, gpu = make_pair(*grid, wth="modified")
    _state(orc, gpu, grid, 5)
    rng = np.random.default_rng(6)
    for n in ("dq1", "dq2", "dq3"):
        a = orc.field(n)
        a[...] = 0.1 * rng.uniform(-1.0, 1.0, size=a.shape)
    copy_to_gpu(orc, gpu, ["dq1", "dq2", "dq3"])
    prep(orc, gpu, 2, 2e-3, 0)
    orc.step()
    gpu.step()
    for n in ("dq1", "dq2", "dq3", "ru1", "ru2", "ru3"):
        assert_field_close(gpu, orc, n, rel=1e-11)


@pytest.mark.parametrize("grid", [(32, 12, 40), (64, 9, 36), (256, 6, 32)], ids=lambda g: "x".join(map(str, g)))
def test_mixed_form_follows_fp64(grid):
    """One step of the mixed form against FP64 on a ring: the fields are stored
    in float in between, so the velocities agree to float rounding."""
    import vring_b200 as V
    from vring_b200.synthetic import ring_fields
    q = ring_fields(*grid, 4.0, 12.0, noise=1e-3, seed=3)
    out = {}
    for form in ("fp64", "mixed"):
        r = V.Run(*grid, 4.0, 12.0, 2e-3, 1000.0, 1.0, 1.0, precision=form, theta_wavenumber="modified")
        for n, a in zip(("q1", "q2", "q3"), q):
            r.set(n, a)
        r.iterate(1)
        out[form] = [r.get(n) for n in ("q1", "q2", "q3")]
        assert r.max_divergence() <= 1e-9
    for a, b in zip(out["fp64"], out["mixed"]):
        assert np.abs(a - b).max() <= 2e-6 * max(np.abs(x).max() for x in out["fp64"])
