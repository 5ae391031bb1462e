"""Copies from host memory and fills go on the stream whose kernels read them.

The library's streams are non-blocking: they do not wait for the legacy stream,
on which cudaMemset and cudaMemcpy are ordered, and both may return before the
device has the bytes (cudaMemcpy from pageable memory once they are staged).  A
kernel on a non-blocking stream can then run ahead of them.  Read from the
sources, since it shows only now and then in a run; the stand-alone tridiagonal
solvers launch on the legacy stream itself."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vring_b200", "csrc")


@pytest.mark.parametrize("name", ["vr_unet.cu", "vr_krylov.cu", "vr_ctx.cu", "vr_analysis.cu",
                                  "vr_particles.cu"])
def test_no_copy_to_the_device_or_fill_on_the_legacy_stream(name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    found = re.findall(r"\bcudaMemset\([^;]*;", src) + \
        [m for m in re.findall(r"\bcudaMemcpy\([^;]*;", src) if "cudaMemcpyHostToDevice" in m]
    assert not found, found
