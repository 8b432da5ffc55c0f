"""Set-up copies and fills are ordered before the kernels that read them.

The library's streams are non-blocking: a kernel on them does not wait for the
default stream, and a copy from pageable memory or a fill there may return to
the host before it has reached the device.  So no source of the library uses
the default-stream forms towards the device; each names the stream of the
kernels that follow."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phd_gb300", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_default_stream_copy_or_fill_towards_the_device(path):
    text = open(path).read()
    found = re.findall(r"\bcudaMemset\s*\(|\bcudaMemcpyToSymbol\s*\(|\bcudaMemcpy\s*\([^;]*?cudaMemcpy\w+", text)
    assert [f for f in found if not f.endswith("cudaMemcpyDeviceToHost")] == []
