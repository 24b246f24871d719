"""Copies and clears of the library are enqueued on the context's stream.

A context may run on a non-blocking stream, which has no order with the legacy
default stream: a host-to-device cudaMemcpy from pageable memory may return
before its transfer is done, so a kernel on that stream could read a table
before it arrives.  The sources are read here; test_gpu_stream_order.py runs
the first calls of a context on such a stream."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "asohf_b200", "csrc")
LEGACY = re.compile(r"\bcuda(Memcpy|Memset)(2D|3D)?\s*\(|\bcudaMemcpy(To|From)Symbol\s*\(")


def _code(path):
    s = open(path).read()
    s = re.sub(r"/\*.*?\*/", "", s, flags=re.S)
    return re.sub(r"//[^\n]*", "", s)


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu*"))))
def test_no_copy_on_the_legacy_stream(name):
    files = glob.glob(os.path.join(CSRC, name))
    assert files
    for f in files:
        assert not LEGACY.findall(_code(f)), os.path.basename(f)
