"""Uploads and clears from the host against kernels on non-blocking streams, which
nothing orders after the legacy stream's work: a device clear is asynchronous to the
host, and so is the end of a copy from pageable memory.  Every such copy goes
through the two routines that wait for it (hostcopy.h)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "glisser_gb300", "csrc")


def code(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    return re.sub(r"/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu"))
                                        if "cudaStreamNonBlocking" in open(f).read()))
def test_no_unordered_copy_beside_non_blocking_streams(name):
    c = code(os.path.join(CSRC, name))
    assert not re.search(r"\bcudaMemset\s*\(", c)
    assert not re.search(r"\bcudaMemcpy\s*\([^;]*cudaMemcpyHostToDevice", c)


def test_the_routines_wait():
    c = code(os.path.join(CSRC, "hostcopy.h"))
    for call in ("cudaMemcpy", "cudaMemset"):
        body = c[c.index(call + "("):]
        assert "cudaStreamSynchronize(nullptr)" in body[:body.index("}")]
