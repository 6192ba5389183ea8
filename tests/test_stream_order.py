"""CPU: uploads are ordered before the kernels that read them.

The library's streams are created with cudaStreamNonBlocking, so they do not
wait for the default stream, and cudaMemcpy from pageable memory may return
before the device copy is complete.  An upload therefore has to be issued on
the stream of its readers (pcf_upload, cudaMemcpyAsync), never by cudaMemcpy."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pincflow.jl_b200", "csrc")


def test_no_upload_on_the_default_stream():
    files = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))
    assert len(files) >= 10
    found = []
    for path in files:
        src = open(path).read()
        for m in re.finditer(r"\bcudaMemcpy(?:2D|3D)?\s*\(([^;]*?)\)\s*[;!=|)]", src):
            if "HostToDevice" in m.group(1):
                found.append((os.path.basename(path), src.count("\n", 0, m.start()) + 1))
    assert not found, found
