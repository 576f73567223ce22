"""Constants that kernels read without waiting for a stream (twiddles, CRT and
sampler tables, control words) are on the device when the call that writes them
returns.  cudaMemcpy from pageable memory and cudaMemset may return earlier,
and the library's non-blocking streams do not wait for the default stream, so
the sources write them through upload() and upload_zeros() only."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yell_gb300", "csrc")


def _code(path):
    return re.sub(r"//[^\n]*|\"[^\"\n]*\"", "", open(path).read())


def test_only_the_helpers_write_device_memory_through_the_default_stream():
    raw = re.compile(r"cudaMemcpy\([^;]*cudaMemcpyHostToDevice|cudaMemcpyToSymbol\(|cudaMemset\(")
    found = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.h"))):
        hits = raw.findall(_code(path))
        if hits:
            found[os.path.basename(path)] = len(hits)
    assert found == {"kernels.h": 2}


def test_the_helpers_wait():
    text = _code(os.path.join(CSRC, "kernels.h"))
    for name in ("upload", "upload_zeros"):
        body = text[text.index(f"cudaError_t {name}("):]
        body = body[:body.index("\n}")]
        assert "cudaStreamSynchronize(nullptr)" in body, name
