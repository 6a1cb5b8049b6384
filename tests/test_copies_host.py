"""Order of host-to-device copies and the kernels that read them.  The solver's
streams are non-blocking ones, which a copy on the legacy stream does not hold
back, and a copy from pageable memory may return before its data have arrived:
a plain cudaMemcpy to the device is right only where the legacy stream is
waited for afterwards, which upload() in mpm_common.cuh does."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cumpm_b200", "csrc")


def test_blocking_copies_to_the_device_go_through_upload():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.c*"))):
        text = open(path).read()
        calls = [m.group(0) for m in re.finditer(r"cudaMemcpy\s*\((?:[^;]*?)\);", text, re.S)
                 if "cudaMemcpyHostToDevice" in m.group(0)]
        if os.path.basename(path) == "mpm_common.cuh":
            body = text[text.index("inline void upload("):]
            body = body[:body.index("\n}")]
            assert len(calls) == 1 and calls[0] in body
            assert "cudaStreamSynchronize(cudaStreamLegacy)" in body[body.index(calls[0]):]
        else:
            assert not calls, (os.path.basename(path), calls)
