"""Order of host-to-device copies and the kernels that read them.  The solver's
streams are non-blocking ones, which a copy on the legacy stream does not hold
back, and a copy from pageable memory may return before its data have arrived:
a plain cudaMemcpy to the device is right only where the legacy stream is
waited for afterwards (upload and uploads_done in mpm_common.cuh)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cumpm_b200", "csrc")


def functions(text):
    """(head, body) of the definitions that start in the first column"""
    for m in re.finditer(r"^[^\s/#}][^;{}]*\{.*?^\}", text, re.S | re.M):
        head, body = m.group(0).split("{", 1)
        yield head, body


def test_blocking_copies_to_the_device_go_through_upload():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.c*"))):
        text = open(path).read()
        calls = [m.group(0) for m in re.finditer(r"cudaMemcpy\s*\((?:[^;]*?)\);", text, re.S)
                 if "cudaMemcpyHostToDevice" in m.group(0)]
        if os.path.basename(path) == "mpm_common.cuh":
            body = text[text.index("inline void upload("):]
            assert len(calls) == 1 and calls[0] in body[:body.index("\n}")]
            assert "inline void uploads_done() { MPM_CUDA(cudaStreamSynchronize(cudaStreamLegacy)); }" in text
        else:
            assert not calls, (os.path.basename(path), calls)


def test_every_set_of_uploads_is_waited_for():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.c*"))):
        if os.path.basename(path) == "mpm_common.cuh":
            continue
        for head, body in functions(open(path).read()):
            uses = [m.start() for m in re.finditer(r"\bupload(?:_table)?\(|(?:dense_|rader_)\.init\(", body)]
            if not uses or re.search(r"(DenseDFT|RaderDFT)::init|::upload_table", head):
                continue
            seen += 1
            assert "uploads_done();" in body[uses[-1]:], (os.path.basename(path), head)
    assert seen >= 4      # the line transforms, both fields' tables, the particle lists
