"""Tables reach the device on the context's stream and are there when the upload returns: kernels
read them ahead of their wait for the previous kernel, and a plain cudaMemcpy from pageable
memory is ordered with nothing on a non-blocking stream."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "steamroller.jl_b200", "csrc")


def test_no_upload_on_the_legacy_stream():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.h"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for call in re.findall(r"\bcudaMemcpy\s*\([^;]*;", text) + re.findall(r"\bcudaMemset\s*\([^;]*;", text):
            if "cudaMemcpyDeviceToHost" not in call:
                found.append((os.path.basename(path), call))
    assert not found
