"""Device memory is filled on the stream whose kernels read it.

The solvers' and batches' streams are non-blocking: the legacy stream, on which
cudaMemset and cudaMemcpy run, is not ordered with them, and both calls may
return before their work on the device is done.  The sources therefore fill
buffers with the asynchronous calls on their own stream, or wait.  No GPU
needed.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mantaflow_gb300", "csrc")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_nothing_is_filled_on_the_legacy_stream(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    assert not re.search(r"\bcudaMemset\s*\(", text)
    for call in re.finditer(r"\bcudaMemcpy(ToSymbol)?\s*\(", text):
        rest = text[call.start():call.start() + 300]
        if call.group(1) or "HostToDevice" in rest.split(";")[0]:
            assert "cudaStreamSynchronize" in rest or "cudaDeviceSynchronize" in rest, rest[:120]
