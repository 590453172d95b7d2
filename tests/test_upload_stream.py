"""What the step kernels read is copied to the device on their own stream.  A
copy on the legacy stream may return before pageable data has reached the
device, and the library's streams (non-blocking) do not wait for that stream:
read from the source, since no run shows it reliably."""
import os
import re

from fletcher_petrobras_gb300.build import CSRC


def test_no_upload_on_the_legacy_stream():
    text = open(os.path.join(CSRC, "driver.cu")).read()
    calls = re.findall(r"\bcudaMemcpy(?:ToSymbol)?\([^;]*cudaMemcpyHostToDevice[^;]*;", text)
    assert calls == []
    assert len(re.findall(r"\bcudaMemcpy(?:ToSymbol)?Async\([^;]*cudaMemcpyHostToDevice[^;]*;", text)) >= 5
