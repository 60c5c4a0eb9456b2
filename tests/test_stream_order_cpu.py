"""The engines run on non-blocking streams, with which nothing on the default stream is ordered: what the host writes to the
device goes through the engine's stream (a pageable copy may return before its data is there, a memset is asynchronous)."""
import os
import re

import pytest

from neuronbridge_gb300 import build


@pytest.mark.parametrize("name", ["nbg_engine.cu", "nbg_dense.cu"])
def test_no_copy_to_the_device_on_the_default_stream(name):
    src = open(os.path.join(build.CSRC, name)).read()
    copies = re.findall(r"cudaMemcpy\(.*?\);", src, re.S)
    assert copies
    # the dense engine waits for the device after its weights, which it converts on the default stream
    made = "cudaMemcpy(tmp.p, w, nn * sizeof(float), cudaMemcpyHostToDevice));"
    for c in copies:
        assert "cudaMemcpyDeviceToHost" in c or c == made, c


@pytest.mark.parametrize("name", ["nbg_engine.cu", "nbg_dense.cu"])
def test_no_memset_on_the_default_stream(name):
    src = open(os.path.join(build.CSRC, name)).read()
    assert "cudaMemsetAsync(" in src and not re.findall(r"cudaMemset(?:2D)?\(|\.zero\(\)", src)


def test_an_upload_waits_for_its_copy():
    src = open(os.path.join(build.CSRC, "nbg_common.cuh")).read()
    body = re.search(r"cudaError_t upload\(.*?\n    }\n", src, re.S).group(0)
    assert body.index("cudaMemcpy(") < body.index("cudaStreamSynchronize(")
