"""`Device::upload` is complete when it returns (backend.hpp), whatever its size: read from the source of the device's own."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vq_b200", "csrc")


def test_upload_waits_on_every_way_out():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "cuda_device.cu")).read())
    start = text.index("void CudaDevice::upload(")
    body = text[start:text.index("\n}\n", start)]
    body = body.replace("if (!bytes) return;", "")
    ways = re.split(r"\breturn;", body)
    assert len(ways) >= 2
    for way in ways:
        statements = [s.strip() for s in way.split(";") if s.strip(" {}\n")]
        assert statements[-1] == "VQB_CUDA_CHECK(cudaStreamSynchronize(stream_))", statements[-1]
