"""What is copied to the device in one call is there before a kernel reads it.

The frame, batch and server streams are non-blocking, so nothing orders their kernels behind a
copy on the legacy stream, and a blocking cudaMemcpy from pageable memory may return once its
source is staged, before the last bytes have arrived (one within the device, once it is queued).
Every copy to the device is therefore queued on the stream of the kernels that read it, or made
by mc_upload, which waits for it."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "master-of-puppets_b200" / "csrc"


@pytest.mark.parametrize("name", sorted(f.name for f in CSRC.glob("*.cu")))
def test_copies_to_the_device_are_ordered(name):
    src = (CSRC / name).read_text()
    upload = re.search(r"^cudaError_t mc_upload\(.*?^}", src, re.M | re.S)
    if upload:
        assert "cudaStreamSynchronize(cudaStreamLegacy)" in upload.group(0)
        src = src.replace(upload.group(0), "")
    off_stream = re.findall(r"cudaMemcpy\([^;]*cudaMemcpy(?:HostToDevice|DeviceToDevice|Default)",
                            src)
    assert not off_stream, off_stream
