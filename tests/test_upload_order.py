"""What is copied to the device in one call is there before a kernel reads it.

The frame, batch and server streams are non-blocking, so nothing orders their kernels behind a
copy on the legacy stream, and a blocking cudaMemcpy from pageable memory may return once its
source is staged, before the last bytes have arrived.  Every copy to the device is therefore
queued on the stream of the kernels that read it."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "master-of-puppets_b200" / "csrc"


@pytest.mark.parametrize("name", ["ibl.cu"])
def test_copies_to_the_device_are_ordered(name):
    src = (CSRC / name).read_text()
    off_stream = re.findall(r"cudaMemcpy\([^;]*cudaMemcpy(?:HostToDevice|DeviceToDevice)", src)
    assert not off_stream, off_stream
