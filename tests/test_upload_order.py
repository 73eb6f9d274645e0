"""What is copied to the device in one call is there before a kernel reads it.

The frame, batch and server streams are non-blocking, so nothing orders their kernels behind a
copy on the legacy stream, and a blocking cudaMemcpy from pageable memory may return once its
source is staged, before the last bytes have arrived (one within the device, once it is queued).
Every copy to the device is therefore queued on the stream of the kernels that read it, or made
by mc_upload: it orders the frames' stream behind the copy, and each launch of a batch or a
server waits for its event."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "master-of-puppets_b200" / "csrc"


@pytest.mark.parametrize("name", sorted(f.name for f in CSRC.glob("*.cu")))
def test_copies_to_the_device_are_ordered(name):
    src = (CSRC / name).read_text()
    off_stream = re.findall(r"cudaMemcpy\([^;]*cudaMemcpy(?:HostToDevice|DeviceToDevice|Default)",
                            src)
    assert not off_stream, off_stream


def test_launches_wait_for_uploads():
    upload = re.search(r"^cudaError_t mc_upload\(.*?^}", (CSRC / "mopcuda_api.cu").read_text(),
                       re.M | re.S).group(0)
    order = [upload.index(c) for c in ("cudaMemcpyAsync(", "cudaEventRecord(d->up_ev, d->up_stream)",
                                       "cudaStreamWaitEvent(d->stream, d->up_ev")]
    assert order == sorted(order)
    stage = re.search(r"^int LaunchCore::stage\(\).*?^}", (CSRC / "batch_api.cu").read_text(),
                      re.M | re.S).group(0)
    assert "cudaStreamWaitEvent(stream, dev->up_ev" in stage
