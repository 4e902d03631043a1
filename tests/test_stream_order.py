"""The handle's stream is created without the default stream's ordering, so device work that kernels on
it depend on must not go by the default stream: its order against them would be left to chance."""
import re

from subsweep_gb300 import build


def test_no_default_stream_copies_outside_creation():
    src = (build.CSRC / "sweep_host.cpp").read_text()
    # sw_create uploads before the first launch and ends its uploads with a device synchronization
    begin = src.index("sw_status sw_create(const sw_params* params")
    end = src.index("cudaDeviceSynchronize()", begin)
    rest = src[:begin] + src[end:]
    found = [m.group(0) for m in re.finditer(r"(?<!\w)cudaMem(cpy|set)\(.*", rest)]
    assert not found, found
