"""The engine's streams are non-blocking: they do not wait for the legacy
stream, where a fill or the last part of a copy from pageable memory may still
run when its call returns.  So the engines and the batch put every copy and
fill on the stream that uses the memory; one on the legacy stream in their
file is a kernel that may read its tables before they are there."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gtopen_b200", "csrc")


def test_engine_copies_name_their_stream():
    with open(os.path.join(CSRC, "kernels", "engine.cu")) as f:
        src = f.read()
    assert re.findall(r"\bcuda(?:Memcpy|Memset|Memcpy2D|Memset2D)\(", src) == []
    calls = re.findall(r"\bcuda(?:MemcpyAsync|MemsetAsync)\(([^;]*)\);", src)
    assert len(calls) > 20
    for c in calls:  # the last argument is a stream by its name
        assert re.search(r",\s*(?:E\.stream|d_->stream|stream|st|s)\)?$", c), c
