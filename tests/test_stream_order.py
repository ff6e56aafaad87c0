"""A handle's stream is created without the implicit wait for the default stream, so everything that writes device
memory has to be issued on the handle's stream: a clear or an upload on the default stream may still be under way when
the next kernel reads or adds."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "tortoise_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


@pytest.mark.parametrize("name", FILES)
def test_device_memory_is_written_in_stream_order(name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    assert not re.search(r"\bcudaMemset\s*\(", src)
    for m in re.finditer(r"\bcudaMemcpy\s*\(", src):
        assert "cudaMemcpyDeviceToHost" in src[m.start():src.index(";", m.start())]
