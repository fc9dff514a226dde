"""The native sources copy host memory to the device on a stream only: a plain
copy runs on the default stream, which the simulations' own streams do not wait
for, and one from pageable memory may return before it has arrived."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "loquat_b200" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cpp")), ids=lambda p: p.name)
def test_host_to_device_copies_name_a_stream(path):
    plain = [m.group(0) for m in re.finditer(r"\bcudaMemcpy\s*\([^;]*;", path.read_text())
             if "cudaMemcpyHostToDevice" in m.group(0)]
    assert not plain, plain
