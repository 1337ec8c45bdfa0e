"""Contexts work on non-blocking streams, which do not wait for the legacy default stream: a plain
cudaMemcpy from pageable memory may return while its last copy is still on the way there, and a
plain cudaMemset always does. Everything the host puts into device memory goes through the
context's stream, in order with the kernels that read it."""
from __future__ import annotations

import os
import re

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "camille_b200", "csrc")


def test_device_memory_is_written_in_stream_order():
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".h", ".cpp")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        assert not re.search(r"\bcudaMemset\s*\(", text), name
        for m in re.finditer(r"\bcudaMemcpy\s*\(", text):
            assert "cudaMemcpyDeviceToHost" in text[m.end():text.index(";", m.end())], name
        seen += len(re.findall(r"\bcudaMemcpyAsync\s*\(", text))
    assert seen > 20
