"""What a captured step may record. A graph's copy from host memory reads that memory again at every
replay, long after the frame it was taken from is gone, so nothing that runs between the begin and
the end of a capture copies from the host: checked in the source, function by function."""
from __future__ import annotations

import os
import re

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "camille_b200", "csrc")
# the functions that step_impl reaches (the launchers of the .cu kernel files copy nothing)
CAPTURED = {
    "lee_host_step.cu": ["fork_sides", "join_sides", "step_impl"],
    "lee_host_batch.cu": ["batch_launch_stage", "batch_launch_filter", "plane_batch_stage", "plane_batch_filter",
                          "batch_step"],
    "lee_host_kernels.cu": ["run_filter", "encode_maps", "field_maps", "launch_stage_any", "launch_filter_fused",
                            "fill_bc_params", "apply_bcs"],
    "lee_host_core.cu": ["fill_stage_common", "wave_refs", "trace_step"],
    "lee_host_scalar.cu": ["scalar_stage", "scalar_bcs", "scalar_overset", "scalar_filter"],
}


def body(text: str, name: str) -> str | None:
    """The braces of the definition of ``name``."""
    for m in re.finditer(rf"^[\w:<>*& ]+\b{name}\(", text, re.M):
        q = m.end()
        while text[q] not in "{;":
            q += 1
        if text[q] == ";":
            continue
        depth, start = 0, q
        while True:
            depth += {"{": 1, "}": -1}.get(text[q], 0)
            q += 1
            if depth == 0:
                return text[start:q]
    return None


def without(text: str, head: str) -> str:
    """``text`` without the blocks that open with ``head``."""
    while (at := text.find(head)) >= 0:
        q, depth = at + len(head), 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[q], 0)
            q += 1
        text = text[:at] + text[q:]
    return text


def test_captured_steps_copy_nothing_from_the_host():
    for name, functions in CAPTURED.items():
        text = open(os.path.join(CSRC, name)).read()
        found = 0
        for fn in functions:
            b = body(text, fn)
            if b is None:
                for other in CAPTURED:
                    b = b or body(open(os.path.join(CSRC, other)).read(), fn)
            assert b is not None, fn
            found += 1
            assert "HostToDevice" not in without(b, "if (!capturing) {"), f"{name}: {fn}"
        assert found == len(functions)


def test_the_batch_parameters_follow_the_capture():
    step = body(open(os.path.join(CSRC, "lee_host_step.cu")).read(), "step_impl")
    assert "batch_step<T>(c, dts, c->graph.capturing)" in step
    capture = body(open(os.path.join(CSRC, "lee_host_step.cu")).read(), "capture_steps")
    begin, end = capture.index("cudaStreamBeginCapture"), capture.index("cudaStreamEndCapture")
    assert begin < capture.index("capturing = true") < capture.index("step_impl<T>")
    assert capture.index("step_impl<T>") < capture.index("capturing = false") < end
