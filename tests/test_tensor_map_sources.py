"""Tensor maps in global memory, which the host rewrites between launches, are acquired by the thread
that issues the copies before it uses them (a kernel could otherwise copy through the old map, of a
buffer that has since been swapped or freed); maps passed as __grid_constant__ parameters need none."""
from __future__ import annotations

import os
import re

from tests.conftest import ROOT
from tests.test_capture_sources import body

CSRC = os.path.join(ROOT, "camille_b200", "csrc")


def _kernels(text: str):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", text):
        q, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[q], 0)
            q += 1
        start = text.index("{", q)
        depth, e = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[e], 0)
            e += 1
            if depth == 0:
                break
        yield m.group(1), text[m.end():q - 1], text[start:e]


def test_maps_in_global_memory_are_acquired():
    seen = {}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        for kernel, params, code in _kernels(open(os.path.join(CSRC, name)).read()):
            m = re.search(r"const CUtensorMap\s*\*\s*(?:__restrict__\s*)?(\w+)", params)
            if m:
                first = code.index("acquire_map(") if "acquire_map(" in code else None
                assert first is not None and first < code.index("tma_load_3d("), f"{name}: {kernel}"
                seen[kernel] = m.group(1)
    assert "k_plane_filter_batch" in seen


def test_the_acquire_is_a_proxy_fence():
    text = open(os.path.join(CSRC, "lee_tma_util.cuh")).read()
    assert "fence.proxy.tensormap::generic.acquire" in body(text, "acquire_map")
