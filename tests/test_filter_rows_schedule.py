"""CPU model of what the two-row fused filter (camille_b200/csrc/lee_filter_pair.cu) adds to the ring
schedule of tests/test_filter_pair_schedule.py: the 16-row tile, whose eight warps each filter two rows
of their own and a share of the 2 h halo rows into a row buffer; the two row buffers, one barrier per
loaded plane; the per-thread ring of h + 1 summed increments; and the zeta queue, whose entries are
addressed statically for three planes and shifted then."""
from __future__ import annotations

import os
import re

import pytest

from tests.conftest import ROOT

WARPS, RY, U = 8, 2, 3
TY = WARPS * RY
CHUNKS = (1, 2, 5, 8, 11, 16, 29, 32, 43, 64, 97, 128)


def test_the_model_has_the_kernels_constants():
    text = open(os.path.join(ROOT, "camille_b200", "csrc", "lee_filter_pair.cu")).read()
    for name, value in (("kPairWarps", WARPS), ("kPairRY", RY), ("kPairUnroll", U)):
        assert int(re.search(rf"constexpr int {name} = (\d+);", text).group(1)) == value


@pytest.mark.parametrize("hf", [2, 4, 5])
def test_every_row_of_the_buffer_is_written_once_and_windows_stay_inside(hf):
    by = TY + 2 * hf
    written = []
    for ty in range(WARPS):
        written += [RY * ty + r + hf for r in range(RY)]
        for r0 in range(0, 2 * hf, WARPS):
            r = r0 + ty
            if r < 2 * hf:
                written.append(r if r < hf else r + TY)
    assert sorted(written) == list(range(by))
    for ty in range(WARPS):
        for m in range(2 * hf + RY):
            assert 0 <= RY * ty + m < by
        for r in range(RY):  # the eta taps of row r are centred on the row itself
            assert [RY * ty + r + o for o in range(2 * hf + 1)][hf] == RY * ty + r + hf


@pytest.mark.parametrize("hf", [2, 4, 5])
def test_queue_increments_and_row_buffers_hold_the_planes_they_are_read_for(hf):
    nq = 2 * hf + 1
    for nz in (2 * hf + 1, 16, 37, 97, 128):
        for chunk in CHUNKS:
            for k0 in range(0, nz, chunk):
                k1 = min(nz, k0 + chunk)
                plo, phi = max(0, k0 - hf), min(nz - 1, k1 - 1 + hf)
                queue = [None] * (nq + U - 1)
                ring, ds = [None] * (hf + 1), 0
                buffers, done = [None, None], []
                pend = k1 - 1 + hf
                for p0 in range(k0 - hf, pend + 1, U):
                    for s in range(U):
                        p = p0 + s
                        if s > 0 and p > pend:
                            continue
                        loaded = plo <= p <= phi
                        if loaded:
                            # written before this plane's barrier: its last readers, of the plane two
                            # before, arrived at the previous plane's barrier after reading
                            b = (p - plo) & 1
                            assert buffers[b] is None or buffers[b] == p - 2
                            buffers[b] = p
                        queue[nq - 1 + s] = p if loaded else None
                        ring[ds] = p if loaded else None
                        ds = 0 if ds == hf else ds + 1
                        kf = p - hf
                        if not k0 <= kf < k1:
                            continue
                        want = [q if plo <= q <= phi else None for q in range(p - 2 * hf, p + 1)]
                        assert queue[s:s + nq] == want
                        # (planes outside the block alone are missing, and their classes carry no weight)
                        assert all(q is not None or not 0 <= p - 2 * hf + o < nz for o, q in enumerate(want))
                        assert ring[ds] == kf
                        done.append(kf)
                    for q in range(nq - 1):
                        queue[q] = queue[q + U]
                assert done == list(range(k0, k1))
