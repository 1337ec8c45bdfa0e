"""Calls long enough to replay several periods of steps at once, and launches that start while the
stream's previous kernel ends: the same bits, clocks and launch counts as steps launched one by one
(also with events between the launches, when nothing starts early), for every remainder, after a
change of the time step, with sources, boundary lines, swapped buffers and batches."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api, cases

pytestmark = pytest.mark.gpu


def _no_filter(case):
    case.filter_scheme = "NONE"  # a step then ends with a swap of buffers
    return case


CASES = {
    "pulse": lambda: cases.pulse2d(n=48, length=47 * 100.0 / 255.0, sponge=6),
    "pulse_odd": lambda: cases.pulse2d(n=67, length=66 * 100.0 / 255.0, sponge=8),
    "no_filter": lambda: _no_filter(cases.pulse2d(n=48, length=47 * 100.0 / 255.0, sponge=6)),
    "shear": lambda: cases.shear2d(nx=64, ny=48),
    "waves": lambda: cases.waves2d(nx=40, ny=32),
    "jet_source": lambda: cases.jet2d_source(nx=64, ny=48),
    "curvi3d": lambda: cases.curvi3d(n=16, nsteps=1, halfwidth=1.5),
    "batch": lambda: cases.batch2d(count=5, nmin=24, nmax=70),
}


@pytest.mark.parametrize("precision", [api.FP64, api.FP32_COMPENSATED])
@pytest.mark.parametrize("label", list(CASES))
def test_same_bits_as_single_steps(product_lib, label, precision):
    case = CASES[label]()
    a, b, t = (api.Solver(product_lib, case, precision=precision) for _ in range(3))
    b.set_graphs(False)
    t.lib.set_timing(t.ctx, 1)
    dt = 0.5 * a.compute_dt()
    for n, h in ((130, dt), (7, dt), (293, dt), (128, 0.9 * dt)):
        counts = []
        for s in (a, b, t):
            s.advance(n, h)
            counts.append((s.stats().kernel_launches, s.stats().stage_launches, s.stats().filter_launches))
        assert counts[1] == counts[2]
        for q, blk in enumerate(case.blocks):
            ya, yb, yt = (s.download(q) for s in (a, b, t))
            assert np.isfinite(ya[0]).all()
            np.testing.assert_array_equal(ya[0], yb[0])
            np.testing.assert_array_equal(ya[0], yt[0])
            assert ya[1:] == yb[1:] == yt[1:]
