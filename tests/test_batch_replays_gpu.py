"""Replayed steps of batches without a source, whose captured launches read their parameters from the
device table like those with one: the same bits, clocks and launch counts as steps launched one by
one, over calls that replay one period and many, after a change of the time steps, of the launches'
shapes and of the buffers' roles."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api, cases

pytestmark = pytest.mark.gpu
PRECISIONS = [api.FP64, api.FP32_COMPENSATED]


def _batch(count=5, source=False):
    case = cases.batch2d(count=count, nmin=24, nmax=70, seed=6)
    rng = np.random.default_rng(2)
    for blk in case.blocks:
        if not source:
            blk.monopole = None
        for v in (0, 1, 2, 4):
            blk.state[v] = 1e-3 * rng.standard_normal(blk.x.shape)
    return case


def _same(a, b, case):
    for q in range(len(case.blocks)):
        ya, yb = a.download(q), b.download(q)
        assert np.isfinite(ya[0]).all()
        np.testing.assert_array_equal(ya[0], yb[0])
        assert ya[1:] == yb[1:]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("source", [False, True])
def test_same_bits_and_counts_as_single_steps(product_lib, source, precision):
    case = _batch(source=source)
    a, b = (api.Solver(product_lib, case, precision=precision) for _ in range(2))
    assert a.info().batched
    b.set_graphs(False)
    dts = 0.5 * a.compute_dt_blocks()
    for n, f in ((2, 1.0), (9, 1.0), (130, 1.0), (300, 0.9), (7, 0.9), (129, 0.8)):
        for s in (a, b):
            s.advance_blocks(n, f * dts)
        sa, sb = a.stats(), b.stats()
        assert (sa.stage_launches, sa.filter_launches) == (sb.stage_launches, sb.filter_launches)
        # (a replayed step with a source counts its step in one launch more)
        assert 0 <= sa.kernel_launches - sb.kernel_launches <= (n if source else 0)
        _same(a, b, case)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_same_bits_after_filter_calls_and_other_shapes(product_lib, precision):
    case = _batch()
    a, b = (api.Solver(product_lib, case, precision=precision) for _ in range(2))
    b.set_graphs(False)
    dts = 0.5 * a.compute_dt_blocks()
    for s in (a, b):
        s.advance_blocks(131, dts)
        s.apply_filter()
        s.advance_blocks(140, dts)
        assert product_lib.set_batch_persistent(s.ctx, 2) == api.LEE_OK
        s.advance_blocks(6, dts)
        assert product_lib.set_batch_persistent(s.ctx, -1) == api.LEE_OK
        s.advance_blocks(20, dts)
        assert product_lib.set_batch_shapes(s.ctx, 1, 3) == api.LEE_OK
        s.advance_blocks(133, dts)
    _same(a, b, case)
