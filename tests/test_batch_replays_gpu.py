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


@pytest.mark.parametrize("precision", PRECISIONS)
def test_maps_of_later_buffers_and_contexts(product_lib, precision):
    """The batched filter's maps are rewritten in place when buffers swap, and a later context's may
    land where a destroyed one's were: what is copied is always the present buffer."""
    want = None
    for turn in range(4):
        case = _batch(count=5 if turn % 2 == 0 else 7)
        s = api.Solver(product_lib, case, precision=precision)
        dts = 0.5 * s.compute_dt_blocks()
        for _ in range(3):
            s.advance_blocks(2, dts)
            s.apply_filter()
        s.advance_blocks(3, dts)
        got = [s.download(q)[0] for q in range(len(case.blocks))]
        s.close()
        if turn == 0:
            want = got
        elif turn == 2:
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
        t = api.Solver(product_lib, case, precision=precision, batching=False)
        for _ in range(3):
            t.advance_blocks(2, dts)
            t.apply_filter()
        t.advance_blocks(3, dts)
        tol = 1e-12 if precision == api.FP64 else 1e-6
        assert all(api.rel_l2(g, t.download(q)[0]) <= tol for q, g in enumerate(got))
        t.close()


def test_info_reports_the_tiles_that_run(product_lib):
    s = api.Solver(product_lib, _batch())
    tiles = lambda: (tuple(s.info().batch_stage_tile), tuple(s.info().batch_filter_tile))
    assert tiles() == ((64, 8), (64, 16))
    assert product_lib.set_batch_persistent(s.ctx, 1) == api.LEE_OK
    strip = tiles()
    assert strip[0] == strip[1] and strip != ((64, 8), (64, 16))
    assert product_lib.set_batch_persistent(s.ctx, -1) == api.LEE_OK
    assert tiles() == ((64, 8), (64, 16))
    assert product_lib.set_batch_shapes(s.ctx, 1, 0) == api.LEE_OK
    assert tiles()[0] == strip[0] and tiles()[1] != strip[1]
