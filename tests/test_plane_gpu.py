"""The direct stage and filter kernels of 2-D blocks (lee_plane.cu), single blocks and batches: sizes
around a warp's 64 columns and a CTA's rows, the smallest blocks the stencils take, every row
remainder, both RK schemes, blended and 4th-order filters, curvilinear coefficient fields, holes.
Against the oracle with the tolerances of the other parity tests; and against the kernels they stand
for, with the same bits where the order of the arithmetic is the same."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api, cases

pytestmark = pytest.mark.gpu
PRECISIONS = [api.FP64, api.FP32_COMPENSATED]


def _block(nx, ny, bend=0.0, mach=0.3, sponge=4, seed=0):
    """A 2-D block of nx x ny points (grid lines bent by ``bend``), uniform mean, smooth noise."""
    y, x = np.meshgrid(np.arange(ny, dtype=np.float64), np.arange(nx, dtype=np.float64), indexing="ij")
    xb = x + bend * np.sin(2.0 * np.pi * y / ny)
    yb = y + bend * np.sin(2.0 * np.pi * x / nx)
    x, y = xb[None], yb[None]
    mean = np.zeros((5,) + x.shape)
    mean[1], mean[2], mean[4] = mach, -0.2 * mach, 1.0 / 1.4
    rng = np.random.default_rng(seed)
    state = np.zeros((5,) + x.shape)
    for v in (0, 1, 2, 4):
        state[v] = 1e-3 * rng.standard_normal(x.shape)
    blk = cases.Block(x.copy(), y.copy(), np.zeros_like(x), mean, state)
    bnd = cases.sponge_frame(2, blk.dims, sponge) if sponge else []
    return cases.Case(name=f"block_{nx}x{ny}", num_dim=2, blocks=[blk], boundaries=bnd, sponge_constant=1.0)


SIZES = [(9, 9), (10, 17), (63, 12), (64, 31), (65, 33), (66, 9), (127, 16), (130, 40)]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("bend", [0.0, 0.3])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_sizes_match_oracle(product_lib, oracle_lib, nx, ny, bend, precision):
    case = _block(nx, ny, bend, sponge=0 if min(nx, ny) < 12 else 4)
    if (nx + ny) % 2:
        case.rk, case.filter_blend = "RUNGE_KUTTA2", 0.7
    if nx % 3 == 0:
        case.filter_order = 4
    o, p = api.Solver(oracle_lib, case), api.Solver(product_lib, case, precision=precision)
    tol = 1e-12 if precision == api.FP64 else 1e-6
    assert api.rel_l2(p.eval_rhs(0, 0.0), o.eval_rhs(0, 0.0)) <= tol
    o.advance(3, 0.2)
    p.advance(3, 0.2)
    assert api.rel_l2(p.download(0)[0], o.download(0)[0]) <= tol


@pytest.mark.parametrize("bend", [0.0, 0.3])
@pytest.mark.parametrize("nx,ny", [(64, 31), (65, 33), (130, 40)])
def test_same_bits_as_the_two_point_kernel(product_lib, nx, ny, bend):
    case = _block(nx, ny, bend)
    a = api.Solver(product_lib, case, precision=api.FP32_COMPENSATED)
    b = api.Solver(product_lib, case, precision=api.FP32_COMPENSATED, stage_kernel=2, filter_kernel=0, filter_form=1)
    a.advance(5, 0.2)
    b.advance(5, 0.2)
    np.testing.assert_array_equal(a.download(0)[0], b.download(0)[0])


def _batch(bend):
    blocks, bnd = [], []
    for q, (nx, ny) in enumerate([(9, 9), (64, 31), (65, 33), (127, 16), (130, 40), (70, 71)]):
        one = _block(nx, ny, bend, mach=0.1 * q, sponge=0 if q == 0 else 4, seed=q)
        blk = one.blocks[0]
        blk.monopole = (0.4 * nx, 0.5 * ny, 0.0, 1e-3, 0.7, 2.0, 5.0)
        blocks.append(blk)
        for b in one.boundaries:
            b.block = q
            bnd.append(b)
    return cases.Case(name="blocks", num_dim=2, blocks=blocks, boundaries=bnd, sponge_constant=1.0)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("bend", [0.0, 0.3])
def test_batch_matches_strips_and_instances(product_lib, bend, precision):
    case = _batch(bend)
    dts = [0.2 - 0.01 * q for q in range(len(case.blocks))]
    a = api.Solver(product_lib, case, precision=precision)
    b = api.Solver(product_lib, case, precision=precision)
    assert product_lib.set_batch_shapes(b.ctx, 0, 0) == api.LEE_OK
    for s in (a, b):
        s.advance_blocks(1, dts)
        s.advance_blocks(6, dts)
    for q in range(len(case.blocks)):
        ya = a.download(q)[0]
        np.testing.assert_array_equal(ya, b.download(q)[0])
        t = api.Solver(product_lib, cases.instance(case, q), precision=precision)
        t.advance(7, dts[q])
        assert api.rel_l2(ya, t.download(0)[0]) <= (1e-12 if precision == api.FP64 else 1e-6)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_batch_after_a_filter_call(product_lib, precision):
    """lee_apply_filter swaps the state's buffers: the batched filter follows them."""
    case = _batch(0.0)
    dts = [0.2] * len(case.blocks)
    a = api.Solver(product_lib, case, precision=precision)
    b = api.Solver(product_lib, case, precision=precision, batching=False)
    for s in (a, b):
        s.advance_blocks(2, dts)
        s.apply_filter()
        s.advance_blocks(3, dts)
    for q in range(len(case.blocks)):
        assert api.rel_l2(a.download(q)[0], b.download(q)[0]) <= (1e-12 if precision == api.FP64 else 1e-6)


def test_batch_wait_limit_zero_reports_timeout_and_recovers(product_lib):
    """The batched filter stages its tiles by TMA; its waits follow lee_set_wait_limit."""
    case = _batch(0.0)
    dts = [0.2] * len(case.blocks)
    s = api.Solver(product_lib, case)
    s.advance_blocks(2, dts)
    assert product_lib.set_wait_limit(s.ctx, 0.0) == api.LEE_OK
    with pytest.raises(api.LeeError) as e:
        s.advance_blocks(2, dts)
    assert e.value.code == 8
    assert product_lib.set_wait_limit(s.ctx, -1.0) == api.LEE_OK
    for b, blk in enumerate(case.blocks):
        s.upload(b, blk.state)
    s.advance_blocks(3, dts)
    t = api.Solver(product_lib, case)
    t.advance_blocks(3, dts)
    for b in range(len(case.blocks)):
        np.testing.assert_array_equal(s.download(b)[0], t.download(b)[0])
