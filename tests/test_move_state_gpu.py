"""A state moved up and down through the staging buffer: fields that all fit at once, a part of them,
one at a time; aligned and ragged rows; several blocks of different size behind one buffer; and the
CFL maxima of several blocks."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api, cases

pytestmark = pytest.mark.gpu


def _case(shapes):
    rng = np.random.default_rng(5)
    blocks = []
    for nx, ny, nz in shapes:
        z, y, x = np.meshgrid(np.arange(nz, dtype=np.float64), np.arange(ny, dtype=np.float64),
                              np.arange(nx, dtype=np.float64) * (1.0 + 0.1 * len(blocks)), indexing="ij")
        mean = np.zeros((5,) + x.shape)
        mean[1], mean[4] = 0.3 + 0.2 * len(blocks), 1.0 / 1.4
        state = rng.standard_normal((5,) + x.shape)
        if nz == 1:
            state[3] = 0.0
        blocks.append(cases.Block(x.copy(), y.copy(), z.copy(), mean, state))
    return cases.Case(name="blocks", num_dim=2 if shapes[0][2] == 1 else 3, blocks=blocks)


# 2^22 points of staging hold all five fields of the first two, three and one of the next two
@pytest.mark.parametrize("precision", [api.FP64, api.FP32_COMPENSATED])
@pytest.mark.parametrize("shapes", [[(16, 9, 12)], [(33, 10, 9), (9, 40, 11)], [(113, 110, 100)], [(161, 180, 170)],
                                    [(65, 33, 1), (64, 9, 1), (131, 47, 1)]])
def test_upload_download(product_lib, shapes, precision):
    case = _case(shapes)
    s = api.Solver(product_lib, case, precision=precision)
    for b, blk in enumerate(case.blocks):
        out = s.download(b)[0]
        if precision == api.FP64:
            np.testing.assert_array_equal(out, blk.state)
        else:  # y = fl32(x), e = fl32(x - y): x to two roundings of 24 bits
            assert np.max(np.abs(out - blk.state) / np.maximum(np.abs(blk.state), 1e-30)) <= 2.0**-47


def test_cfl_of_several_blocks(product_lib, oracle_lib):
    case = _case([(33, 10, 9), (16, 40, 11), (9, 9, 9)])
    p, o = api.Solver(product_lib, case), api.Solver(oracle_lib, case)
    for dt in (1e-3, 0.2):
        assert abs(p.compute_cfl(dt) - o.compute_cfl(dt)) <= 1e-14 * o.compute_cfl(dt)
    assert abs(p.compute_dt() - o.compute_dt()) <= 1e-14 * o.compute_dt()


def test_a_two_dimensional_state_with_w_is_refused(product_lib):
    case = _case([(65, 33, 1)])
    s = api.Solver(product_lib, case)
    for at in (0, 1023, 1024, 65 * 33 - 1):
        for bad in (1e-300, np.nan):
            st = case.blocks[0].state.copy()
            st[3].reshape(-1)[at] = bad
            with pytest.raises(api.LeeError):
                s.upload(0, st)
    s.upload(0, case.blocks[0].state)
