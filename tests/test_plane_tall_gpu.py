"""Blocks of very many rows, around what the grids of the direct 2-D kernels and of the 11-point stage
kernel hold in their second dimension (65535 groups of four rows, for the direct filter of eight or
sixteen): both sides of the line run, with the oracle's results, and the direct kernels with the
bits of the kernels that take over."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api
from tests.test_mean_flow_gpu import _block

pytestmark = pytest.mark.gpu
LINE = 65535 * 4


@pytest.mark.parametrize("precision,tol", [(api.FP64, 1e-12), (api.FP32_COMPENSATED, 1e-6)])
@pytest.mark.parametrize("ny", [LINE, LINE + 1, 2 * LINE + 1, 4 * LINE + 1])
def test_rows_around_the_grid_limit(product_lib, oracle_lib, ny, precision, tol):
    case = _block(12 if ny <= LINE + 1 else 9, ny, 1)
    p = api.Solver(product_lib, case, precision=precision)
    q = api.Solver(product_lib, case, precision=precision, stage_kernel=1 if precision == api.FP64 else 2,
                   filter_kernel=0, filter_form=1)
    o = api.Solver(oracle_lib, case)
    assert api.rel_l2(p.eval_rhs(0, 0.0), o.eval_rhs(0, 0.0)) <= tol
    for s in (p, q, o):
        s.advance(1, 0.2)
    got = p.download(0)[0]
    assert api.rel_l2(got, o.download(0)[0]) <= tol
    np.testing.assert_array_equal(got, q.download(0)[0])


@pytest.mark.parametrize("precision,tol", [(api.FP64, 1e-12), (api.FP32_COMPENSATED, 1e-6)])
@pytest.mark.parametrize("ny", [LINE, LINE + 1])
def test_eleven_points_around_the_grid_limit(product_lib, oracle_lib, ny, precision, tol):
    case = _block(11, ny, 1)
    case.fd_scheme, case.filter_scheme, case.filter_strength = "FDO11P", "SFO11P", 0.2
    p, o = api.Solver(product_lib, case, precision=precision), api.Solver(oracle_lib, case)
    assert api.rel_l2(p.eval_rhs(0, 0.0), o.eval_rhs(0, 0.0)) <= tol
    for s in (p, o):
        s.advance(1, 0.2)
    assert api.rel_l2(p.download(0)[0], o.download(0)[0]) <= tol
