"""The fused filter of two rows per thread (two points of each in FP32, one in FP64): row counts around its tiles of 16 rows (an odd last
row, a tile of one row, the shortest lines), every half-width, compensated and plain (the adjoint's
transposed filter is covered by the adjoint tests); the same bits as the one-row kernel, and the
oracle on ragged rows (FP32: a filter is a sum of up to 33 terms per point, 1e-6; FP64 1e-13)."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api
from tests.test_mean_flow_gpu import _block

pytestmark = pytest.mark.gpu
FILTERS = {"4": ("STANDARD_CENTRAL", 4), "8": ("STANDARD_CENTRAL", 8), "11": ("SFO11P", 8)}


def _case(nx, ny, nz, name):
    case = _block(nx, ny, nz)
    case.filter_scheme, case.filter_order = FILTERS[name]
    case.filter_strength = 0.2 if name == "11" else case.filter_strength
    return case


@pytest.mark.parametrize("name", list(FILTERS))
@pytest.mark.parametrize("nx,ny,nz", [(16, 11, 13), (64, 15, 11), (68, 16, 30), (32, 17, 12), (36, 33, 14), (132, 34, 19)])
def test_same_bits_as_the_one_row_kernel(product_lib, nx, ny, nz, name):
    case = _case(nx, ny, nz, name)
    a = api.Solver(product_lib, case, precision=api.FP32_COMPENSATED, filter_kernel=0, filter_form=3)
    b = api.Solver(product_lib, case, precision=api.FP32_COMPENSATED, filter_kernel=0, filter_form=1)
    for s in (a, b):
        s.advance(2, 0.2)
        s.apply_filter()
    np.testing.assert_array_equal(a.download(0)[0], b.download(0)[0])


@pytest.mark.parametrize("precision,tol", [(api.FP64, 1e-13), (api.FP32_COMPENSATED, 1e-6)])
@pytest.mark.parametrize("name", list(FILTERS))
@pytest.mark.parametrize("nx,ny,nz", [(11, 11, 11), (33, 17, 12), (67, 31, 13), (64, 34, 20)])
def test_ragged_rows_match_oracle(product_lib, oracle_lib, nx, ny, nz, name, precision, tol):
    case = _case(nx, ny, nz, name)
    p, o = api.Solver(product_lib, case, precision=precision), api.Solver(oracle_lib, case)
    p.apply_filter()
    o.apply_filter()
    assert api.rel_l2(p.download(0)[0], o.download(0)[0]) <= tol


def test_the_two_point_form_stays_a_choice_of_the_compensated_filter(product_lib):
    with pytest.raises(api.LeeError):
        api.Solver(product_lib, _case(32, 17, 12, "8"), precision=api.FP64, filter_kernel=0, filter_form=3)
