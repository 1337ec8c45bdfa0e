"""Every form of the scalar fused filter gives the same bits, the default included: with and without a
blend, in both precisions, 2-D (the direct kernel by default) and 3-D (the two-row kernel where it
applies), every half-width, aligned and ragged rows."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api
from tests.test_filter_rows_gpu import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [api.FP64, api.FP32_COMPENSATED])
@pytest.mark.parametrize("blend", [1.0, 0.7])
@pytest.mark.parametrize("name", ["4", "8", "11"])
@pytest.mark.parametrize("nx,ny,nz", [(32, 17, 12), (67, 34, 19), (100, 21, 13), (72, 40, 1), (131, 19, 1)])
def test_the_default_has_the_bits_of_forms_1_and_2(product_lib, nx, ny, nz, name, blend, precision):
    case = _case(nx, ny, nz, name)
    case.filter_blend = blend
    got = []
    for form in (0, 1, 2):
        s = api.Solver(product_lib, case, precision=precision, filter_form=form)
        s.apply_filter()
        s.advance(2, 0.2)
        got.append(s.download(0)[0])
    np.testing.assert_array_equal(got[0], got[1])
    np.testing.assert_array_equal(got[0], got[2])


@pytest.mark.parametrize("precision", [api.FP64, api.FP32_COMPENSATED])
@pytest.mark.parametrize("blend", [1.0, 0.7])
@pytest.mark.parametrize("nx,ny,nz", [(32, 17, 12), (67, 34, 19)])
def test_the_transposed_filter_has_the_same_bits(product_lib, nx, ny, nz, blend, precision):
    case = _case(nx, ny, nz, "8")
    case.filter_blend = blend
    got = []
    for form in (0, 1, 2):
        s = api.Solver(product_lib, case, precision=precision, filter_form=form)
        s.apply_adjoint(2, 0.2)
        got.append(s.download(0)[0])
    np.testing.assert_array_equal(got[0], got[1])
    np.testing.assert_array_equal(got[0], got[2])
