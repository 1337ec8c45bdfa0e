"""Around the sizes where a 2-D block changes between the direct and the TMA-staged stage and filter
kernels (narrow blocks, a column of tiles partly idle, the 11-point filter on large blocks): both give
the same bits, so a block's results do not depend on the side it falls on."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api
from tests.test_filter_rows_gpu import _case

pytestmark = pytest.mark.gpu
SIZES = {
    api.FP64: [(32, 592), (32, 593), (31, 1200), (72, 592), (72, 593), (66, 1500), (64, 3552), (64, 3553), (12, 3600)],
    api.FP32_COMPENSATED: [(32, 2368), (32, 2369), (30, 2500), (72, 1200)],
}


@pytest.mark.parametrize("name", ["8", "11"])
@pytest.mark.parametrize("precision,nx,ny", [(p, *s) for p, sizes in SIZES.items() for s in sizes])
def test_same_bits_on_both_sides(product_lib, precision, nx, ny, name):
    case = _case(nx, ny, 1, name)
    case.filter_blend = 0.8
    a = api.Solver(product_lib, case, precision=precision)
    b = api.Solver(product_lib, case, precision=precision, stage_kernel=1 if precision == api.FP64 else 2,
                   filter_kernel=0, filter_form=1)
    for s in (a, b):
        s.advance(3, 0.2)
        s.apply_filter()
    np.testing.assert_array_equal(a.download(0)[0], b.download(0)[0])
