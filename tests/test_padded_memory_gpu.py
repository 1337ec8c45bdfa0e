"""Blocks whose rows are padded take about the device memory of a block without pads (their coefficients
are copies at the row pitch, whose sources go back), and report the same setup products."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api
from tests.test_mean_flow_gpu import _block

pytestmark = pytest.mark.gpu
PRECISIONS = [api.FP64, api.FP32_COMPENSATED]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("terms", ["", "u", "sup"])
@pytest.mark.parametrize("nx,ny,nz", [(33, 18, 12), (32, 18, 12), (67, 19, 1)])
def test_setup_products_match_the_oracle(product_lib, oracle_lib, nx, ny, nz, terms, precision):
    case = _block(nx, ny, nz, terms, bend=0.3, sponge=3)
    p, o = api.Solver(product_lib, case, precision=precision), api.Solver(oracle_lib, case)
    p.advance(2, 0.1)
    for what in (api.SETUP_METRICS, api.SETUP_JACOBIAN, api.SETUP_MEAN_GRADIENT, api.SETUP_SPONGE):
        want = o.get_setup(0, what)
        got = p.get_setup(0, what)
        assert np.linalg.norm(got - want) <= 1e-14 * max(np.linalg.norm(want), 1.0)


# Beyond the pads (257 -> 258 or 260 columns): FP64 alone stages its copies (8 bytes a point), and copies
# of the mean velocity and pressure stay beside their sources, 32 bytes, and p_bar's once more, 8 (of
# about 700 with a varying mean flow: 7 %).
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("terms,bound", [("", 1.03), ("sup", 1.10)])
def test_padded_rows_take_about_the_memory_of_others(product_lib, terms, bound, precision):
    per_point = []
    for nx in (256, 257):
        s = api.Solver(product_lib, _block(nx, 131, 128, terms, bend=0.3), precision=precision)
        s.advance(1, 0.1)
        i = s.info()
        per_point.append(i.device_bytes / i.points)
        s.close()
    assert per_point[1] <= bound * per_point[0]
