"""Choices of a kernel or form by number: refused on blocks of aligned rows that cannot run them, left at
the default (as before these blocks had other kernels to choose) where the rows are padded, and
followed on padded rows that can."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api
from tests.test_mean_flow_gpu import _block

pytestmark = pytest.mark.gpu


def _run(lib, case, precision, **kw):
    s = api.Solver(lib, case, precision=precision, **kw)
    s.advance(2, 0.2)
    return s.download(0)[0], s.info()


# (choice, precision, mean-flow terms): what an aligned block refuses
REFUSED = [({"filter_form": 3}, api.FP64, ""), ({"stage_kernel": 2}, api.FP64, ""),
           ({"stage_kernel": 2}, api.FP32_COMPENSATED, "su"), ({"filter_kernel": 4}, api.FP64, "")]


@pytest.mark.parametrize("choice,precision,terms", REFUSED)
def test_a_choice_that_does_not_apply(product_lib, choice, precision, terms):
    with pytest.raises(api.LeeError) as e:
        api.Solver(product_lib, _block(32, 17, 12, terms), precision=precision, **choice)
    assert e.value.code == api.LEE_ERR_UNSUPPORTED
    case = _block(33, 17, 12, terms)
    got, info = _run(product_lib, case, precision, **choice)
    want, default = _run(product_lib, case, precision)
    np.testing.assert_array_equal(got, want)
    assert (info.stage_kernel, info.filter_kernel) == (default.stage_kernel, default.filter_kernel)


@pytest.mark.parametrize("nx", [32, 33])
def test_a_choice_that_applies_is_followed(product_lib, nx):
    case = _block(nx, 17, 12)
    for form in (1, 2, 3):
        assert _run(product_lib, case, api.FP32_COMPENSATED, filter_form=form)[1].filter_rows == form
    for kernel in (1, 2):
        assert _run(product_lib, case, api.FP32_COMPENSATED, stage_kernel=kernel)[1].stage_kernel == kernel
    assert _run(product_lib, case, api.FP32_COMPENSATED, filter_kernel=4)[1].filter_kernel == 4
