"""Objectives and gradients over calls long enough to replay several periods of steps at once: the
microphone traces that the replayed steps record are those of steps launched one by one, bit for bit,
and so are the gradients whose segments are recomputed from them."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [api.FP64, api.FP32_COMPENSATED])
@pytest.mark.parametrize("n", [48, 51])
def test_long_objectives_and_gradients_have_the_bits_of_single_steps(product_lib, n, precision):
    case = cases.adjoint3d(n=n, nsteps=300, lattice=4, nmics=16)
    a, b = (api.Solver(product_lib, case, precision=precision) for _ in range(2))
    b.set_graphs(False)
    dt = a.compute_dt()
    for steps in (300, 131, 7, 300):
        got = []
        for s in (a, b):
            s.upload(0, case.blocks[0].state)
            got.append(s.eval_objective(steps, dt))
        assert got[0] == got[1] and np.isfinite(got[0])
        np.testing.assert_array_equal(a.download(0)[0], b.download(0)[0])
    got = []
    for s in (a, b):
        s.upload(0, case.blocks[0].state)
        got.append(s.adjoint_gradient(290, dt, checkpoint_every=145))
    assert got[0][0] == got[1][0] and got[0][2] == got[1][2] == 0
    np.testing.assert_array_equal(got[0][1], got[1][1])
