"""Mean flows with one gradient component (the one-point stage kernels read and add each component by
itself): every component of the entropy, velocity and pressure gradients alone, on the two-point, the
one-point and, under a harmonic-wave zone, the generic kernel, and around holes, against the oracle
with the tolerances of the other mean-flow tests (FP64 1e-12, FP32 1e-6)."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api, cases
from tests.test_mean_flow_gpu import _block

pytestmark = pytest.mark.gpu
COMPONENTS = [f"{f}{x}" for f in "sp" for x in range(3)] + [f"u{a}{x}" for a in range(3) for x in range(3)]


def _case(component, dim, path):
    """A Cartesian block whose mean flow varies in one field along one direction only."""
    nx, ny, nz = (36, 26, 1) if dim == 2 else (34, 20, 18)
    case = cases.holes(dim) if path == "holes" else _block(nx, ny, nz)
    blk = case.blocks[0]
    f, x = component[0], int(component[-1])
    along = np.tanh(((blk.x, blk.y, blk.z)[x] - 8.0) / 4.0)
    if f == "s":
        blk.mean[0] = 0.1 * along
    elif f == "p":
        blk.mean[4] *= 1.0 + 0.05 * along
    else:
        blk.mean[1 + int(component[1])] += 0.1 * along
    if path == "wave":
        case.harmonic_wave = cases.HarmonicWave("WAVE_ACOUSTIC", "WAVEFORM_PLANE", 0, 1e-3, 10.0)
        case.boundaries = [cases.Boundary(0, "sponge_freund_harmonicwave", 0, 0, (0, 0, 0), (4, ny - 1, nz - 1))]
    return case


@pytest.mark.parametrize("precision", [api.FP64, api.FP32_COMPENSATED])
@pytest.mark.parametrize("path", ["default", "one_point", "wave", "holes"])
@pytest.mark.parametrize("component", COMPONENTS)
def test_one_component_matches_the_oracle(product_lib, oracle_lib, component, path, precision):
    for dim in (3, 2):
        if dim == 2 and "2" in component[1:]:
            continue
        case = _case(component, dim, path)
        o = api.Solver(oracle_lib, case)
        p = api.Solver(product_lib, case, precision=precision, stage_kernel=1 if path == "one_point" else -1)
        tol = 1e-12 if precision == api.FP64 else 1e-6
        keep = np.ones(case.blocks[0].x.shape, bool)
        if path == "holes":
            h = case.overset.hole_ijk
            keep[h[:, 2], h[:, 1], h[:, 0]] = False
        assert api.rel_l2(p.eval_rhs(0, 0.3)[:, keep], o.eval_rhs(0, 0.3)[:, keep]) <= tol
        for s in (o, p):
            s.advance(3, 0.2)
        assert api.rel_l2(p.download(0)[0], o.download(0)[0]) <= tol
