"""Stage kernels with a non-uniform mean flow: which of the entropy, velocity and pressure gradients
are present, constant and varying coefficients, curvilinear metrics, aligned and ragged rows, single
planes of a chunk; and the 11-point difference, whose kernel moves each point's window into the line
(lines of 11 points, the shortest it takes, and up).

Tolerances: FP64 1e-12. In FP32 a right-hand side is a sum of up to 40 rounded terms of the size of
the result (the state is noise, nothing cancels): sqrt(40) * 6e-8 = 4e-7, so 1e-6."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api, cases

pytestmark = pytest.mark.gpu
PRECISIONS = [api.FP64, api.FP32_COMPENSATED]


def _block(nx, ny, nz, terms="", bend=0.0, sponge=0, seed=0):
    dim = 2 if nz == 1 else 3
    z, y, x = np.meshgrid(np.arange(nz, dtype=np.float64), np.arange(ny, dtype=np.float64),
                          np.arange(nx, dtype=np.float64), indexing="ij")
    xb = x + bend * np.sin(2.0 * np.pi * y / ny)
    yb = y + bend * np.sin(2.0 * np.pi * x / nx)
    mean = np.zeros((5,) + x.shape)
    mean[1], mean[2], mean[4] = 0.3, -0.1, 1.0 / 1.4
    wave = np.sin(0.4 * x + 0.3 * y + 0.2 * z)
    if "s" in terms:
        mean[0] = 0.1 * wave
    if "u" in terms:
        mean[1] += 0.1 * wave
        mean[2] += 0.05 * wave**2
        mean[3] = 0.05 * wave if dim == 3 else 0.0
    if "p" in terms:
        mean[4] *= 1.0 + 0.05 * wave
    rng = np.random.default_rng(seed)
    state = 1e-3 * rng.standard_normal((5,) + x.shape)
    if dim == 2:
        state[3] = 0.0
    blk = cases.Block(xb, yb, z.copy(), mean, state)
    bnd = cases.sponge_frame(dim, blk.dims, sponge) if sponge else []
    return cases.Case(name=f"block_{nx}x{ny}x{nz}", num_dim=dim, blocks=[blk], boundaries=bnd, sponge_constant=1.0)


def _check(case, product_lib, oracle_lib, precision):
    o, p = api.Solver(oracle_lib, case), api.Solver(product_lib, case, precision=precision)
    tol = 1e-12 if precision == api.FP64 else 1e-6
    assert api.rel_l2(p.eval_rhs(0, 0.0), o.eval_rhs(0, 0.0)) <= tol
    o.advance(3, 0.2)
    p.advance(3, 0.2)
    assert api.rel_l2(p.download(0)[0], o.download(0)[0]) <= tol
    assert api.rel_l2(p.eval_rhs(0, 0.0), o.eval_rhs(0, 0.0)) <= 10 * tol


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("terms", ["s", "u", "p", "su", "sp", "up", "sup"])
@pytest.mark.parametrize("nx,ny,nz", [(32, 16, 9), (36, 9, 21), (33, 18, 12), (64, 24, 1), (67, 19, 1)])
def test_mean_gradients_match_oracle(product_lib, oracle_lib, nx, ny, nz, terms, precision):
    case = _block(nx, ny, nz, terms, bend=0.3 if len(terms) != 2 else 0.0, sponge=3 if min(nx, ny) >= 12 else 0)
    if terms == "up":
        case.rk = "RUNGE_KUTTA2"
    _check(case, product_lib, oracle_lib, precision)


def test_the_two_point_kernel_stays_a_choice_of_uniform_blocks(product_lib):
    with pytest.raises(api.LeeError):
        api.Solver(product_lib, _block(32, 16, 9, "su"), precision=api.FP32_COMPENSATED, stage_kernel=2)
    api.Solver(product_lib, _block(32, 16, 9, "su"), precision=api.FP32_COMPENSATED, stage_kernel=1).advance(1, 0.2)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("terms", ["", "sup"])
@pytest.mark.parametrize("nx,ny,nz", [(11, 11, 11), (12, 13, 17), (33, 11, 15), (34, 15, 11), (40, 21, 1), (11, 37, 1)])
def test_eleven_points_match_oracle(product_lib, oracle_lib, nx, ny, nz, terms, precision):
    case = _block(nx, ny, nz, terms, bend=0.2, sponge=3 if min(nx, ny) >= 12 else 0)
    case.fd_scheme, case.filter_scheme, case.filter_strength = "FDO11P", "SFO11P", 0.2
    if terms:
        case.rk = "RUNGE_KUTTA2"
    _check(case, product_lib, oracle_lib, precision)
