"""Blocks whose rows are no whole number of 16 bytes: their time-loop arrays are padded to one (the
row pitch), and they run the TMA-staged kernels. Every remainder of the row length, the smallest
blocks, BC lines, holes, overset receivers and donors, reports, right-hand sides and the adjoint
against the oracle, with the tolerances of the other parity tests (FP64 1e-12 after one step,
1e-10 after N; FP32-compensated 1e-5 in p')."""
from __future__ import annotations

import numpy as np
import pytest

from camille_b200 import api, cases
from tests.test_adjoint_general_gpu import _adjoint, _dot, _fields, _run

pytestmark = pytest.mark.gpu


def _filter11(case):
    case.fd_scheme, case.filter_scheme, case.filter_strength = "FDO11P", "SFO11P", 0.2
    return case


CASES = {
    "pulse2d_33": lambda: cases.pulse2d(n=33, length=32 * 100.0 / 255.0, sponge=6, nsteps=12),
    "pulse2d_66": lambda: cases.pulse2d(n=66, length=65 * 100.0 / 255.0, sponge=8, nsteps=12),
    "pulse2d_131": lambda: cases.pulse2d(n=131, length=130 * 100.0 / 255.0, sponge=10, nsteps=12),
    "curvi3d_9": lambda: cases.curvi3d(n=9, nsteps=3, halfwidth=1.5),
    "curvi3d_33": lambda: cases.curvi3d(n=33, nsteps=8, halfwidth=2.5, sponge=4),
    "curvi3d_34": lambda: cases.curvi3d(n=34, nsteps=8, halfwidth=2.5),
    "curvi3d_67": lambda: cases.curvi3d(n=67, nsteps=4, halfwidth=3.0, sponge=5),
    "fdo11p_3d_27": lambda: _filter11(cases.curvi3d(n=27, nsteps=4, halfwidth=2.5)),
    "shear2d_131x47": lambda: cases.shear2d(nx=131, ny=47, nsteps=20),
    "wall3d_37": lambda: cases.wall3d(n=37, nsteps=6, halfwidth=3.0),
    "waves2d_95x61": lambda: cases.waves2d(nx=95, ny=61, nsteps=20),
    "jet3d_29": lambda: cases.jet3d(n=29, nsteps=6),
    "cylinder2d_67": lambda: cases.cylinder2d(nb=67, length=16.0, ntheta=73, nr=25, r_wall=0.5, r_out=4.5,
                                              first_cell=0.1, r_cut=1.9, nsteps=12, pulse=(2.0, 1.0, 1e-3, 0.8)),
}


def _cmp(case, p, o, tol):
    for b in range(len(case.blocks)):
        assert api.rel_l2(p.download(b)[0], o.download(b)[0]) <= tol


@pytest.mark.parametrize("label", list(CASES))
def test_padded_rows_match_oracle(product_lib, oracle_lib, label):
    case = CASES[label]()
    o, p = api.Solver(oracle_lib, case), api.Solver(product_lib, case)
    assert p.info().points == sum(b.npoints for b in case.blocks)
    dt = o.compute_dt()
    assert abs(p.compute_dt() - dt) <= 1e-14 * dt
    for b in range(len(case.blocks)):
        assert api.rel_l2(p.eval_rhs(b, 0.3), o.eval_rhs(b, 0.3)) <= 1e-12
    if case.overset is not None:
        mp, mo = p.get_overset(), o.get_overset()
        for k in mp:
            np.testing.assert_array_equal(mp[k], mo[k])
    o.advance(1, dt)
    p.advance(1, dt)
    _cmp(case, p, o, 1e-12)
    o.advance(case.nsteps - 1, dt)
    p.advance(case.nsteps - 1, dt)
    _cmp(case, p, o, 1e-10)
    # the reports see the points and no pad
    mn, mx = p.state_minmax()
    ys = [p.download(b)[0] for b in range(len(case.blocks))]
    np.testing.assert_array_equal(mn, np.min([y.reshape(5, -1).min(1) for y in ys], axis=0))
    np.testing.assert_array_equal(mx, np.max([y.reshape(5, -1).max(1) for y in ys], axis=0))
    f = api.Solver(product_lib, case, precision=api.FP32_COMPENSATED)
    f.advance(case.nsteps, dt)
    for b in range(len(case.blocks)):
        assert api.rel_l2(f.download(b)[0][4], o.download(b)[0][4]) <= 1e-5
    # the filter alone (it zeroes holes, which spatial::apply_filter leaves to the step's hole mask)
    p.apply_filter()
    o.apply_filter()
    for b, blk in enumerate(case.blocks):
        keep = np.ones(blk.x.shape, bool)
        if case.overset is not None:
            h = case.overset.hole_ijk[case.overset.hole_block == b]
            keep[h[:, 2], h[:, 1], h[:, 0]] = False
        assert api.rel_l2(p.download(b)[0][:, keep], o.download(b)[0][:, keep]) <= 1e-10


@pytest.mark.parametrize("precision,tol", [(api.FP64, 1e-12), (api.FP32_COMPENSATED, 2e-5)])
@pytest.mark.parametrize("label", ["curvi3d_33", "curvi3d_34", "pulse2d_66", "wall3d_37", "shear2d_131x47",
                                   "cylinder2d_67"])
def test_padded_rows_dot_product(product_lib, label, precision, tol):
    case = CASES[label]()
    rng = np.random.default_rng(3)
    x, lam = _fields(case, rng), _fields(case, rng)
    s = api.Solver(product_lib, case, precision=precision, upload=False)
    dt = s.compute_dt()
    sx = _run(s, case, x, 2, dt)
    s0 = _run(s, case, [np.zeros_like(f) for f in x], 2, dt)
    mtl = _adjoint(s, case, lam, 2, dt)
    mx = [a - b for a, b in zip(sx, s0)]
    lhs, rhs = _dot(lam, mx, case.num_dim), _dot(mtl, x, case.num_dim)
    scale = np.sqrt(_dot(lam, lam, case.num_dim) * _dot(mx, mx, case.num_dim))
    assert abs(lhs - rhs) <= tol * (max(abs(lhs), abs(rhs)) if precision == api.FP64 else scale)


@pytest.mark.parametrize("precision", [api.FP64, api.FP32_COMPENSATED])
def test_padded_rows_gradient(product_lib, oracle_lib, precision):
    """Odd sides: the objective against the oracle's, and the gradient along one direction against
    central differences of oracle objectives (exact for the quadratic objective)."""
    case = cases.adjoint3d(n=51, nsteps=12, lattice=4, nmics=16)
    s = api.Solver(product_lib, case, precision=precision)
    dt = s.compute_dt()
    J, g, mism = s.adjoint_gradient(case.nsteps, dt, checkpoint_every=4)
    tol = 1e-9 if precision == api.FP64 else 1e-4
    a0 = case.distributed.amplitudes.copy()

    def objective(a):
        case.distributed.amplitudes = a
        return api.Solver(oracle_lib, case).eval_objective(case.nsteps, dt)

    d = np.random.default_rng(1).standard_normal(a0.shape) * 1e-3
    fd = 0.5 * (objective(a0 + d) - objective(a0 - d))
    assert mism == 0
    assert abs(J - objective(a0)) <= tol * abs(J)
    assert abs(float(np.vdot(g, d)) - fd) <= 10 * tol * np.linalg.norm(g) * np.linalg.norm(d)


@pytest.mark.parametrize("precision", [api.FP64, api.FP32_COMPENSATED])
def test_padded_rows_recover_from_a_diverged_state(product_lib, precision):
    case = CASES["curvi3d_33"]()
    s = api.Solver(product_lib, case, precision=precision)
    dt = s.compute_dt()
    bad = np.full_like(case.blocks[0].state, np.nan)
    s.upload(0, bad)
    with pytest.raises(api.LeeError):
        s.advance(3, dt)
    s.upload(0, case.blocks[0].state)
    s.advance(3, dt)
    t = api.Solver(product_lib, case, precision=precision)
    t.advance(3, dt)
    np.testing.assert_array_equal(s.download(0)[0], t.download(0)[0])


@pytest.mark.parametrize("precision", [api.FP64, api.FP32_COMPENSATED])
def test_padded_batch_matches_instances(product_lib, precision):
    case = cases.batch2d(count=5, nmin=35, nmax=131, seed=9, nsteps=8)
    s = api.Solver(product_lib, case, precision=precision)
    dts = s.compute_dt_blocks()
    s.advance_blocks(case.nsteps, dts)
    for b in range(len(case.blocks)):
        one = cases.instance(case, b)
        one.monopole = one.blocks[0].monopole
        t = api.Solver(product_lib, one, precision=api.FP64)
        t.advance(case.nsteps, dts[b])
        tol = 1e-12 if precision == api.FP64 else 1e-5
        assert api.rel_l2(s.download(b)[0][4], t.download(0)[0][4]) <= tol
