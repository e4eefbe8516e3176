"""Line and x passes over the transform lengths their plans differ in.

Every length with compile-time kernels (free axes of 16 k points with their ghosts, the
explicit grids' lengths, common periodic lengths), lengths that take the run-time
engine (odd halves, one group of digits, Bluestein) and, in FP32, lines too long for
two lines a vector: a thin grid with the length along one axis, against the
out-of-place Stockham passes, which share no plan with them (the long lines against
the oracle).  Relative L2 bounds as for the other engine comparisons: 1e-14 in FP64,
1e-6 in FP32 (1e-5 against the oracle).
"""
import numpy as np
import pytest

from pmlib3d_b200 import pmlib as P
from tests.helpers import gaussian_field, rel_l2, setup_pair
from tests.test_gpu_parity import oracle_solve

pytestmark = pytest.mark.gpu

FREE = [40, 48, 64, 72, 80, 96, 104, 112, 128, 136, 144, 160, 176, 192, 200, 208, 224, 240, 256, 264, 272]
FREE_RUN_TIME = [18, 33, 54, 75, 95, 121, 150, 171, 243, 289, 330, 408]
PERIODIC = [2, 6, 34, 64, 96, 128, 150, 160, 190, 192, 256, 326, 512]
H = 0.125


def _grid(length, axis, periodic):
    n = [8, 8, 8]
    n[axis] = length if periodic else length - 8
    bc = [0, 0, 0]
    bc[axis] = 1 if periodic else 0
    return [-0.5 * H * c for c in n], [0.5 * H * c for c in n], (H,) * 3, tuple(bc), 4


def _solve(pg, tg, qg, w, prec, engine, reproj):
    old = P.fft_engine(engine)
    try:
        ierr, plan = P.pmlib_poisson_setup(pg, tg, qg, prec)
    finally:
        P.fft_engine(old)
    assert ierr == 0, P.last_error()
    dt = np.float64 if prec == P.FP64 else np.float32
    wg, vel = w.astype(dt), np.zeros(w.shape, dt)
    assert P.pmlib_poisson_solve(plan, wg, vel, reproj=reproj) == 0, P.last_error()
    plan.close()
    return vel, wg


@pytest.mark.parametrize("prec", [P.FP64, P.FP32])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("length,periodic", [(n, False) for n in FREE + FREE_RUN_TIME] + [(n, True) for n in PERIODIC])
def test_lengths(length, periodic, axis, prec):
    po, to, qo, pg, tg, qg = setup_pair(*_grid(length, axis, periodic), interp=3, order=6)
    w = gaussian_field(to, seed=length + axis, noise=0.05)
    reproj = length % 3 == 0
    a, wa = _solve(pg, tg, qg, w, prec, 0, reproj)
    b, wb = _solve(pg, tg, qg, w, prec, 1, reproj)
    tol = 1e-14 if prec == P.FP64 else 1e-6
    assert np.abs(b).max() > 0
    assert rel_l2(a, b) < tol, rel_l2(a, b)
    assert rel_l2(wa, wb) < tol, rel_l2(wa, wb)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_long_single_lines(axis):
    """2048 points (4096 transformed): FP32 tiles of single lines."""
    po, to, qo, pg, tg, qg = setup_pair(*_grid(2048, axis, False), interp=3, order=6)
    w = gaussian_field(to, seed=3 + axis, noise=0.05)
    vel_o, _, _ = oracle_solve(po, to, qo, w)
    vel, _ = _solve(pg, tg, qg, w, P.FP32, 0, False)
    assert rel_l2(vel, vel_o) < 1e-5, rel_l2(vel, vel_o)
