"""Periodic ghosts of a solve's velocity: every ghost holds its image, exactly.

Grids with one, two and three periodic axes, down to as many cells as ghosts of a periodic
face (the one-launch fill's limit), against the axes filled in turn on the host; corners and
edges included.
"""
import numpy as np
import pytest

from pmlib3d_b200 import pmlib as P
from tests.helpers import gaussian_field, setup_pair

pytestmark = pytest.mark.gpu

H = 0.125


@pytest.mark.parametrize("prec", [P.FP64, P.FP32])
@pytest.mark.parametrize("n,bc", [
    ((2, 8, 12), (1, 0, 0)), ((8, 2, 12), (0, 1, 0)), ((8, 10, 2), (0, 0, 1)),
    ((4, 4, 10), (1, 1, 0)), ((6, 10, 4), (1, 0, 1)), ((2, 2, 2), (1, 1, 1)),
    ((34, 18, 6), (1, 1, 1)), ((40, 24, 16), (1, 1, 0)),
])
def test_images(n, bc, prec):
    lo, hi = [-0.5 * H * c for c in n], [0.5 * H * c for c in n]
    po, to, qo, pg, tg, qg = setup_pair(lo, hi, (H,) * 3, bc, 4, interp=3, order=6)
    dt = np.float64 if prec == P.FP64 else np.float32
    w = gaussian_field(to, seed=sum(n), noise=0.05).astype(dt)
    ierr, plan = P.pmlib_poisson_setup(pg, tg, qg, prec)
    assert ierr == 0, P.last_error()
    vel = np.zeros_like(w)
    assert P.pmlib_poisson_solve(plan, w, vel, reproj=True) == 0, P.last_error()
    plan.close()
    assert np.abs(w).max() > 0
    for f in (vel, w):
        want = f.copy()
        for e in range(3):
            if not bc[e]:
                continue
            ng = tg.nghost[2 * e]
            idx = (np.arange(n[e] + 2 * ng) - ng) % n[e] + ng
            want = np.take(want, idx, axis=2 - e)  # fields are [z][y][x][component]
        assert np.array_equal(f, want)
