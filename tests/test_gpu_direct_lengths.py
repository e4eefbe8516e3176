"""Padded lines of 11, 13 and 17 and their products have direct plans.

Half lengths whose only register radices are 11, 13 and 17, against the out-of-place
passes with the bounds of the other engine comparisons (1e-14 in FP64, 1e-6 in FP32).  The tuner measures schedules of direct plans only and skips
lines that run as convolutions, so along y and z its table tells the two apart; its plan is
held to the same bounds.
"""
import numpy as np
import pytest

from pmlib3d_b200 import pmlib as P
from tests.helpers import gaussian_field, rel_l2

pytestmark = pytest.mark.gpu

H = 0.125


def _solve(pa, t, w, prec, engine=0, tune=False):
    old = P.fft_engine(engine), P.fft_tune(tune)
    try:
        ierr, plan = P.pmlib_poisson_setup(pa, t, P.make_params(order=6, kernel=1, radius=2.0, interp=3), prec)
    finally:
        P.fft_engine(old[0])
        P.fft_tune(old[1])
    assert ierr == 0, P.last_error()
    wg, vel = w.copy(), np.zeros_like(w)
    assert P.pmlib_poisson_solve(plan, wg, vel, reproj=True) == 0, P.last_error()
    plan.close()
    return vel, wg


@pytest.mark.parametrize("prec", [P.FP64, P.FP32])
@pytest.mark.parametrize("axis,half", [(a, h) for a in (1, 2) for h in (11, 13, 17, 121, 143, 169, 187, 221, 289)] +
                         [(0, h) for h in (26, 34, 338, 442, 578)])
def test_direct(half, axis, prec):
    n = [12, 10, 8]
    n[axis] = half - 8
    pa = P.make_patch([-0.5 * H * c for c in n], [0.5 * H * c for c in n], (H,) * 3, bound_cond=(0, 0, 0), nghost=4)
    ierr, t = P.pmlib_topology_cuboid(pa, 3)
    assert ierr == 0
    w = gaussian_field(t, seed=half, noise=0.05).astype(np.float64 if prec == P.FP64 else np.float32)
    tol = 1e-14 if prec == P.FP64 else 1e-6
    plain = _solve(pa, t, w, prec, engine=1)
    before = {(e["length"], e["precision"], e["axis"]) for e in P.fft_tuned()}
    try:
        for tune in (False, True):
            for a, b in zip(_solve(pa, t, w, prec, tune=tune), plain):
                assert np.abs(b).max() > 0
                assert rel_l2(a, b) < tol, (tune, rel_l2(a, b))
        if axis:
            name = "fp64" if prec == P.FP64 else "fp32"
            assert any(e["length"] == 2 * half and e["axis"] == axis and e["precision"] == name for e in P.fft_tuned())
    finally:
        for e in P.fft_tuned():
            if (e["length"], e["precision"], e["axis"]) not in before:
                P.fft_set_schedule(e["length"], P.FP64 if e["precision"] == "fp64" else P.FP32, e["axis"], None)
