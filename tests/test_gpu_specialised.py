"""Compile-time-plan passes against the run-time register engine.

Every plan of line_plans.inc (x, y and z lines of three-component fields, FP32 and FP64, padded
and periodic) on a thin grid with its length along its axis: the plan reports that the
axis's passes run compiled kernels, none with them turned off, and velocity and reprojected
vorticity agree bit for bit (the kernels do the run-time engine's arithmetic in its order,
with products that are never contracted).  The last test takes the lengths of the 256^3 and
512 x 512 x 256 steps together with several tiles along every axis.
"""
import os
import re

import numpy as np
import pytest

from pmlib3d_b200 import pmlib as P
from tests.helpers import gaussian_field

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
H = 1.0 / 128
AXES = "XYZ"
PASSES = {0: (0, 4), 1: (1, 3), 2: (2,)}  # x forward and inverse, y forward and inverse, z


def _plans():
    txt = open(os.path.join(ROOT, "pmlib3d_b200", "csrc", "line_plans.inc")).read()
    out = re.findall(r"^PMGPU_PLAN_([XYZ])_F(32|64)\((\d), (\d+),", txt, re.M)
    return [(AXES.index(a), P.FP32 if p == "32" else P.FP64, int(s), int(n)) for a, p, s, n in out]


def _solve(n, bc, prec, specialised, w):
    old = P.fft_specialised(specialised)
    try:
        pa = P.make_patch([-0.5 * H * c for c in n], [0.5 * H * c for c in n], (H,) * 3, bound_cond=bc, nghost=4)
        ierr, topo = P.pmlib_topology_cuboid(pa, 3)
        assert ierr == 0
        params = P.make_params(order=6, kernel=1, radius=2.0, interp=3)
        for axis in (1, 2):  # the default plans, not a schedule measured earlier in the process
            P.fft_set_schedule(n[axis] if bc[axis] else 2 * (n[axis] + 8), prec, axis, None)
        ierr, plan = P.pmlib_poisson_setup(pa, topo, params, prec)
        assert ierr == 0, P.last_error()
        wg = w(topo).astype(np.float32 if prec == P.FP32 else np.float64)
        vel = np.zeros_like(wg)
        assert P.pmlib_poisson_solve(plan, wg, vel, reproj=True) == 0, P.last_error()
        compiled = P.plan_compiled(plan)
        plan.close()
        return vel, wg, compiled
    finally:
        P.fft_specialised(old)


def _compare(n, bc, prec, passes):
    seed = sum(n)
    v1, w1, c1 = _solve(n, bc, prec, True, lambda t: gaussian_field(t, seed=seed, noise=0.05))
    v0, w0, c0 = _solve(n, bc, prec, False, lambda t: gaussian_field(t, seed=seed, noise=0.05))
    assert all(c1[p] for p in passes), c1
    assert not any(c0)
    assert np.abs(v0).max() > 0 and np.abs(w0).max() > 0
    assert np.array_equal(v1, v0) and np.array_equal(w1, w0)


def test_all_plans_listed():
    assert len(_plans()) == 154


@pytest.mark.parametrize("axis,prec,split,points", _plans())
def test_plan_equals_runtime_engine(axis, prec, split, points):
    length = points * (1 + split) * (2 if axis == 0 else 1)  # x: the packed half-length transform
    n, bc = [8, 8, 8], [0, 0, 0]
    n[axis], bc[axis] = (length // 2 - 8, 0) if split else (length, 1)
    _compare(n, tuple(bc), prec, PASSES[axis])


@pytest.mark.parametrize("prec", [P.FP32, P.FP64])
@pytest.mark.parametrize("n,bc,passes", [
    ((256, 16, 56), (0, 0, 0), (0, 2, 4)), ((24, 256, 56), (0, 0, 0), (1, 2, 3)), ((24, 56, 256), (0, 0, 0), (1, 2, 3)),
    ((512, 64, 56), (1, 1, 0), (0, 1, 2, 3, 4)), ((64, 512, 56), (1, 1, 0), (0, 1, 2, 3, 4))])
def test_step_lengths_equal_runtime_engine(n, bc, passes, prec):
    _compare(n, bc, prec, passes)
