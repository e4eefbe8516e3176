"""Batches whose plans carry a schedule: every patch equals its solve alone, bit for bit.

A schedule's kx tile decides which kernels hold a patch, in a batch otherwise than in a plan
of its own (the batched kernels keep less shared memory for the tile).  Lines of 136, 200 and
264 points with the digits of their compiled plans and every tile, along y and along z, and
plans made while the autotuner is on.  Bit equality needs no tolerance: both run the same
phases; the solve alone is held against the out-of-place passes with the bounds of the other
engine comparisons (1e-14 in FP64, 1e-6 in FP32).
"""
import numpy as np
import pytest

from pmlib3d_b200 import pmlib as P
from tests.helpers import gaussian_field, rel_l2

pytestmark = pytest.mark.gpu

H = 0.125
# whole-line radices of the compiled digits, by (precision, axis, half length)
RADICES = {
    (P.FP32, 1, 136): (16, 17), (P.FP32, 1, 200): (20, 20), (P.FP32, 1, 264): (22, 24),
    (P.FP64, 1, 136): (16, 17), (P.FP64, 1, 200): (10, 5, 8), (P.FP64, 1, 264): (16, 11, 3),
    (P.FP32, 2, 136): (16, 17), (P.FP32, 2, 200): (16, 5, 5), (P.FP32, 2, 264): (16, 11, 3),
    (P.FP64, 2, 136): (16, 17), (P.FP64, 2, 200): (16, 5, 5), (P.FP64, 2, 264): (16, 11, 3),
}


def _patches(half, axis):
    out = []
    for n in ([8, 8, 8], [16, 12, 10]):
        n[axis] = half - 8
        pa = P.make_patch([-0.5 * H * c for c in n], [0.5 * H * c for c in n], (H,) * 3, bound_cond=(0, 0, 0), nghost=4)
        ierr, t = P.pmlib_topology_cuboid(pa, 3)
        assert ierr == 0
        out.append((pa, t))
    return out


def _alone(pa, t, par, prec, w):
    import torch
    ierr, plan = P.pmlib_poisson_setup(pa, t, par, prec)
    assert ierr == 0, P.last_error()
    u = torch.zeros_like(w)
    assert P.pmlib_poisson_solve_dev(plan, w.data_ptr(), u.data_ptr()) == 0, P.last_error()
    torch.cuda.synchronize()
    plan.close()
    return u


def _check(half, axis, prec, tune=False):
    import torch
    dt = torch.float32 if prec == P.FP32 else torch.float64
    par = P.make_params(order=6, kernel=1, radius=2.0, interp=3)
    pts = _patches(half, axis)
    vort = [torch.from_numpy(gaussian_field(t, seed=half + i, noise=0.05)).to("cuda", dt) for i, (_, t) in enumerate(pts)]
    old = P.batch_mode(True), P.fft_tune(tune)
    try:
        b = P.Batch([p for p, _ in pts], [t for _, t in pts], par, prec)
        alone = [_alone(pa, t, par, prec, w) for (pa, t), w in zip(pts, vort)]
    finally:
        P.batch_mode(old[0])
        P.fft_tune(old[1])
    assert b.fused
    vel = [torch.full_like(w, 7.0) for w in vort]
    assert b.solve([w.data_ptr() for w in vort], [v.data_ptr() for v in vel], 0) == 0, P.last_error()
    torch.cuda.synchronize()
    b.close()
    engine = P.fft_engine(1)
    try:
        plain = [_alone(pa, t, par, prec, w) for (pa, t), w in zip(pts, vort)]
    finally:
        P.fft_engine(engine)
    for v, u, s in zip(vel, alone, plain):
        assert torch.equal(v, u), rel_l2(v.cpu().numpy(), u.cpu().numpy())
        assert float(s.abs().max()) > 0
        assert rel_l2(u.cpu().numpy(), s.cpu().numpy()) < (1e-14 if prec == P.FP64 else 1e-6)


@pytest.mark.parametrize("prec", [P.FP32, P.FP64])
@pytest.mark.parametrize("axis", [1, 2])
@pytest.mark.parametrize("half", [136, 200, 264])
@pytest.mark.parametrize("tile", [8, 4, 2])
def test_scheduled_batch(half, axis, prec, tile):
    assert P.fft_set_schedule(2 * half, prec, axis, RADICES[prec, axis, half], tile) == 0, P.last_error()
    try:
        _check(half, axis, prec)
    finally:
        P.fft_set_schedule(2 * half, prec, axis, None)


@pytest.mark.parametrize("prec", [P.FP32, P.FP64])
@pytest.mark.parametrize("half", [136, 264])
def test_tuned_batch(half, prec):
    """The tuner runs when the batch is made; the plans made after it read its table."""
    before = {(e["length"], e["precision"], e["axis"]) for e in P.fft_tuned()}
    try:
        _check(half, 2, prec, tune=True)
    finally:
        for e in P.fft_tuned():
            if (e["length"], e["precision"], e["axis"]) not in before:
                P.fft_set_schedule(e["length"], P.FP64 if e["precision"] == "fp64" else P.FP32, e["axis"], None)
