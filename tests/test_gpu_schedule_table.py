"""The schedule table serves padded and periodic lines of one length, and takes back its own
entries.

A padded line of 98 points is transformed as two halves of 49 = 7 x 7: the tuner's entry
for it has to name radices that a periodic line of 98 points can run as well, and that
fft_set_schedule accepts.  Against the out-of-place passes with the bounds of the other engine
comparisons (1e-14 in FP64, 1e-6 in FP32).
"""
import numpy as np
import pytest

from pmlib3d_b200 import pmlib as P
from tests.helpers import gaussian_field, rel_l2

pytestmark = pytest.mark.gpu

H = 0.125


def _solve(n, bc, prec, engine=0, tune=False):
    pa = P.make_patch([-0.5 * H * c for c in n], [0.5 * H * c for c in n], (H,) * 3, bound_cond=bc, nghost=4)
    ierr, t = P.pmlib_topology_cuboid(pa, 3)
    assert ierr == 0
    old = P.fft_engine(engine), P.fft_tune(tune)
    try:
        ierr, plan = P.pmlib_poisson_setup(pa, t, P.make_params(order=6, kernel=1, radius=2.0, interp=3), prec)
    finally:
        P.fft_engine(old[0])
        P.fft_tune(old[1])
    assert ierr == 0, P.last_error()
    dt = np.float64 if prec == P.FP64 else np.float32
    w = gaussian_field(t, seed=sum(n), noise=0.05).astype(dt)
    for e in range(3):  # the periodic ghosts repeat the interior
        if bc[e]:
            idx = (np.arange(w.shape[2 - e]) - t.nghost[2 * e]) % n[e] + t.nghost[2 * e]
            w = np.ascontiguousarray(np.take(w, idx, axis=2 - e))
    vel = np.zeros_like(w)
    assert P.pmlib_poisson_solve(plan, w, vel) == 0, P.last_error()
    plan.close()
    return vel


def _prec(e):
    return P.FP64 if e["precision"] == "fp64" else P.FP32


@pytest.mark.parametrize("prec", [P.FP64, P.FP32])
@pytest.mark.parametrize("axis", [1, 2])
@pytest.mark.parametrize("length", [98, 224, 448])
def test_padded_then_periodic(length, axis, prec):
    tol = 1e-14 if prec == P.FP64 else 1e-6
    before = {(e["length"], e["precision"], e["axis"]) for e in P.fft_tuned()}
    free, per, bc = [8, 8, 8], [8, 8, 8], [0, 0, 0]
    free[axis], per[axis], bc[axis] = length // 2 - 8, length, 1
    try:
        a = _solve(free, (0, 0, 0), prec, tune=True)
        assert rel_l2(a, _solve(free, (0, 0, 0), prec, engine=1)) < tol
        b = _solve(per, tuple(bc), prec)
        assert rel_l2(b, _solve(per, tuple(bc), prec, engine=1)) < tol
        # the table's own entries, saved and put back
        for e in P.fft_tuned():
            assert P.fft_set_schedule(e["length"], _prec(e), e["axis"], e["radices"], e["tile"]) == 0, (e, P.last_error())
        assert np.array_equal(_solve(free, (0, 0, 0), prec), a)
    finally:
        for e in P.fft_tuned():
            if (e["length"], e["precision"], e["axis"]) not in before:
                P.fft_set_schedule(e["length"], _prec(e), e["axis"], None)


def test_tuning_returns_its_memory():
    """The tuner's scratch spectra (80 MB for these grids) go back to the pool: tuning three more
    z lengths, each a little shorter, takes no further device memory.  Bound: half of one
    length's spectrum of 50 MB."""
    import torch
    lengths = (128, 124, 120, 116)
    for n in lengths:
        P.fft_set_schedule(n, P.FP32, 2, None)
    free = []
    for n in lengths:
        _solve((112, 112, n // 2 - 8), (0, 0, 0), P.FP32, tune=True)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    for n in lengths:
        P.fft_set_schedule(n, P.FP32, 2, None)
    assert free[0] - free[-1] < 25e6, free
