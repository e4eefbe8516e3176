"""Launch shapes of small grids and small batches.

An x tile of short rows holds 8, 16 or 32 of them (FP64 4, 8, 16) by the number of rows (two
tiles an SM: 4736 and 9472 rows on 148 SMs, FP64 2368 and 4736): row counts on both sides, for
a periodic x of 20 cells and a free one of 5, against the out-of-place passes with the
bounds of the other engine comparisons (1e-14 in FP64, 1e-6 in FP32).  A batch of patches with
and without compiled plans runs a pass as one launch while it is small and as two beyond
(three tiles an SM): every patch equals its solve alone, bit for bit.
"""
import numpy as np
import pytest

from pmlib3d_b200 import pmlib as P
from tests.helpers import gaussian_field, rel_l2

pytestmark = pytest.mark.gpu

H = 0.125
PAR = P.make_params(order=6, kernel=1, radius=2.0, interp=3)


def _patch(n, bc):
    pa = P.make_patch([-0.5 * H * c for c in n], [0.5 * H * c for c in n], (H,) * 3, bound_cond=bc, nghost=4)
    ierr, t = P.pmlib_topology_cuboid(pa, 3)
    assert ierr == 0
    return pa, t


def _solve(pa, t, w, prec, engine=0):
    old = P.fft_engine(engine)
    try:
        ierr, plan = P.pmlib_poisson_setup(pa, t, PAR, prec)
    finally:
        P.fft_engine(old)
    assert ierr == 0, P.last_error()
    vel = np.zeros_like(w)
    assert P.pmlib_poisson_solve(plan, w.copy(), vel) == 0, P.last_error()
    plan.close()
    return vel


@pytest.mark.parametrize("prec", [P.FP64, P.FP32])
@pytest.mark.parametrize("x,periodic", [(20, 1), (5, 0)])
@pytest.mark.parametrize("rows", [(48, 49), (49, 49), (68, 69), (69, 69), (97, 97), (97, 98)])
def test_rows_of_a_tile(rows, x, periodic, prec):
    pa, t = _patch((x, rows[0] - 8, rows[1] - 8), (periodic, 0, 0))
    w = gaussian_field(t, seed=rows[0] + x, noise=0.05).astype(np.float64 if prec == P.FP64 else np.float32)
    a, b = _solve(pa, t, w, prec), _solve(pa, t, w, prec, engine=1)
    assert np.abs(b).max() > 0
    assert rel_l2(a, b) < (1e-14 if prec == P.FP64 else 1e-6), rel_l2(a, b)


@pytest.mark.parametrize("prec", [P.FP64, P.FP32])
@pytest.mark.parametrize("count", [2, 3, 12, 40])
def test_mixed_batch(count, prec):
    import torch
    dt = torch.float64 if prec == P.FP64 else torch.float32
    # 24 and 40 cells have compiled passes (lines of 32 and 48 points), 21 and 26 none
    sizes = [(24, 24, 24), (21, 26, 23), (40, 24, 40), (26, 21, 29), (20, 40, 24)]
    pts = [_patch(sizes[i % 5], ((i + 1) % 5 == 0, 0, 0)) for i in range(count)]
    vort = [torch.from_numpy(gaussian_field(t, seed=i, noise=0.05)).to("cuda", dt) for i, (_, t) in enumerate(pts)]
    b = P.Batch([p for p, _ in pts], [t for _, t in pts], PAR, prec)
    assert b.fused
    vel = [torch.full_like(w, 7.0) for w in vort]
    assert b.solve([w.data_ptr() for w in vort], [v.data_ptr() for v in vel], 0) == 0, P.last_error()
    torch.cuda.synchronize()
    b.close()
    for (pa, t), w, v in zip(pts, vort, vel):
        assert np.array_equal(v.cpu().numpy(), _solve(pa, t, w.cpu().numpy(), prec))
