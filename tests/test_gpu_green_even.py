"""The Green's function from an eighth of its samples and from all of them.

The register-engine plan reads mirrored rows; a plan on the Stockham passes samples and
transforms the whole grid.  Small and ragged lengths (halves odd and even), periodic axes and
every kernel order.  Relative
L2 bound 1e-13 in FP64: the samples of a point and its mirror differ by the rounding of a
coordinate, up to 2^-53 x the length (272) in units of a cell, next to transforms of 1e-15.
"""
import numpy as np
import pytest

from pmlib3d_b200 import pmlib as P
from tests.helpers import gaussian_field, rel_l2, setup_pair

pytestmark = pytest.mark.gpu

H = 0.125


@pytest.mark.parametrize("n,bc,order", [
    ((8, 8, 8), (0, 0, 0), 2), ((9, 13, 11), (0, 0, 0), 4), ((33, 8, 57), (0, 0, 0), 8),
    ((30, 17, 41), (0, 0, 0), 10), ((24, 40, 28), (0, 0, 0), 0), ((136, 20, 12), (0, 0, 0), 6),
    ((16, 24, 20), (1, 0, 0), 6), ((24, 20, 16), (0, 1, 0), 6), ((20, 16, 24), (1, 0, 1), 6),
    ((30, 24, 20), (1, 1, 0), 6), ((16, 18, 20), (1, 1, 0), 4), ((2, 16, 2), (1, 0, 1), 6),
])
def test_even_samples(n, bc, order):
    lo, hi = [-0.5 * H * c for c in n], [0.5 * H * c for c in n]
    po, to, qo, pg, tg, qg = setup_pair(lo, hi, (H,) * 3, bc, 4, interp=3, order=order)
    w = gaussian_field(to, seed=sum(n), noise=0.05)
    out = []
    for engine in (0, 1):
        old = P.fft_engine(engine)
        try:
            ierr, plan = P.pmlib_poisson_setup(pg, tg, qg, P.FP64)
        finally:
            P.fft_engine(old)
        assert ierr == 0, P.last_error()
        vel = np.zeros_like(w)
        assert P.pmlib_poisson_solve(plan, w.copy(), vel) == 0, P.last_error()
        plan.close()
        out.append(vel)
    assert np.abs(out[1]).max() > 0
    assert rel_l2(out[0], out[1]) < 1e-13, rel_l2(out[0], out[1])
