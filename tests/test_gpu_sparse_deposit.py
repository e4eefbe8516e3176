"""Deposition of particles that fill few cells, on grids large enough that the deposit's
shares follow the particles: against the oracle (FP64 relative L2 1e-13, as for the other
deposition tests; FP32 4e-5: a position up to 100 cells from the origin is off by at most
2 * 100 * 2^-24 = 1.2e-5 cells after two roundings, times weight slopes of up to 1.5 on
three axes, and sums of a few terms), for clusters in a corner, across a periodic face and in one
cell, an empty particle set and one just on either side of the rule (half the cells)."""
import numpy as np
import pytest

from oracle import oracle as O
from pmlib3d_b200 import pmlib as P
from tests.helpers import rel_l2, setup_pair

pytestmark = pytest.mark.gpu

N, H = (96, 64, 100), 0.0625


def _particles(kind, rng):
    L = np.array(N) * H
    cells = N[0] * N[1] * N[2]
    if kind == "corner":
        return 0.1 * L * rng.random((3000, 3))
    if kind == "face":
        p = rng.random((5000, 3)) * np.array([0.05, 0.3, 0.3]) * L
        p[::2, 0] = L[0] - p[::2, 0]
        return p
    if kind == "one cell":
        return 0.5 * L + H * (0.3 + 0.4 * rng.random((2500, 3)))
    if kind == "empty":
        return np.zeros((0, 3))
    n = cells // 2 + (1 if kind == "above half" else -1)
    return rng.random((n, 3)) * np.array([1.0, 1.0, 0.6]) * L


@pytest.mark.parametrize("kind", ["corner", "face", "one cell", "empty", "below half", "above half"])
@pytest.mark.parametrize("bc,interp", [((0, 0, 0), 3), ((1, 0, 1), 3), ((0, 1, 0), 4)])
@pytest.mark.parametrize("prec", [P.FP64, P.FP32])
def test_sparse_deposit(kind, bc, interp, prec):
    rng = np.random.default_rng(11)
    po, to, qo, pg, tg, qg = setup_pair((0.0,) * 3, tuple(c * H for c in N), (H,) * 3, bc, 4, interp=interp, order=6)
    dt = np.float64 if prec == P.FP64 else np.float32
    pos = np.ascontiguousarray(_particles(kind, rng).astype(dt))
    val = np.ascontiguousarray(rng.standard_normal(pos.shape).astype(dt))
    to.npart = tg.npart = pos.shape[0]
    mo = np.zeros(O.topo_shape(to))
    assert O.interp_particle_mesh(to, interp, pos.astype(np.float64), val.astype(np.float64), mo, clear=True) == 0
    out = []
    for _ in range(2):
        mg = np.full(P.topo_shape(tg), 3.0, dt)
        assert P.pmlib_interp_particle_mesh(tg, qg, pos, val, mg, clear=True) == 0, P.last_error()
        out.append(mg)
    assert np.array_equal(out[0], out[1])
    if kind == "empty":
        assert not out[0].any()
    else:
        assert rel_l2(out[0], mo) < (1e-13 if prec == P.FP64 else 4e-5), rel_l2(out[0], mo)
