"""The stage update at particle counts around its CTAs' 256: bit-identical to the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from pmlib3d_b200 import pmlib as P
from tests.helpers import setup_pair
from tests.test_gpu_advance import CASES, _particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 511, 513])
def test_counts(n, case):
    _, xmin, xmax, dx, bc, ng = CASES[case]
    po, to, _, pg, tg, _ = setup_pair(xmin, xmax, dx, bc, ng)
    arrs = [np.ascontiguousarray(a[:n]) for a in _particles(to, 600, seed=n, far=40 if bc[0] else 0)]
    ao, ag = [a.copy() for a in arrs], [a.copy() for a in arrs]
    ierr, mo = O.particles_advance(po, to, 3, 2, 0.05, *ao)
    assert ierr == 0
    ierr, mg = P.pmlib_particles_advance(pg, tg, 3, 2, 0.05, *ag)
    assert ierr == 0, P.last_error()
    assert mg == mo
    for i in (0, 1, 4, 5):
        assert np.array_equal(ag[i][:mg], ao[i][:mo]), i
