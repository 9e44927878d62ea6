"""A root cube whose float child bounds have gaps: the paths of some bodies end
early.  Where no cell that deep holds several bodies, nothing is lost: with theta 0
every body meets every other one, as in the direct sum."""
import numpy as np
import pytest

import nbody_gb300 as nb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [700, 4000, 9000])
def test_bodies_in_gaps_are_kept(n):
    pm, v = nb.seed_plummer(3, n)
    keep = (np.abs(pm[:, :3]) < 10).all(1)
    pm, v = pm[keep].copy(), v[keep].copy()
    n = len(pm)
    with nb.NBodySim(kind=nb.SIM_BARNES_HUT, theta=0.0, softening2=1e-4, bounds_half=10.1) as s:
        s.init_soa(pm, v)
        F = s.compute_forces()
        assert s.last_interactions() == n * (n - 1)
        assert s.tree_stats()["gaps"] > 0
        np.testing.assert_array_equal(F, s.compute_forces())
        F64 = s.fp64_forces(np.arange(n))
    assert O.rel_l2(F, F64) < 5e-7
