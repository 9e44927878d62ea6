"""The plain traversal on either side of every size at which it changes: a group
walked by four warps, by two, by one with more registers and by one with fewer.
With theta 0 every cell is opened and the count of interactions is known: every
body meets every other one once.  A source that one of a group's warps lost or took
twice would change it.  At theta 0.6 the oracle's forces, within the bound of the
other sizes (its count only up to the last bit of the opening test's distance)."""
import numpy as np
import pytest

import nbody_gb300 as nb
from oracle import oracle as O

pytestmark = pytest.mark.gpu
EPS2 = 0.005 ** 2


def switch_sizes():
    """The last size of each variant: 64 bodies a group; 4, then 2 warps a group
    while they number at most 16.5 an SM, then one warp at up to 16 groups an SM."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    slots = 33 * sms // 2
    return [64 * (slots // 4), 64 * (slots // 2), 64 * 16 * sms]


def galaxy(n):
    pm, v = nb.seed_collision(45, n)
    pm[n // 3:n // 3 + 5, :3] = pm[7, :3]   # a depth-cap cell of coincident bodies
    return pm, v


@pytest.mark.parametrize("law", [nb.LAW_REFERENCE, nb.LAW_PLUMMER])
@pytest.mark.parametrize("switch", [0, 1, 2])
@pytest.mark.parametrize("past", [0, 1])
def test_every_body_meets_every_other_at_theta_zero(switch, past, law):
    n = switch_sizes()[switch] + past
    pm, v = galaxy(n)
    t = np.linspace(0, n - 1, 400).astype(np.int64)
    with nb.NBodySim(kind=nb.SIM_BARNES_HUT, theta=0.0, softening2=EPS2, law=law) as s:
        s.init_soa(pm, v)
        F = s.compute_forces()
        assert s.last_interactions() == n * (n - 1)
        assert s.tree_stats()["outside"] == 0
        F64 = s.fp64_forces(t)
    assert O.rel_l2(F[t], F64) < 1e-6


@pytest.mark.parametrize("law", [nb.LAW_REFERENCE, nb.LAW_PLUMMER])
@pytest.mark.parametrize("switch", [0, 1, 2])
@pytest.mark.parametrize("past", [0, 1])
def test_forces_are_the_oracles(switch, past, law):
    n = switch_sizes()[switch] + past
    pm, v = galaxy(n)
    pm[1, 0] = 5000.0   # outside the root
    rec = nb.records_from_soa(pm, v)
    with nb.NBodySim(kind=nb.SIM_BARNES_HUT, theta=0.6, softening2=EPS2, law=law) as s:
        s.init(rec)
        F = s.compute_forces()
        np.testing.assert_array_equal(F, s.compute_forces())
    Fo, _ = O.OracleTree(rec).forces(G=1.0, S=EPS2, theta=0.6, law=law)
    assert O.rel_l2(F, Fo) < 1e-5
