"""The plain traversal on either side of every size at which it changes: a group
walked by four warps, by two, by one with more registers and by one with fewer.
The oracle's decisions, counted, and its forces.  The galaxies are spread so that
no depth-cap cell holds bodies that differ, which the two count apart, in a cube
whose child bounds are exact; some bodies coincide, and one lies outside."""
import numpy as np
import pytest

import nbody_gb300 as nb
from oracle import oracle as O

pytestmark = pytest.mark.gpu
HALF, SCALE, EPS2 = 4096.0, 50.0, (0.005 * 50) ** 2


def switch_sizes():
    """The last size of each variant: 64 bodies a group; 4, then 2 warps a group
    while they number at most 16.5 an SM, then one warp at up to 16 groups an SM."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    slots = 33 * sms // 2
    return [64 * (slots // 4), 64 * (slots // 2), 64 * 16 * sms]


@pytest.mark.parametrize("law", [nb.LAW_REFERENCE, nb.LAW_PLUMMER])
@pytest.mark.parametrize("switch", [0, 1, 2])
@pytest.mark.parametrize("past", [0, 1])
def test_either_side_of_a_switch_decides_like_the_oracle(switch, past, law):
    n = switch_sizes()[switch] + past
    pm, v = nb.seed_collision(45, n)
    pm[:, :3] *= np.float32(SCALE)
    pm[n // 3:n // 3 + 5, :3] = pm[7, :3]
    pm[1, 0] = 5000.0
    rec = nb.records_from_soa(pm, v)
    with nb.NBodySim(kind=nb.SIM_BARNES_HUT, theta=0.6, softening2=EPS2, law=law, bounds_half=HALF) as s:
        s.init(rec)
        F = s.compute_forces()
        inter = s.last_interactions()
        np.testing.assert_array_equal(F, s.compute_forces())
        st = s.tree_stats()
        assert st["deeper_buckets"] == 0 and st["gaps"] == 0
    Fo, inter_o = O.OracleTree(rec, half=HALF).forces(G=1.0, S=EPS2, theta=0.6, law=law)
    assert inter == inter_o
    assert O.rel_l2(F, Fo) < 1e-5
