"""Direct-sum members whose partials do not fit one launch: the batch takes them
in several, with the results of smaller batches, and the number of members is
bound by the state's memory alone."""
import numpy as np
import pytest

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu


def generated(seeds, n, bh=()):
    b = nb.NBodyBatch(bh_threshold=1 << 14, softening2=1e-4)
    for s in seeds:
        b.add_generated(1, s, n)
    for s in bh:
        b.add_generated(0, s, 20000)
    b.commit()
    return b


@pytest.mark.parametrize("bh", [(), (7,)], ids=["direct", "with_barnes_hut"])
def test_members_of_several_launches_equal_those_of_one(bh):
    """129 members of 8191 bodies fill a launch: 140 take two, twice 70 one each."""
    n, seeds = 8191, list(range(500, 640))
    got = []
    for part in (seeds, seeds[:70], seeds[70:]):
        with generated(part, n, bh) as b:
            b.step(1e-3, 2)
            pm, vel = (np.empty((n * len(part) + 20000 * len(bh), 4), np.float32) for _ in range(2))
            b.read_state(pm, vel)
            got.append((pm[:n * len(part)], vel[:n * len(part)]))
    for k in range(2):
        np.testing.assert_array_equal(got[0][k], np.concatenate([got[1][k], got[2][k]]))


def test_many_members_are_accepted():
    """4200 members of 8191 bodies: 2.2e9 entries of partials in all."""
    n, count = 8191, 4200
    with generated(range(count), n) as b, generated([0, 2077, count - 1], n) as few:
        for x in (b, few):
            x.step(1e-3, 1)
        for k, g in enumerate([0, 2077, count - 1]):
            for a, c in zip(b.read(g), few.read(k)):
                np.testing.assert_array_equal(a, c)
