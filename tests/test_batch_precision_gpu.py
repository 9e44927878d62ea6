"""Batched direct members too large to take each pair once keep the sum and the
compensation of each source range apart until they are folded.  A body midway
between two equal heavy clumps, one in each of two source ranges, feels only a
light clump in the first: the ranges' sums cancel exactly and their low parts,
far below one unit in the last place of the sums, are the force.  A term carries
a few units of 2^-24 and 32 equal ones are summed in FP32: 4e-6 bounds that."""
import numpy as np
import pytest

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("law", [nb.LAW_REFERENCE, nb.LAW_PLUMMER])
@pytest.mark.parametrize("n", [8193, 10000])
def test_low_parts_of_source_ranges_are_kept(n, law):
    pm = np.zeros((n, 4), np.float32)
    pm[:, :3] = (0.0, 3.0, 0.0)           # everything else: massless
    pm[0] = (0.0, 0.0, 0.0, 1e-3)         # the body between the clumps
    pm[32:64] = (1.0, 0.0, 0.0, 1.0)
    pm[1024:1056] = (-1.0, 0.0, 0.0, 1.0)
    pm[64:96] = (0.5, 0.0, 0.0, 1e-9)
    eps2 = 1e-4
    q = 0.25 + eps2
    want = 1e-3 * 32 * 1e-9 * 0.5 / (0.5 * q if law == nb.LAW_REFERENCE else q ** 1.5)
    with nb.NBodyBatch(bh_threshold=1 << 20, softening2=eps2, law=law) as b:
        b.add(pm, np.zeros_like(pm))
        b.commit()
        F = b.forces(0)[0]
    assert F[0] == pytest.approx(want, rel=4e-6, abs=0.0)
    assert F[1] == F[2] == 0.0
