"""The energy with a softening whose square underflows in FP32 (lengths in units
in which it is tiny): the pair terms are those of bare distances, and a body's
own pair, and padding, add nothing.  As for other softenings, 1e-6 bounds the sum."""
import numpy as np
import pytest

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 255, 256, 2048, 3001])
def test_plummer_energy_without_fp32_softening(n):
    pm, v = nb.seed_plummer(23, n)
    with nb.NBodySim(kind=nb.SIM_BRUTE_FORCE, law=nb.LAW_PLUMMER, softening2=1e-50) as s:
        s.init_soa(pm, v)
        d = s.diagnostics()
    x, m = pm[:, :3].astype(np.float64), pm[:, 3].astype(np.float64)
    U = sum(-m[i] * (m[i + 1:] / np.sqrt(((x[i + 1:] - x[i]) ** 2).sum(1))).sum() for i in range(n - 1))
    assert d["potential"] == pytest.approx(U, rel=1e-6, abs=0.0)
    assert d["total"] == pytest.approx(d["kinetic"] + U, rel=1e-6, abs=0.0)
