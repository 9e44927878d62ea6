"""The direct sums under the Plummer law in units far from N-body ones: metres
and kilograms at the scale of a planetary system and beyond, and very small
lengths with small masses.  Every force kernel takes them: single warps and
blocks of a handle, both sizes of the allocation-free call, batched members that
take each pair once and those that do not.  A term carries a few units of 2^-24
and the sums are compensated: 5e-7 bounds their total, as in N-body units."""
import numpy as np
import pytest

import nbody_gb300 as nb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# length and mass of a unit: up to where the product m / r^3 stays in FP32's range
UNITS = [(1e10, 1e30), (1e13, 1e30), (1e15, 1e30), (1e17, 1e31), (1e-16, 1e-20)]


def state(n, unit):
    length, mass = unit
    pm, v = nb.seed_plummer(17, n)
    pm = pm.copy()
    pm[:, :3] *= np.float32(length)
    pm[:, 3] = (np.random.default_rng(n).uniform(0.1, 2.0, n) * mass).astype(np.float32)
    return pm, np.zeros_like(v)


def accel64(pm, eps2):
    x, m = pm[:, :3].astype(np.float64), pm[:, 3].astype(np.float64)
    t = np.unique(np.concatenate([[0, len(x) - 1], np.linspace(0, len(x) - 1, 300).astype(np.int64)]))
    d = x[None, :, :] - x[t][:, None, :]
    w = m[None, :] * ((d * d).sum(2) + eps2) ** -1.5
    return t, (w[:, :, None] * d).sum(1)


@pytest.mark.parametrize("unit", UNITS, ids=lambda u: "%g" % u[0])
@pytest.mark.parametrize("n", [700, 12000, 30000])
def test_handle_in_large_and_small_units(n, unit):
    pm, v = state(n, unit)
    eps2 = (0.05 * unit[0]) ** 2
    t, want = accel64(pm, eps2)
    with nb.NBodySim(kind=nb.SIM_BRUTE_FORCE, law=nb.LAW_PLUMMER, softening2=eps2) as s:
        s.init_soa(pm, v)
        a = s.compute_forces()[t] / pm[t, 3:].astype(np.float64)
    assert O.rel_l2(a / unit[1] * unit[0] ** 2, want / unit[1] * unit[0] ** 2) < 5e-7


@pytest.mark.parametrize("unit", UNITS, ids=lambda u: "%g" % u[0])
@pytest.mark.parametrize("n", [700, 30000])
def test_noalloc_in_large_and_small_units(n, unit):
    import torch

    pm, _ = state(n, unit)
    eps2 = (0.05 * unit[0]) ** 2
    t, want = accel64(pm, eps2)
    d_in = torch.from_numpy(pm).cuda()
    d_out = torch.empty_like(d_in)
    assert nb.lib().nb_direct_accel_noalloc(d_in.data_ptr(), n, d_out.data_ptr(), 1.0, eps2, nb.LAW_PLUMMER,
                                            None) == nb.NB_OK
    a = d_out.cpu().numpy()[t, :3].astype(np.float64)
    assert O.rel_l2(a / unit[1] * unit[0] ** 2, want / unit[1] * unit[0] ** 2) < 5e-7


@pytest.mark.parametrize("unit", UNITS, ids=lambda u: "%g" % u[0])
def test_batched_direct_members_in_large_and_small_units(unit):
    eps2 = (0.05 * unit[0]) ** 2
    gals = [state(n, unit) for n in (300, 5000, 9000)]
    with nb.NBodyBatch(bh_threshold=1 << 20, softening2=eps2, law=nb.LAW_PLUMMER) as b:
        for pm, v in gals:
            b.add(pm, v)
        b.commit()
        for g, (pm, _) in enumerate(gals):
            t, want = accel64(pm, eps2)
            a = b.forces(g)[t] / pm[t, 3:].astype(np.float64)
            assert O.rel_l2(a / unit[1] * unit[0] ** 2, want / unit[1] * unit[0] ** 2) < 5e-7, len(pm)
