"""nb_direct_accel_noalloc at the sizes where its launches change: the first
that takes each pair once, row edges, sizes whose partials need several
launches in the fixed array, the largest, and a small one after it."""
import ctypes

import numpy as np
import pytest

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("law", [nb.LAW_REFERENCE, nb.LAW_PLUMMER])
@pytest.mark.parametrize("n", [8192, 8193, 10240, 12289, 16385, 33000, 50001, 65536, 700])
def test_noalloc_sizes_match_fp64(n, law):
    """A term carries a few units of 2^-24 and the sums are compensated: 5e-7
    bounds their total.  Uneven masses, some zero, and a coincident pair."""
    import torch

    L = nb.lib()
    pm, v = nb.seed_collision(41, n)
    rng = np.random.default_rng(n)
    pm[:, 3] *= rng.uniform(0.01, 2.0, n).astype(np.float32)
    pm[rng.integers(0, n, 20), 3] = 0.0
    pm[3, :3] = pm[n - 1, :3]
    m = np.where(pm[:, 3] == 0, 1, pm[:, 3]).astype(np.float64)
    t = np.unique(np.concatenate([[3, n - 1], np.linspace(0, n - 1, 1200).astype(np.int64)]))
    t = t[pm[t, 3] != 0]
    with nb.NBodySim(kind=nb.SIM_BRUTE_FORCE, law=law, softening2=1e-4) as s:
        s.init_soa(pm, v)
        ref = s.fp64_forces(t) / m[t, None]
    d_in = torch.from_numpy(pm).cuda()
    outs = []
    for _ in range(2):
        d_out = torch.full((n, 4), float("nan"), dtype=torch.float32, device="cuda")
        assert L.nb_direct_accel_noalloc(d_in.data_ptr(), n, d_out.data_ptr(), 1.0, 1e-4, law, None) == nb.NB_OK
        outs.append(d_out.cpu().numpy())
    acc = outs[0][t, :3].astype(np.float64)
    assert np.isfinite(outs[0]).all()
    assert np.linalg.norm(acc - ref) / np.linalg.norm(ref) < 5e-7
    np.testing.assert_array_equal(outs[0], outs[1])
