"""The work that users of this framework have it do, as measurable cases.

A case is one pass through a public entry point of the Python binding:

  step      NBodySim.step / update, the drop-in for INBodySim::Update: `steps`
            kick-drift steps of one galaxy, its records (position, velocity)
            written back at the end of the pass.  The same call serves the direct sum
            and Barnes-Hut.
  accel     nb_direct_accel_noalloc on device buffers: accelerations for a
            program that keeps its own state on the GPU.
  energy    NBodySim.diagnostics: the energy and momenta that every run states.
  batch     NBodyBatch: many galaxies stepped together, their state read back
            at the end of the pass.
  serve     NBodyServer: a burst of jobs submitted, ticked until all are done,
            and fetched.

Galaxies are this repository's own synthetic ones (exponential disk + bulge,
Plummer sphere, colliding spheres, the reference's spiral galaxy), in the
sizes, softenings and time steps of its benchmark configurations.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "procedural-universe_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import nbody_gb300 as nb  # noqa: E402
import nbody_serve as serve  # noqa: E402

DIRECT, BARNES_HUT = nb.SIM_BRUTE_FORCE, nb.SIM_BARNES_HUT
SEEDERS = {"disk": nb.seed_disk, "plummer": nb.seed_plummer, "collision": nb.seed_collision}
MODELS = ("disk", "plummer", "collision")   # nb_batch_add_generated's numbers

# the precompute driver's constants (the reference's SI-like units)
REF_G, REF_S, REF_SCALE, REF_DT = 6.674e-11, 10.0, 20 * 1.15e12, 0.02 / 60


def listed():
    return [
        # an interactive frame of a small scene: one update, the records back; all latency
        dict(name="frame_direct_1k", do="step", kind=DIRECT, model="plummer", n=1000, steps=1, law=0, eps=0.01,
             dt=1e-3, theta=0.5),
        # the small direct-sum configuration of the benchmark, five steps between looks
        dict(name="direct_4k", do="step", kind=DIRECT, model="plummer", n=4096, steps=5, law=0, eps=0.01, dt=1e-3,
             theta=0.5),
        # a ragged set of a program with its own device buffers
        dict(name="accel_50k", do="accel", model="plummer", n=50001, law=0, eps=0.01),
        # the large direct-sum configuration of the benchmark
        dict(name="direct_262k", do="step", kind=DIRECT, model="collision", n=262144, steps=1, law=0, eps=0.01,
             dt=1e-3, theta=0.5),
        # an update of the reference's own galaxy at the precompute driver's constants, theta and body count
        dict(name="frame_bh_4k", do="step", kind=BARNES_HUT, model="reference", n=4000, steps=1, law=0, eps=0.0, dt=0.0,
             theta=2.0),
        # a mid-sized run on an odd count, with the Plummer law
        dict(name="bh_100k", do="step", kind=BARNES_HUT, model="collision", n=100003, steps=2, law=1, eps=0.01,
             dt=1e-3, theta=0.6),
        # the benchmark's headline configuration
        dict(name="bh_1m", do="step", kind=BARNES_HUT, model="disk", n=1 << 20, steps=1, law=0, eps=0.005, dt=5e-4,
             theta=0.5),
        # the energy statement of a run
        dict(name="energy_32k", do="energy", model="disk", n=32768, law=0, eps=0.005),
        # many small galaxies, all below the Barnes-Hut threshold
        dict(name="batch_small", do="batch", made="host", galaxies=200, n_min=256, n_max=4096, threshold=8192,
             theta=0.6, eps=0.01, dt=1e-3, steps=10),
        # the benchmark's batch: uneven galaxies on both sides of the threshold
        dict(name="batch_512", do="batch", made="device", galaxies=512, n_min=256, n_max=65536, threshold=8192,
             theta=0.6, eps=0.01, dt=1e-3, steps=8),
        # one large galaxy in the batched form
        dict(name="batch_1m", do="batch", made="device", galaxies=1, n_min=1 << 20, n_max=1 << 20, threshold=8192,
             theta=0.5, eps=0.005, dt=5e-4, steps=8),
        # a burst of uneven jobs through the server
        dict(name="serve_12", do="serve", jobs=12, n_min=1024, n_max=262144, steps=20, theta=0.5, eps=0.005, dt=5e-4),
    ]


def _log_int(rng, lo, hi):
    """Log-uniform over [lo, hi], made odd half of the time."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, n | rng.randint(0, 1)))


def draw(rng):
    do = rng.choice(["direct", "direct", "accel", "bh", "bh", "bh", "energy", "batch", "batch", "serve"])
    law = rng.choice([0, 0, 1])
    if do == "direct":
        n = _log_int(rng, 300, 250000)
        return dict(do="step", kind=DIRECT, model=rng.choice(MODELS), n=n, steps=rng.randint(1, 5) if n < 20000 else 1,
                    law=law, eps=0.01, dt=1e-3, theta=0.5)
    if do == "accel":
        return dict(do="accel", model=rng.choice(MODELS), n=_log_int(rng, 500, 65536), law=law, eps=0.01)
    if do == "bh":
        n = _log_int(rng, 2000, 1 << 20)
        if n < 20000 and rng.random() < 0.3:
            return dict(do="step", kind=BARNES_HUT, model="reference", n=n, steps=rng.randint(1, 4), law=0, eps=0.0, dt=0.0,
                        theta=2.0)
        return dict(do="step", kind=BARNES_HUT, model=rng.choice(MODELS), n=n, steps=rng.randint(1, 3), law=law,
                    eps=0.005, dt=5e-4, theta=round(rng.uniform(0.4, 0.9), 2))
    if do == "energy":
        return dict(do="energy", model=rng.choice(MODELS), n=_log_int(rng, 16000, 130000), law=law, eps=0.005)
    if do == "batch":
        if rng.random() < 0.3:
            n = _log_int(rng, 100000, 1 << 20)
            return dict(do="batch", made="device", galaxies=1, n_min=n, n_max=n, threshold=8192, theta=0.5, eps=0.005,
                        dt=5e-4, steps=rng.randint(2, 8))
        return dict(do="batch", made="device", galaxies=rng.randint(16, 400), n_min=256,
                    n_max=_log_int(rng, 2000, 65536), threshold=rng.choice([1024, 8192]),
                    theta=round(rng.uniform(0.4, 0.7), 2), eps=0.01, dt=1e-3, steps=rng.randint(2, 8))
    return dict(do="serve", jobs=rng.randint(3, 16), n_min=1024, n_max=_log_int(rng, 20000, 262144),
                steps=rng.randint(5, 20), theta=0.5, eps=0.005, dt=5e-4)


def _sizes(case, count):
    """The galaxy sizes of a batch or burst: log-uniform, the same for every
    seed (the bodies are the seed's)."""
    r = np.random.default_rng(count)
    s = np.exp(r.uniform(math.log(case["n_min"]), math.log(case["n_max"]), count))
    return [int(min(case["n_max"], max(case["n_min"], round(x)))) for x in s]


def _galaxy(case, seed):
    """(pos+mass, velocity) of a single galaxy in N-body units."""
    return SEEDERS[case["model"]](seed, case["n"])


def _records(case, seed):
    if case["model"] == "reference":
        return nb.seed_reference(nb.SEEDER_GALAXY, seed, case["n"])
    return nb.records_from_soa(*_galaxy(case, seed))


def _physics(case):
    """G, softening^2, position scale, dt."""
    if case.get("model") == "reference":
        return REF_G, REF_S, REF_SCALE, REF_DT
    return 1.0, case["eps"] ** 2, 1.0, case.get("dt", 0.0)


def _batch_galaxies(case, seed):
    return [(SEEDERS[MODELS[g % 3]], seed * 1000 + g, n) for g, n in
            enumerate(_sizes(case, case["galaxies"]))]


def prepare(case, seed):
    do = case["do"]
    st = {"case": case}
    if do in ("step", "energy"):
        G, S, scale, dt = _physics(case)
        rec = _records(case, seed)
        sim = nb.NBodySim(kind=case.get("kind", DIRECT), law=case["law"], G=G, softening2=S, theta=case.get("theta", 0.5),
                          pos_scale=scale)
        sim.init(rec)
        st.update(sim=sim, rec=rec, dt=dt)
    elif do == "accel":
        pm, _ = _galaxy(case, seed)
        st["pos"] = torch.from_numpy(pm).cuda()
        st["acc"] = torch.empty_like(st["pos"])
    elif do == "batch":
        b = nb.NBodyBatch(bh_threshold=case["threshold"], bh_theta=case["theta"], softening2=case["eps"] ** 2)
        total = 0
        for seeder, s, n in _batch_galaxies(case, seed):
            if case["made"] == "host":
                b.add(*seeder(s, n))
            else:
                b.add_generated([SEEDERS[m] for m in MODELS].index(seeder), s, n)
            total += n
        b.commit()
        # pinned host buffers that the program reads the state into
        st.update(batch=b, pm=torch.empty((total, 4), pin_memory=True).numpy(),
                  vel=torch.empty((total, 4), pin_memory=True).numpy())
    else:
        srv = serve.NBodyServer(softening2=case["eps"] ** 2, theta=case["theta"])
        st.update(server=srv, jobs=[(seed * 1000 + j, n, j % 2) for j, n in enumerate(_sizes(case, case["jobs"]))])
    return st


def run(st):
    case = st["case"]
    do = case["do"]
    if do == "step":
        if case["steps"] > 1:
            st["sim"].step(st["dt"], case["steps"] - 1)
        st["sim"].update(st["dt"], st["rec"])
        # The records' velocity is a double v + a dt kept with compensation, so it
        # shows the accelerations; Forces is the same acceleration again
        # (Barnes-Hut) or zero (direct sum).
        return {"position": st["rec"]["position"], "velocity": st["rec"]["velocity"]}
    if do == "accel":
        rc = nb.lib().nb_direct_accel_noalloc(ctypes.c_void_p(st["pos"].data_ptr()), case["n"],
                                              ctypes.c_void_p(st["acc"].data_ptr()), 1.0, case["eps"] ** 2, case["law"],
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise nb.NBodyError(rc, "nb_direct_accel_noalloc")
        return st["acc"]
    if do == "energy":
        d = st["sim"].diagnostics()
        return np.concatenate([[d["kinetic"], d["potential"], d["total"], d["mass"]], d["momentum"],
                               d["angular_momentum"], d["centre_of_mass"]])
    if do == "batch":
        st["batch"].step(case["dt"], case["steps"])
        st["batch"].read_state(st["pm"], st["vel"])
        return {"pos_mass": st["pm"], "vel": st["vel"]}
    srv = st["server"]
    ids = [srv.submit(seed, n, case["steps"], case["dt"], model) for seed, n, model in st["jobs"]]
    while any(srv.tick()):
        pass
    out = []
    for j in ids:
        out.append(srv.result(j))
        srv.release(j)
    return out


# Interactions per body of a Barnes-Hut walk at theta = 0.5: 2178 measured on the
# 1,048,576-body disk with the reference's rule; they grow with log n and 1 / theta^2.
def _bh_interactions(n, theta):
    return min(n - 1.0, 109.0 * math.log2(n) * (0.5 / theta) ** 2)


def work(case):
    """Every body's state read and written once a step; 20 flops an interaction."""
    do = case["do"]
    if do == "step":
        n = case["n"]
        per = n - 1.0 if case["kind"] == DIRECT else _bh_interactions(n, case["theta"])
        return {"bytes": case["steps"] * 144.0 * n + 104.0 * n, "flops": case["steps"] * 20.0 * n * per}
    if do == "accel":
        return {"bytes": 32.0 * case["n"], "flops": 20.0 * case["n"] * (case["n"] - 1.0)}
    if do == "energy":
        n = case["n"]
        return {"bytes": 64.0 * n, "flops": 10.0 * n * (n - 1.0)}   # each pair once
    count, theta = (case["galaxies"], case["theta"]) if do == "batch" else (case["jobs"], case["theta"])
    threshold = case["threshold"] if do == "batch" else 1024
    bytes_, flops = 0.0, 0.0
    for n in _sizes(case, count):
        per = n - 1.0 if n < threshold else _bh_interactions(n, theta)
        bytes_ += case["steps"] * 144.0 * n + 32.0 * n
        flops += case["steps"] * 20.0 * n * per
    return {"bytes": bytes_, "flops": flops}


def _accel64(x, m, law, S):
    """Direct-sum accelerations / G in 64 bits (x: n x 3, m: n, on the GPU)."""
    n = x.shape[0]
    out = torch.empty_like(x)
    rows = max(1, (1 << 26) // n)
    for r in range(0, n, rows):
        d = [x[None, :, a] - x[r:r + rows, None, a] for a in range(3)]
        r2 = d[0] * d[0]
        r2 += d[1] * d[1]
        r2 += d[2] * d[2]
        w = r2.sqrt() * (r2 + S) if law == 0 else (r2 + S) ** 1.5
        w = torch.where(r2 > 0, m[None, :] / w, 0.0)
        for a in range(3):
            out[r:r + rows, a] = (w * d[a]).sum(1)
    return out


def _steps64(pm, vel, law, G, S, scale, dt, steps):
    x = torch.from_numpy(np.ascontiguousarray(pm[:, :3], np.float64)).cuda()
    m = torch.from_numpy(np.ascontiguousarray(pm[:, 3], np.float64)).cuda()
    v = torch.from_numpy(np.ascontiguousarray(vel[:, :3], np.float64)).cuda()
    for _ in range(steps):
        v = v + G * _accel64(x, m, law, S) * dt
        x = x + v * dt / scale
    return x.cpu().numpy(), v.cpu().numpy()


def exact(case, seed):
    """The direct sum and the kick-drift in 64 bits.  For the Barnes-Hut forms
    this is what they approximate, so their error is the algorithm's."""
    do = case["do"]
    if do == "step":
        if float(case["n"]) ** 2 * case["steps"] > 7e10:
            return None
        G, S, scale, dt = _physics(case)
        rec = _records(case, seed)
        pm = np.concatenate([rec["position"].astype(np.float64), rec["mass"][:, None].astype(np.float32)], axis=1)
        x, v = _steps64(pm, rec["velocity"], case["law"], G, S, scale, dt, case["steps"])
        return {"position": x, "velocity": v}
    if do == "accel":
        pm = torch.from_numpy(_galaxy(case, seed)[0].astype(np.float64)).cuda()
        a = _accel64(pm[:, :3].contiguous(), pm[:, 3].contiguous(), case["law"], case["eps"] ** 2)
        return torch.cat([a, torch.zeros_like(a[:, :1])], 1)
    if do == "energy":
        pm, vel = _galaxy(case, seed)
        x, m, v = pm[:, :3].astype(np.float64), pm[:, 3].astype(np.float64), vel[:, :3].astype(np.float64)
        gx, gm, n, eps = torch.from_numpy(x).cuda(), torch.from_numpy(m).cuda(), x.shape[0], case["eps"]
        U = 0.0
        rows = max(1, (1 << 26) // n)
        for r in range(0, n, rows):
            r2 = sum((gx[None, :, a] - gx[r:r + rows, None, a]) ** 2 for a in range(3))
            phi = torch.atan2(torch.full_like(r2, eps), r2.sqrt()) / eps if case["law"] == 0 else (r2 + eps * eps).rsqrt()
            phi[torch.arange(phi.shape[0]), torch.arange(r, r + phi.shape[0])] = 0.0
            U -= 0.5 * float((gm[r:r + rows, None] * gm[None, :] * phi).sum())
        K = 0.5 * float((m * (v * v).sum(1)).sum())
        return np.concatenate([[K, U, K + U, m.sum()], (m[:, None] * v).sum(0), (m[:, None] * np.cross(x, v)).sum(0),
                               (m[:, None] * x).sum(0) / m.sum()])
    if do == "batch" and case["made"] == "host":
        xs, vs = [], []
        for seeder, s, n in _batch_galaxies(case, seed):
            pm, vel = seeder(s, n)
            x, v = _steps64(pm, vel, 0, 1.0, case["eps"] ** 2, 1.0, case["dt"], case["steps"])
            xs.append(np.concatenate([x, pm[:, 3:].astype(np.float64)], 1))
            vs.append(np.concatenate([v, np.zeros_like(v[:, :1])], 1))
        return {"pos_mass": np.concatenate(xs), "vel": np.concatenate(vs)}
    return None
