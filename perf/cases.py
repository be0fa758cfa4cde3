"""The calls this framework is used for, as cases that can be timed.

Each case is one public call, or the few calls that a program makes in a row,
from the smallest (one beaded axon, two thousand walkers) to the largest (a
packed substrate, a batch of substrates).  ``listed`` names them, ``draw``
gives more of the same ranges, ``prepare`` makes what a program has in hand
before the call, ``run`` makes the call, ``work`` counts the bytes and
operations it cannot do without and ``exact`` gives 64-bit values where the
outputs have some.

Walks have no 64-bit values: a walker that passes within a rounding error of
a membrane takes another path in other arithmetic, so single precision and
double precision walks of the same draws part after some reflections.
"""
from __future__ import annotations

import math
import random  # noqa: F401  (draw takes a random.Random)

import numpy as np
import torch

from nozomi_b200 import batch, collide, engine, serve, simulate
from nozomi_b200.cli.simulation_main import narrow_pulse
from nozomi_b200.diffsim3d import DiffSim3d, DwiSim3d
from nozomi_b200.substrates import Substrate, beaded_axon, cell_grid, ingest_on_device
from nozomi_b200.waveforms import PGDiffWaveform

BVALUES = np.array([0.0, 1.0, 2.0, 3.0])  # ms/um^2


def listed():
    return [
        # the smallest call: one beaded axon, a few walkers, a few steps; launches and latency
        {"name": "axon_small", "kind": "walk", "axons": 1, "zspheres": 40, "N": 2003, "steps": 301, "ndir": 6,
         "cell": 1.0, "margin": 0.5, "coarsen": 4, "launch": 500},
        # one dense substrate under a PGSE protocol, from given positions, at the launch shape for packed substrates
        {"name": "packed_dwi", "kind": "walk", "axons": 200, "zspheres": 100, "N": 400000, "steps": 2000, "ndir": 30,
         "cell": 0.5, "margin": 0.5, "coarsen": 8, "launch": 2000},
        # a substrate of more than 65,536 spheres (32-bit lists) at the default shape, walkers seeded in the axons
        {"name": "large_seeded", "kind": "seeded", "axons": 500, "zspheres": 170, "N": 100003, "steps": 1000,
         "ndir": 12, "cell": 1.0, "margin": 0.5, "coarsen": 4, "launch": 500},
        # many uneven substrates and protocols in one call, positions from pinned host memory, signals back
        {"name": "batch_mixed", "kind": "batch", "jobs": 12, "axons": 120, "N": 80000, "steps": 1600, "ndir": 60,
         "threads": 256, "cell": 1.0, "launch": 1000},
        # the narrow-pulse command's work: set-up and D(t), K(t) with T2 weighting and moments at every step
        {"name": "narrow_pulse", "kind": "narrow", "axons": 300, "zspheres": 100, "N": 200000, "steps": 768},
        # the object API: phase of every walker along every direction, on the host
        {"name": "dropin_dwi", "kind": "dwi", "axons": 100, "zspheres": 100, "N": 100000, "steps": 800, "ndir": 30,
         "exact": False},
        # the same with the reference's own sums, one launch per waveform sample
        {"name": "dropin_exact", "kind": "dwi", "axons": 100, "zspheres": 100, "N": 50000, "steps": 120, "ndir": 30,
         "exact": True},
        # requests through a running server, their substrates resident
        {"name": "serve", "kind": "serve", "jobs": 6, "axons": 80, "N": 60000, "steps": 1500, "ndir": 24},
        # a substrate file's matrix to the device: fibres split and padded, cell lists and near lists built
        {"name": "ingest_build", "kind": "ingest", "axons": 400, "zspheres": 151, "cell": 0.667, "margin": 0.4},
        # the reference's padded cell table of a dense geometry
        {"name": "segments", "kind": "segments", "axons": 200, "zspheres": 100, "nseg": 20},
        # the signal of walked spins: every direction and b-value
        {"name": "signal", "kind": "signal", "N": 1000000, "ndir": 30},
        # the substrate generator's collision test, once per step of its optimisation
        {"name": "collide", "kind": "collide", "axons": 500, "zspheres": 200, "buff": 0.05},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["walk", "walk", "walk", "seeded", "batch", "batch", "narrow", "dwi", "dwi", "serve", "ingest",
                       "segments", "signal", "collide"])
    shape = {"cell": rng.choice([0.5, 0.667, 1.0]), "margin": rng.choice([0.4, 0.5]), "coarsen": rng.choice([4, 8]),
             "launch": rng.choice([500, 1000, 2000])}
    if kind == "walk":
        return {"kind": kind, "axons": _log(rng, 2, 200), "zspheres": rng.randint(40, 100), "N": _log(rng, 2000, 400000),
                "steps": rng.randint(300, 2000), "ndir": rng.randint(3, 60), **shape}
    if kind == "seeded":
        return {"kind": kind, "axons": _log(rng, 20, 500), "zspheres": rng.randint(60, 170), "N": _log(rng, 5000, 150000),
                "steps": rng.randint(300, 1500), "ndir": rng.randint(3, 60), **shape}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(3, 12), "axons": rng.randint(20, 120), "N": _log(rng, 15000, 80000),
                "steps": rng.randint(500, 1600), "ndir": rng.randint(6, 60), "threads": rng.choice([128, 256]),
                "cell": rng.choice([0.667, 1.0]), "launch": rng.choice([500, 1000])}
    if kind == "narrow":
        return {"kind": kind, "axons": _log(rng, 10, 300), "zspheres": rng.randint(50, 100), "N": _log(rng, 5000, 200000),
                "steps": rng.randint(200, 800)}
    if kind == "dwi":
        exact = rng.random() < 0.5
        return {"kind": kind, "axons": _log(rng, 5, 150), "zspheres": rng.randint(40, 100),
                "N": _log(rng, 2000, 50000 if exact else 100000), "steps": rng.randint(20, 120) if exact else
                rng.randint(200, 900), "ndir": rng.randint(3, 60), "exact": exact}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(2, 6), "axons": rng.randint(10, 100), "N": _log(rng, 5000, 60000),
                "steps": rng.randint(400, 1600), "ndir": rng.randint(6, 60)}
    if kind == "ingest":
        return {"kind": kind, "axons": _log(rng, 20, 400), "zspheres": rng.randint(60, 180),
                "cell": rng.choice([0.5, 0.667, 1.0]), "margin": round(rng.uniform(0.3, 0.6), 2)}
    if kind == "segments":
        return {"kind": kind, "axons": _log(rng, 10, 220), "zspheres": rng.randint(40, 100), "nseg": rng.randint(5, 20)}
    if kind == "signal":
        return {"kind": kind, "N": _log(rng, 10000, 1000000), "ndir": rng.randint(1, 30)}
    return {"kind": kind, "axons": _log(rng, 30, 500), "zspheres": rng.randint(60, 200),
            "buff": rng.choice([0.0, 0.05])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _profiles(rng, n, k, Lz, pitch):
    """Radii [n, k] of n beaded axons of k spheres: lognormal base radii, a
    bulge every 8 um or so, below half the pitch so that axons stay apart."""
    z = -Lz / 2 + Lz / k * (0.5 + np.arange(k))
    r0 = np.clip(rng.lognormal(-0.05, 0.3, n), 0.45, None)
    amp, beads = rng.uniform(0.2, 0.5, n), max(1, round(Lz / 8.0))
    spacing = Lz / beads
    d = np.abs((z[None, :] - rng.uniform(0, spacing, n)[:, None] + spacing / 2) % spacing - spacing / 2)
    R = r0[:, None] * (1.0 + amp[:, None] * np.exp(-d ** 2 / 4.5))
    return z, np.minimum(R, 0.49 * pitch)


def _bundle(n, k, seed, dz=0.8, pitch=2.5):
    """n parallel beaded axons of k spheres dz apart on a jittered square
    lattice of a periodic box, with images across its faces."""
    rng = np.random.default_rng(seed)
    nx = max(2, math.ceil(math.sqrt(n)))
    ny = max(2, math.ceil(n / nx))
    L = (nx * pitch, ny * pitch, k * dz)
    z, R = _profiles(rng, n, k, L[2], pitch)
    spots = rng.permutation(nx * ny)[:n]
    room = np.maximum(0.0, 0.5 * pitch - R.max(1) - 0.01)  # shifts that keep a gap to the neighbours
    P = np.stack([(spots % nx + 0.5) * pitch - L[0] / 2, (spots // nx + 0.5) * pitch - L[1] / 2], 1)
    P = P + rng.uniform(-1, 1, P.shape) * room[:, None] / math.sqrt(2)
    fibers = []
    for i in range(n):
        base = np.stack([np.full(k, P[i, 0]), np.full(k, P[i, 1]), z, R[i]], 1)
        reach = R[i].max() + 2.0
        h = min(k, math.ceil(reach / dz) + 1)
        line = np.concatenate([base[-h:] - [0, 0, L[2], 0], base, base[:h] + [0, 0, L[2], 0]])
        sx = [0.0] + [s * L[0] for s in (1, -1) if s * P[i, 0] - reach < -L[0] / 2]
        sy = [0.0] + [s * L[1] for s in (1, -1) if s * P[i, 1] - reach < -L[1] / 2]
        fibers.append(np.concatenate([line + [ox, oy, 0, 0] for ox in sx for oy in sy]))
    return Substrate(fibers, L)


def _substrate(case, seed):
    if case["axons"] == 1:
        return beaded_axon(n=case["zspheres"], Lz=float(case["zspheres"]), seed=seed)
    return _bundle(case["axons"], case["zspheres"], seed)


def _protocol(steps, ndir, seed, dt=0.005):
    te = steps * dt
    gw = PGDiffWaveform(2 * te / 3, te / 3, te, time_step=dt)
    d = np.random.default_rng(seed).standard_normal((3, ndir))
    return gw, d / np.linalg.norm(d, axis=0), gw.amplitude_for_b(BVALUES)


def _tuning(case):
    return simulate.Tuning(cell=case["cell"], near_margin=case["margin"], coarsen=case["coarsen"],
                           steps_per_launch=case["launch"])


def _job_sizes(case, seed):
    """Uneven jobs: axon counts, walkers and steps over most of an octave or two below the case's."""
    rng = np.random.default_rng(seed)
    for i in range(case["jobs"]):
        yield (max(2, int(case["axons"] * rng.uniform(0.15, 1.0))), int(case["N"] * math.exp(rng.uniform(-1.8, 0.0))),
               int(case["steps"] * rng.uniform(0.35, 1.0)), max(3, int(case["ndir"] * rng.uniform(0.2, 1.0))))


def _specs(case, seed):
    out = []
    for i, (axons, N, steps, ndir) in enumerate(_job_sizes(case, 7)):  # sizes are the case's, contents the seed's
        gw, dirs, amps = _protocol(steps, ndir, seed * 100 + i)
        out.append(batch.JobSpec(_bundle(axons, 48, seed * 100 + i), gw, dirs, amps, N, seed=seed * 100 + i,
                                 key=("case", seed, i)))
    return out


def _ordered(fibers, seed):
    """The fibres in an order of the seed's, mirrored in x and y as it says.
    Lists and pairs then differ from seed to seed while their lengths, which
    the geometry sets, stay a case's own."""
    rng = np.random.default_rng(seed)
    sign = rng.choice([-1.0, 1.0], 2)
    out = [np.array(fibers[i]) for i in rng.permutation(len(fibers))]
    for f in out:
        f[:, :2] *= sign
    return out


def _matrix(case, seed, push=0.0):
    """A substrate file's matrix: undulating fibres from z = -L/2 to z = L/2
    that continue through the face as themselves; push: the standard
    deviation of a sideways shift of each fibre (they overlap then)."""
    rng = np.random.default_rng(case["axons"] * 1000 + case["zspheres"])
    n, k = case["axons"], case["zspheres"]
    side = math.ceil(math.sqrt(n))
    pitch = 2.5
    L = max(side * pitch, 20.0)
    z = np.linspace(-L / 2, L / 2, k)
    z[-1] = L / 2
    _, R = _profiles(rng, n, k, L, pitch)
    spots = rng.permutation(side * side)[:n]
    rows = np.empty((n, k, 5))
    for a, col in enumerate((spots % side, spots // side)):
        wave = rng.uniform(0, 0.4, n)[:, None] * np.sin(2 * np.pi * z / L + rng.uniform(0, 2 * np.pi, n)[:, None])
        rows[:, :, a] = ((col + 0.5) * (L / side) - L / 2)[:, None] + wave
        rows[:, -1, a] = rows[:, 0, a]
    rows[:, :, :2] += rng.normal(0, push, (n, 1, 2)) if push else 0.0
    rows[:, :, 2] = z
    rows[:, :, 3] = R
    rows = np.stack(_ordered(rows, seed))
    rows[:, :, 4] = np.arange(n)[:, None]
    return rows.reshape(n * k, 5), L


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "seed": seed}
    if kind in ("walk", "seeded"):
        sub = _substrate(case, seed)
        gw, dirs, amps = _protocol(case["steps"], case["ndir"], seed)
        t = _tuning(case)
        dsub = simulate.device_substrate(sub, cell=t.cell, near_margin=t.near_margin)
        targets = list(range(sub.nstructures)) if kind == "seeded" else None
        st["run"] = simulate.DwiRun(dsub, gw, dirs, amps, case["N"], seed=seed, targets=targets, tuning=t)
        if kind == "walk":
            st["positions"], st["labels"] = st["run"].initial_positions()
    elif kind == "batch":
        st["specs"] = _specs(case, seed)
        st["tuning"] = simulate.Tuning(cell=case["cell"], steps_per_launch=case["launch"])
        st["cache"] = batch.SubstrateCache()
        run = batch.BatchRun(st["specs"], tuning=st["tuning"], threads=case["threads"], cache=st["cache"])
        st["positions"] = [(x.cpu().pin_memory(), lab.cpu().pin_memory()) for x, lab in run.seed_positions()]
    elif kind in ("narrow", "dwi", "segments"):
        if kind == "segments":
            sub = _bundle(case["axons"], case["zspheres"], case["axons"])
            sub = Substrate(_ordered(sub.fibers, seed), sub.L)
            st["sim"] = DiffSim3d(sub.geometry(D=2.0, T2=80.0), 1000)
            return st
        geom = _bundle(case["axons"], case["zspheres"], seed).geometry(D=2.0, T2=80.0)
        if kind == "narrow":
            sim = DiffSim3d(geom, case["N"])
        else:
            st["gwave"], dirs, _ = _protocol(case["steps"], case["ndir"], seed)
            sim = DwiSim3d(geom, case["N"], diffdir=dirs)
        sim.set_segments(20, 20, 20)
        st["sim"] = sim
    elif kind == "serve":
        st["specs"] = _specs(case, seed)
        st["cache"] = batch.SubstrateCache()
        for sp in st["specs"]:
            st["cache"].get(sp.key, sp.substrate, sp.D, sp.T2, simulate.Tuning())
        st["server"] = serve.Server(threads=256, cache=st["cache"])
    elif kind == "ingest":
        st["matrix"], st["L"] = _matrix(case, seed)
    elif kind == "signal":
        N = case["N"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        # phase of the unit waveform per axis, of freely and less freely diffusing spins, and its compensation terms
        phi = torch.randn((6, N), generator=g, device="cuda") * torch.tensor(
            [[1.0], [1.0], [1.4], [1e-7], [1e-7], [1e-7]], device="cuda")
        x = torch.rand((3, N), generator=g, device="cuda") * 40 - 20
        st["state"] = engine.FusedState.from_walkers(engine.Walkers(x, x.clone(), phi=phi))
        st["phi"] = phi
        d = np.random.default_rng(seed).standard_normal((3, case["ndir"]))
        st["dirs"] = torch.from_numpy((d / np.linalg.norm(d, axis=0)).astype(np.float32)).cuda()
        st["amps"] = torch.as_tensor(np.sqrt(1.6 * BVALUES).astype(np.float32), device="cuda")
    else:  # collide: a bundle part way through the generator's optimisation, its axons pushed into one another
        rows, st["L"] = _matrix(case, seed, push=0.25)
        st["pos"], st["r"], st["fid"] = (torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
                                         for a in (rows[:, :3], rows[:, 3], rows[:, 4]))
    return st


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("walk", "seeded"):
        r = st["run"].prepare(st.get("positions"), st.get("labels")).walk()
        sums = r.signal_sums()
        w = r.walkers()
        return {"sums": sums, "spins": w.spins, "spins0": w.spins0, "phi": w.phi, "label": w.label, "flags": w.flags}
    if kind == "batch":
        return batch.simulate_batch(st["specs"], positions=st["positions"], tuning=st["tuning"],
                                    threads=case["threads"], cache=st["cache"])
    if kind == "narrow":
        sim = st["sim"]
        sim.setup(structures=list(range(sim.geom.nstructures)), initstates_int=st["seed"])
        _, D, K = narrow_pulse(sim, case["steps"], 0.002)
        return {"D": D, "K": K, "spins": sim.spins_d.t, "spins0": sim.spins0_d.t, "sig": sim.sig_d.t}
    if kind == "dwi":
        sim = st["sim"]
        sim.setup(initstates_int=st["seed"])
        phase = sim.simulate_multi_directions(st["gwave"], exact=case["exact"])
        return {"phase": phase, "spins": sim.spins_d.t, "spins0": sim.spins0_d.t}
    if kind == "serve":
        tickets = [st["server"].submit(sp) for sp in st["specs"]]
        st["server"].drain()
        return [t.signal for t in tickets]
    if kind == "ingest":
        L = (st["L"],) * 3
        rows, spheres, lengths = ingest_on_device(st["matrix"], st["L"])
        n = len(lengths)
        sub = engine.DeviceSubstrate(spheres.cpu().numpy(), n, L, cell_grid(L, case["cell"]), np.full(n + 1, 2.0),
                                     np.full(n + 1, 80.0), near_margin=case["margin"])
        return {"rows": rows, "spheres": spheres, "lengths": lengths, "cell_start": sub.cell_start,
                "cell_count": sub.cell_count, "cell_items": sub.cell_items}
    if kind == "segments":
        sim = st["sim"]
        sim.set_segments(case["nseg"], case["nseg"], case["nseg"])
        return {"K": sim.spheres_per_segment, "segments": sim.segments}
    if kind == "signal":
        return st["state"].signal(st["dirs"], st["amps"])
    return collide.detect_collision(st["pos"], st["r"], st["fid"], st["L"], st["L"], st["L"], case["buff"])


# ---------------------------------------------------------------------------
# what a pass cannot do without, and 64-bit values
# ---------------------------------------------------------------------------
# Operations of one walker-step on these substrates: about 2.5 inside tests of
# 10, two ray-sphere fractions of 36, three phase sums of 4 and a draw of
# three normals (about 110).
STEP_FLOPS = 220


def work(case):
    kind = case["kind"]
    S = case.get("axons", 0) * case.get("zspheres", 0) * 1.4  # spheres with their images, roughly
    if kind in ("walk", "seeded"):
        N, nd = case["N"], case["ndir"]
        return {"bytes": 16 * N * (kind == "walk") + 60 * N + 16 * S + 16 * nd * 4,
                "flops": STEP_FLOPS * N * case["steps"] + 30 * N * nd * 4}
    if kind in ("batch", "serve"):
        jobs = list(_job_sizes(case, 7))
        return {"bytes": sum(16 * N + 16 * a * 68 * 1.4 for a, N, _, _ in jobs),
                "flops": sum(STEP_FLOPS * N * s + 30 * N * nd * 4 for _, N, s, nd in jobs)}
    if kind == "narrow":
        return {"bytes": 16 * S + 28 * case["N"] + 48 * case["steps"],
                "flops": (STEP_FLOPS + 20) * case["N"] * case["steps"]}
    if kind == "dwi":
        return {"bytes": 16 * S + case["N"] * (24 + 4 * case["ndir"]),
                "flops": (STEP_FLOPS + 8 * case["ndir"] * case["exact"]) * case["N"] * case["steps"]}
    if kind == "ingest":
        L = max(math.ceil(math.sqrt(case["axons"])) * 2.5, 20.0)
        cells = round(L / case["cell"]) ** 3
        members = case["axons"] * case["zspheres"] * (2.0 * (1.0 + 1.0) / case["cell"] + 1) ** 3
        return {"bytes": 40 * case["axons"] * (3 * case["zspheres"] + 100) + 8 * cells + 4 * members, "flops": 20 * members}
    if kind == "segments":
        return {"bytes": 40 * S + 4 * case["nseg"] ** 3 * 0.02 * S, "flops": 12.0 * case["nseg"] ** 3 * S}
    if kind == "signal":
        return {"bytes": 32 * case["N"], "flops": 30 * case["N"] * case["ndir"] * 4}
    n = case["axons"] * case["zspheres"]
    return {"bytes": 20 * n, "flops": 10.0 * n * 30}


def exact(case, seed):
    if case["kind"] == "signal":
        st = prepare(case, seed)
        phi = st["phi"].double()
        ph = st["dirs"].double().T @ (phi[:3] - phi[3:])
        a = st["amps"].double()
        out = torch.empty((2, case["ndir"], a.numel()), dtype=torch.float64, device=phi.device)
        for b in range(a.numel()):
            out[0, :, b] = torch.cos(a[b] * ph).sum(1)
            out[1, :, b] = torch.sin(a[b] * ph).sum(1)
        return out
    if case["kind"] == "ingest":  # each fibre with 25 spheres of itself before and after, shifted by the box
        rows, L = _matrix(case, seed)
        out = []
        for f in rows.reshape(case["axons"], case["zspheres"], 5):
            before, after = f[-25:] - [0, 0, L, 0, 0], f[:25] + [0, 0, L, 0, 0]
            out.append(np.concatenate([before, f, after]))
        out = np.concatenate(out)
        sid = np.repeat(np.arange(case["axons"], dtype=np.float64), case["zspheres"] + 50)
        return {"rows": out, "spheres": np.ascontiguousarray(np.concatenate([out[:, :4], sid[:, None]], 1).T),
                "lengths": None, "cell_start": None, "cell_count": None, "cell_items": None}
    return None  # whole numbers, or walks (see the head of this file)
