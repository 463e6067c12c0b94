"""What this framework is timed on: the work its users have it do, through its
public entry points, from a few hundred particles to millions.

A case is a dict of plain values. Its ``kind`` says which work it is:

* ``run``       molecular dynamics of one system: ``Simulation.run`` (Langevin)
                or ``run_leap_frog`` (NVE), then the new state is read;
* ``analyse``   stored configurations gone through one after another: forces,
                energy, pressure and Laplacian of each;
* ``rdf``       the radial distribution function of one configuration;
* ``replicas``  thousands of independent systems of uneven size advanced
                together (``Replicas.run``), then observables and state;
* ``surrogate`` dynamics and forces with the learned pair surrogate;
* ``train``     training steps of that surrogate (``PairSurrogate.train``).

Modes whose pair forces are float32 hand their results over as float32 arrays
(what a program with that precision keeps); the float64 mode as float64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dompap_gb300 import Simulation
from dompap_gb300.batched import ReplicaSpec, Replicas, fcc_cells_for
from dompap_gb300.mlp import PairSurrogate
from dompap_gb300.positions import FCC, generate_positions

LJ = "4*(r**-12-r**-6)"
HARMONIC = "(1-r)**2"
COSTLY_CUT = 3.0

# ------------------------------------------------------------------ the cases


def listed():
    return [
        # the classic small liquid: LJ, fcc 5^3, float64, all pairs searched for
        # the list; every step is shorter than a handful of kernel launches
        {"name": "lj500_run", "kind": "run", "potential": "lj", "basis": "fcc", "cells": "5,5,5", "density": 0.8442,
         "temperature": 1.0, "dt": 0.005, "skin": 0.5, "precision": "fp64", "integrator": "gjf",
         "list": "double loop", "forces": "neighbor list", "steps": 200},
        # energy-conserving run of a medium liquid with float32 pair forces,
        # uneven box sides
        {"name": "lj21k_nve_fp32", "kind": "run", "potential": "lj", "basis": "fcc", "cells": "19,17,16",
         "density": 0.8442, "temperature": 1.2, "dt": 0.004, "skin": 0.4, "precision": "fp32", "integrator": "nve",
         "list": "cell list", "forces": "neighbor list", "steps": 100},
        # the headline system: a million soft spheres, float64
        {"name": "harmonic3d_1M", "kind": "run", "potential": "harmonic", "basis": "fcc", "cells": "64,64,64",
         "density": 1.0, "temperature": 0.002, "dt": 0.01, "skin": 0.2, "precision": "fp64", "integrator": "gjf",
         "list": "cell list", "forces": "neighbor list", "steps": 200},
        # the same fluid in four dimensions, odd sides
        {"name": "harmonic4d_130k", "kind": "run", "potential": "harmonic", "basis": "sc", "cells": "19,19,19,19",
         "density": 1.0, "temperature": 0.002, "dt": 0.01, "skin": 0.2, "precision": "fp64", "integrator": "gjf",
         "list": "cell list", "forces": "neighbor list", "steps": 200},
        # a binary glass former: two types, two masses, per-type sigma, float64
        {"name": "mixture256k", "kind": "run", "potential": "mixture", "basis": "sc", "cells": "80,80,40",
         "density": 0.75, "temperature": 0.7, "dt": 0.004, "skin": 0.5, "precision": "fp64", "integrator": "gjf",
         "list": "cell list", "forces": "neighbor list", "steps": 60},
        # a large liquid with float32 pair forces
        {"name": "lj500k_fp32", "kind": "run", "potential": "lj", "basis": "fcc", "cells": "50,50,50",
         "density": 0.8442, "temperature": 1.35, "dt": 0.005, "skin": 0.5, "precision": "fp32", "integrator": "gjf",
         "list": "cell list", "forces": "neighbor list", "steps": 60},
        # a script that reads a few small configurations: the smallest calls
        {"name": "lj256_analyse", "kind": "analyse", "potential": "lj", "basis": "fcc", "cells": "4,4,4",
         "density": 0.8442, "temperature": 1.0, "dt": 0.005, "skin": 0.3, "precision": "fp64",
         "list": "double loop", "forces": "neighbor list", "frames": 2},
        # analysis of a stored trajectory of a larger liquid, float64
        {"name": "lj108k_analyse", "kind": "analyse", "potential": "lj", "basis": "fcc", "cells": "30,30,30",
         "density": 0.8442, "temperature": 1.0, "dt": 0.005, "skin": 0.5, "precision": "fp64",
         "list": "cell list", "forces": "neighbor list", "frames": 2},
        # structure of a liquid: all pairs of 27,436 particles into 200 bins
        {"name": "rdf27k", "kind": "rdf", "basis": "fcc", "cells": "19,19,19", "density": 0.8442, "bins": 200,
         "types": 0},
        # a parameter study: 4,096 liquids of 64 to 8,192 particles, T 0.7 to 2.0
        {"name": "replicas4096", "kind": "replicas", "replicas": 4096, "n_min": 64, "n_max": 8192, "steps": 60,
         "sample_every": 10},
        # dynamics of a costly potential through its learned surrogate
        {"name": "surrogate256k", "kind": "surrogate", "dim": 3, "basis": "fcc", "cells": "40,40,40",
         "density": 0.8, "skin": 0.3, "steps": 10},
        # training of that surrogate
        {"name": "train_b16384", "kind": "train", "samples": 262144, "batch": 16384, "steps": 64},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sides(rng, cells, dim, least):
    """Uneven sides whose product is about ``cells``."""
    k = cells ** (1.0 / dim)
    return ",".join(str(max(least, int(round(k * rng.uniform(0.88, 1.12))))) for _ in range(dim))


def draw(rng):
    kind = rng.choices(["run", "analyse", "rdf", "replicas", "surrogate", "train"], [10, 3, 2, 2, 2, 2])[0]
    if kind in ("run", "analyse"):
        potential = rng.choice(["lj", "lj", "harmonic", "harmonic", "mixture"])
        dim = rng.choice([2, 3, 4]) if potential == "harmonic" else 3
        basis = "fcc" if potential == "lj" or (potential == "harmonic" and dim == 3) else "sc"
        per_cell = 4 if basis == "fcc" else 1
        n = _log(rng, 300, 1.0e6 if potential == "harmonic" else 4.0e5)
        least = {"lj": 4, "harmonic": 4, "mixture": 8}[potential]
        c = {"kind": kind, "potential": potential, "basis": basis, "cells": _sides(rng, n / per_cell, dim, least),
             "density": {"lj": rng.uniform(0.75, 0.9), "harmonic": rng.uniform(0.9, 1.1),
                         "mixture": 0.75}[potential],
             "temperature": {"lj": rng.uniform(0.8, 1.6), "harmonic": _log(rng, 0.001, 0.01),
                             "mixture": rng.uniform(0.6, 1.0)}[potential],
             "dt": {"lj": 0.005, "harmonic": 0.01, "mixture": 0.004}[potential],
             "skin": rng.uniform(0.15, 0.3) if potential == "harmonic" else rng.uniform(0.25, 0.35),
             "precision": rng.choice(["fp64", "fp64", "fp32"]), "list": "cell list", "forces": "neighbor list"}
        if potential != "harmonic" and n > 1000:
            c["skin"] = rng.uniform(0.3, 0.6)
        if n < 12000 and rng.random() < 0.5:
            c["list"] = "double loop"
        if n < 1500 and rng.random() < 0.3:
            c["forces"] = "double loop"
        if kind == "run":
            c["integrator"] = rng.choice(["gjf", "gjf", "nve"])
            c["steps"] = int(max(20, min(200, 3e7 / n)))
        else:
            c["frames"] = rng.choice([2, 3])
        return c
    if kind == "rdf":
        return {"kind": kind, "basis": "fcc", "cells": _sides(rng, _log(rng, 500, 30000) / 4, 3, 4),
                "density": rng.uniform(0.7, 0.9), "bins": int(_log(rng, 40, 800)), "types": rng.choice([0, 2])}
    if kind == "replicas":
        top = int(_log(rng, 500, 8192))
        return {"kind": kind, "replicas": int(_log(rng, 150, 2048)), "n_min": 64, "n_max": top,
                "steps": rng.choice([20, 40, 60]), "sample_every": rng.choice([0, 5, 10])}
    if kind == "surrogate":
        dim = rng.choice([3, 3, 4])
        n = _log(rng, 3000, 180000 if dim == 3 else 36000)
        return {"kind": kind, "dim": dim, "basis": "fcc" if dim == 3 else "sc",
                "cells": _sides(rng, n / (4 if dim == 3 else 1), dim, 6 if dim == 3 else 8), "density": 0.8,
                "skin": rng.uniform(0.25, 0.4), "steps": rng.choice([4, 10])}
    return {"kind": kind, "samples": 2 ** rng.randint(14, 20), "batch": int(_log(rng, 512, 32768)),
            "steps": rng.choice([32, 64])}


# ------------------------------------------------------- inputs from the seed


def _lattice(case):
    """Lattice sites and box at the case's density."""
    cells = tuple(int(s) for s in case["cells"].split(","))
    unit = FCC if case["basis"] == "fcc" else ((0.0,) * len(cells),)
    sites = generate_positions(unit, cells, (1.0,) * len(cells))
    box = np.array(cells, dtype=np.float64)
    scale = (sites.shape[0] / np.prod(box) / case["density"]) ** (1.0 / len(cells))
    return sites * scale, box * scale


def _jitter(case):
    # soft spheres and the mixture start as the benchmark's do, other liquids
    # with about the spread that thermal motion gives them
    return {"harmonic": 0.01, "mixture": 0.02}.get(case.get("potential"), 0.05)


def _system(case, seed):
    """positions, velocities, box, types, masses of a case (host arrays)."""
    sites, box = _lattice(case)
    rng = np.random.default_rng(seed)
    n = sites.shape[0]
    pos = sites + rng.normal(0.0, _jitter(case), size=sites.shape)
    pos -= np.floor(pos / box) * box
    types = np.zeros(n, dtype=np.int32)
    masses = np.ones(n)
    if case.get("potential") == "mixture":
        types[rng.permutation(n)[: n // 2]] = 1
        masses = np.where(types == 0, 2.0, 1.0)
    elif case.get("types"):
        types = rng.integers(0, case["types"], size=n).astype(np.int32)
    vel = rng.normal(0.0, 1.0, size=pos.shape) * np.sqrt(case.get("temperature", 1.0) / masses)[:, None]
    return pos, vel, box, types, masses


SIGMA = np.array([[1.0, 1.1], [1.1, 1.2]])
EPSILON = np.ones((2, 2))


def _potential(case):
    """(expression, r_cut) of the case's pair potential."""
    name = case.get("potential", "lj")
    return (HARMONIC, 1.0) if name == "harmonic" else (LJ, 2.5)


def _simulation(case, seed):
    pos, vel, box, types, masses = _system(case, seed)
    np.random.seed(seed)
    capacity = {2: 64, 3: 64, 4: 96}[pos.shape[1]] if case.get("potential") == "harmonic" else 256
    sim = Simulation(positions=pos, velocities=vel, box_vectors=box, particle_types=types, masses=masses,
                     neighbor_list_skin=case.get("skin", 0.3), max_number_of_neighbors=capacity,
                     precision=case.get("precision", "fp64"))
    sim.force_method_str = case.get("forces", "neighbor list")
    sim.set_pair_potential(*_potential(case))
    if case.get("potential") == "mixture":
        sim.set_pair_potential_parameters(sigma=SIGMA, epsilon=EPSILON)
    sim.set_neighbor_list(skin=case.get("skin", 0.3), max_number_of_neighbors=capacity,
                          method_str=case.get("list", "cell list"))
    sim.set_integrator(time_step=case.get("dt", 0.005), target_temperature=case.get("temperature", 1.0),
                       temperature_damping_time=0.1)
    return sim


def _frames(case, seed):
    """Configurations far apart, as the frames of a stored trajectory are."""
    sites, box = _lattice(case)
    rng = np.random.default_rng([seed, 7])
    out = []
    for _ in range(case["frames"]):
        pos = sites + rng.uniform(0.0, 1.0, size=box.shape) * box + rng.normal(0.0, _jitter(case), size=sites.shape)
        out.append(np.ascontiguousarray(pos - np.floor(pos / box) * box))
    return out


def _replica_specs(case, seed):
    """fcc liquids of log-uniform sizes (the study's, the same for every seed;
    boxes shorter than two cuts drawn again) at density 0.8442, T 0.7 to 2.0."""
    study = np.random.default_rng([case["replicas"], case["n_min"], case["n_max"]])
    rng = np.random.default_rng(seed)
    a = (4.0 / 0.8442) ** (1.0 / 3.0)
    specs = []
    while len(specs) < case["replicas"]:
        cells = fcc_cells_for(int(round(np.exp(study.uniform(np.log(case["n_min"]), np.log(case["n_max"]))))))
        box = np.array(cells, dtype=np.float64) * a
        if box.min() < 5.0:
            continue
        pos = generate_positions(FCC, cells, (a, a, a))
        pos += rng.normal(0.0, 0.02, size=pos.shape)
        pos -= np.floor(pos / box) * box
        temperature = float(rng.uniform(0.7, 2.0))
        specs.append(ReplicaSpec(pos, rng.normal(0.0, np.sqrt(temperature), size=pos.shape), box, temperature))
    return specs


def _costly_terms(r):
    """u and f = -du/dr of the terms the surrogate learns (numpy, float64)."""
    g = 0.5 * np.exp(-((r - 1.5) ** 2) / 0.02)
    e = 0.1 * np.exp(-r)
    u = g + e * np.cos(4 * r)
    f = g * (r - 1.5) / 0.01 + e * (np.cos(4 * r) + 4 * np.sin(4 * r))
    return u, f


def _shift():
    """u and du/dr of the costly potential at its cut."""
    r = np.float64(COSTLY_CUT)
    u, f = _costly_terms(r)
    return float(u + 4 * (r**-12 - r**-6)), float(-f - 48 * r**-13 + 24 * r**-7)


def _costly_string():
    u, du = _shift()
    raw = LJ + " + 0.5*exp(-(r-1.5)**2/0.02) + 0.1*cos(4*r)*exp(-r)"
    return f"{raw} - ({u!r}) - (r - {COSTLY_CUT!r})*({du!r})"


def _samples(seed, n):
    """Training radii, and the normalisation PairSurrogate takes from them."""
    r = np.random.default_rng(seed).uniform(0.8, COSTLY_CUT, size=n)
    u, f = _costly_terms(r)
    s = r * r
    norm = np.array([s.mean(), 1.0 / s.std(), np.max(np.abs(u)), np.max(np.abs(f * r))], dtype=np.float32)
    return r, norm


def _bf16(x):
    return torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).bfloat16().double().numpy()


def _network(seed, norm, fitted):
    """Weights of a 1-64-64-2 tanh network: steps spread over the range, a
    random second layer and, when ``fitted``, a read-out by regularised least
    squares on the costly terms (a network in use, without training time)."""
    rng = np.random.default_rng([seed, 3])
    x0, x1 = ((np.array([0.8, COSTLY_CUT]) ** 2) - float(norm[0])) * float(norm[1])
    centres = x0 + (x1 - x0) * (np.arange(64) + 0.5) / 64
    w1 = 0.7 * 64 / (x1 - x0) * np.where(rng.random(64) < 0.5, -1.0, 1.0)
    p = np.zeros(64 + 64 + 4096 + 64 + 128 + 2)
    p[0:64], p[64:128] = w1, -w1 * centres
    p[128:4224] = rng.normal(0.0, 1.0 / 8.0, 4096)
    p[4288:4416] = rng.normal(0.0, 1.0 / 8.0, 128)
    if fitted:
        r = np.linspace(0.8, COSTLY_CUT, 4096)
        u, f = _costly_terms(r)
        x = (r * r - float(norm[0])) * float(norm[1])
        h1 = np.tanh(np.outer(x, p[0:64]) + p[64:128])
        h2 = np.tanh(h1 @ _bf16(p[128:4224]).reshape(64, 64).T)
        a = np.concatenate([h2, np.ones((4096, 1))], axis=1)
        y = np.stack([u / float(norm[2]), f * r / float(norm[3])], axis=1)
        w = np.linalg.solve(a.T @ a + 0.3 * np.eye(65), a.T @ y)
        p[4288:4416] = w[:64].T.reshape(-1)
        p[4416:4418] = w[64]
    return p.astype(np.float32)


# -------------------------------------------------------------------- running


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        return {"case": case, "sim": _simulation(case, seed)}
    if kind == "analyse":
        return {"case": case, "sim": _simulation(case, seed), "frames": _frames(case, seed)}
    if kind == "rdf":
        sim = _simulation(case, seed)
        return {"case": case, "sim": sim, "bins": np.linspace(0.5, float(np.min(_lattice(case)[1])) / 2,
                                                              case["bins"] + 1)}
    if kind == "replicas":
        specs = _replica_specs(case, seed)
        return {"case": case, "replicas": Replicas(specs, LJ, 2.5, seed=seed)}
    n = case.get("samples", 4096)
    surrogate = PairSurrogate(_costly_string(), COSTLY_CUT, n_samples=n, seed=seed)
    surrogate.set_params(_network(seed, surrogate.norm, fitted=kind == "surrogate"))
    if kind == "train":
        return {"case": case, "surrogate": surrogate}
    pos, vel, box, types, masses = _system(case, seed)
    np.random.seed(seed)
    capacity = 256 if case["dim"] == 3 else 512
    sim = Simulation(positions=pos, velocities=vel, box_vectors=box, particle_types=types, masses=masses,
                     neighbor_list_skin=case["skin"], max_number_of_neighbors=capacity)
    sim.set_pair_potential(_costly_string(), COSTLY_CUT)
    sim.set_pair_surrogate(surrogate)
    sim.set_neighbor_list(skin=case["skin"], max_number_of_neighbors=capacity, method_str="cell list")
    sim.set_integrator(time_step=0.004, target_temperature=1.0, temperature_damping_time=0.1)
    return {"case": case, "sim": sim, "surrogate": surrogate}


def _single(array):
    """What a program with float32 forces keeps of a result."""
    return torch.from_numpy(np.asarray(array)).float()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        sim = state["sim"]
        if case["integrator"] == "nve":
            sim.run_leap_frog(case["steps"])
        else:
            sim.run(case["steps"])
        out = [sim.positions, sim.velocities, sim.image_positions]
        return [_single(out[0]), _single(out[1]), out[2]] if case["precision"] == "fp32" else out
    if kind == "analyse":
        sim = state["sim"]
        out = []
        for frame in state["frames"]:
            sim.positions = frame
            res = [sim.get_forces(), sim.get_laplacian(),
                   np.array([sim.get_potential_energy(), sim.get_virial(), sim.get_pressure()])]
            out.append([_single(x) for x in res] if case["precision"] == "fp32" else res)
        return out
    if kind == "rdf":
        sim, bins = state["sim"], state["bins"]
        if not case["types"]:
            return list(sim.get_radial_distribution_function(bins))
        return [sim.get_radial_distribution_function(bins, type_a=a, type_b=b)[1] for a, b in ((0, 0), (0, 1))]
    if kind == "replicas":
        reps = state["replicas"]
        reps.run(case["steps"], sample_every=case["sample_every"])
        pos, vel, img = reps.state()
        obs = reps.observables()
        out = [_single(pos), _single(vel), img]
        if case["sample_every"]:
            out += [_single(obs[k]) for k in ("potential_energy_per_particle", "temperature", "pressure")]
        return out
    if kind == "train":
        sur = state["surrogate"]
        losses = sur.train(case["steps"], batch=case["batch"])
        return [losses, sur.params()]
    sim = state["sim"]
    sim.run(case["steps"])
    return [_single(sim.positions), _single(sim.velocities), _single(sim.get_forces()),
            np.float32(sim.get_potential_energy())]


# ----------------------------------------------------- what a pass has to move


def _sphere(dim, r):
    return math.pi ** (dim / 2) / math.gamma(dim / 2 + 1) * r**dim


def _replica_particles(case):
    """Expected particles of a batch: sizes are log-uniform; boxes shorter than
    two cuts (about 130 particles) are drawn again."""
    lo, hi = max(case["n_min"], 130), max(case["n_max"], 140)
    return case["replicas"] * (hi - lo) / math.log(hi / lo)


def work(case):
    """Bytes: each step (or frame) reads the state once and writes the new one
    once. Flops: each pair inside the cut once, with its displacement, its
    pair terms and the two accumulations, and the update of each particle."""
    kind = case["kind"]
    if kind == "train":
        per = 2 * (64 + 4096 + 128) * 3
        return {"bytes": case["steps"] * case["batch"] * 12.0, "flops": float(case["steps"] * case["batch"] * per)}
    if kind == "replicas":
        n, dim = _replica_particles(case), 3
        pairs = n * 0.8442 * _sphere(3, 2.5) / 2
        return {"bytes": case["steps"] * n * 6.0 * 8 * dim, "flops": case["steps"] * (pairs * 30 + n * 20 * dim)}
    cells = [int(s) for s in case["cells"].split(",")]
    dim = len(cells)
    n = float(np.prod(cells)) * (4 if case["basis"] == "fcc" else 1)
    if kind == "rdf":
        return {"bytes": n * 8 * dim + case["bins"] * 16.0, "flops": n * n / 2 * 12 * (1 if not case["types"] else 0.75)}
    if kind == "surrogate":
        pairs = n * case["density"] * _sphere(dim, COSTLY_CUT) / 2
        per = 2 * (64 + 4096 + 128) + 30
        return {"bytes": (case["steps"] + 1) * n * 6.0 * 8 * dim, "flops": (case["steps"] + 2) * pairs * per}
    cut = {"lj": 2.5, "harmonic": 1.0, "mixture": 2.5 * 1.1}[case["potential"]]
    pairs = n * case["density"] * _sphere(dim, cut) / 2
    if kind == "analyse":
        return {"bytes": case["frames"] * n * (2 * 8 * dim + 8.0), "flops": case["frames"] * pairs * 80}
    arrays = 4.0 if case["integrator"] == "nve" else 6.0
    return {"bytes": case["steps"] * n * arrays * 8 * dim, "flops": case["steps"] * (pairs * 30 + n * 20 * dim)}


# -------------------------------------------------- the same results in 64 bits


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pairs(x, box, cut):
    """All ordered pairs (i, j) closer than ``cut`` in the periodic box."""
    n, dim = x.shape
    nc = torch.floor(box / cut).long()
    found = []
    if int(nc.min()) < 3 or n < 2000:
        for a in range(0, n, 2048):
            d = x[a:a + 2048, None] - x[None]
            d -= box * torch.round(d / box)
            i, j = torch.nonzero((d * d).sum(-1) < cut * cut, as_tuple=True)
            keep = i + a != j
            found.append((i[keep] + a, j[keep]))
    else:
        stride = torch.ones(dim, dtype=torch.long, device=x.device)
        for k in range(dim - 2, -1, -1):
            stride[k] = stride[k + 1] * nc[k + 1]
        c = torch.minimum((x / box * nc).long(), nc - 1)
        key = (c * stride).sum(1)
        order = torch.argsort(key)
        cells = int(torch.prod(nc))
        count = torch.bincount(key, minlength=cells)
        start = torch.cumsum(count, 0) - count
        table = torch.full((cells, int(count.max())), -1, dtype=torch.long, device=x.device)
        rank = torch.arange(n, device=x.device) - start[key[order]]
        table[key[order], rank] = order
        for o in range(3**dim):
            off = torch.tensor([(o // 3**k) % 3 - 1 for k in range(dim)], device=x.device)
            other = (((c + off) % nc) * stride).sum(1)
            for a in range(0, n, 1 << 18):
                j = table[other[a:a + (1 << 18)]]
                d = x[a:a + (1 << 18), None] - x[j.clamp(min=0)]
                d -= box * torch.round(d / box)
                i = torch.arange(a, min(n, a + (1 << 18)), device=x.device)[:, None].expand_as(j)
                keep = ((d * d).sum(-1) < cut * cut) & (j >= 0) & (i != j)
                found.append((i[keep], j[keep]))
    return torch.cat([p[0] for p in found]), torch.cat([p[1] for p in found])


class _Terms:
    """u, f = -du/dr and c = d2u/dr2 of a case's pair potential, 0 past the cut."""

    def __init__(self, case, types, network=None):
        self.name, self.cut = case.get("potential", "lj"), _potential(case)[1]
        self.types, self.network = types, network
        if network is not None:
            self.cut, self.du = COSTLY_CUT, _shift()[1]
        self.sigma_max = float(SIGMA.max()) if self.name == "mixture" else 1.0

    def __call__(self, i, j, r):
        sigma = torch.from_numpy(SIGMA).to(r)[self.types[i], self.types[j]] if self.name == "mixture" else 1.0
        s = r / sigma
        inside = (s <= self.cut).to(r)
        if self.name == "harmonic":
            return (1 - s) ** 2 * inside, 2 * (1 - s) * inside, 2 * inside
        t = s**-2
        t6 = t * t * t
        shift = 4 * (self.cut**-12 - self.cut**-6)
        u, f = 4 * (t6 * t6 - t6) - shift, (48 * t6 * t6 - 24 * t6) / s
        c = (624 * t6 * t6 - 168 * t6) * t
        if self.network is not None:
            nu, nf = self.network(s)
            u, f = u - (s - self.cut) * self.du + nu, f + self.du + nf
        return u * inside, f * inside, c * inside


class _Net:
    """The surrogate's network with exact tanh: u and f of the costly terms."""

    def __init__(self, p, norm, device):
        t = lambda v: torch.from_numpy(np.asarray(v, dtype=np.float64)).to(device)  # noqa: E731
        self.norm = [float(v) for v in norm]
        self.w1, self.b1, self.w2 = t(p[0:64]), t(p[64:128]), t(_bf16(p[128:4224]).reshape(64, 64))
        self.b2, self.w3, self.b3 = t(p[4224:4288]), t(p[4288:4416].reshape(2, 64)), t(p[4416:4418])

    def __call__(self, r):
        u, f = torch.empty_like(r), torch.empty_like(r)
        for a in range(0, r.numel(), 1 << 20):
            q = r[a:a + (1 << 20)]
            x = (q * q - self.norm[0]) * self.norm[1]
            h = torch.tanh(torch.tanh(x[:, None] * self.w1 + self.b1) @ self.w2.T + self.b2)
            y = h @ self.w3.T + self.b3
            u[a:a + (1 << 20)] = y[:, 0] * self.norm[2]
            f[a:a + (1 << 20)] = y[:, 1] * self.norm[3] / q
        return u, f


def _sums(x, box, pairs, terms, all_of=False):
    """Forces, and with ``all_of`` also Laplacian, energy and virial."""
    i, j = pairs
    d = x[i] - x[j]
    d -= box * torch.round(d / box)
    r = torch.sqrt((d * d).sum(1))
    u, f, c = terms(i, j, r)
    force = torch.zeros_like(x).index_add_(0, i, d * (f / r)[:, None])
    if not all_of:
        return force
    dim = x.shape[1]
    lap = torch.zeros(x.shape[0], dtype=x.dtype, device=x.device).index_add_(0, i, c - (dim - 1) * f / r)
    return force, lap, float(u.sum()) / 2, float((f * r).sum()) / (2 * dim)


def _philox(c, key):
    """Philox4x32-10 of Salmon, Moraes, Dror and Shaw (2011) on int64 tensors."""
    mask = 0xFFFFFFFF
    k0, k1 = key & mask, (key >> 32) & mask
    for _ in range(10):
        p, q = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((q >> 32) & mask) ^ c[1] ^ k0, q & mask, ((p >> 32) & mask) ^ c[3] ^ k1, p & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _normals(seed, step, n, dim, device):
    """The deviates of particles 0..n-1 in a step (Box-Muller, uniform numbers
    as the framework rounds them, the rest in 64 bits)."""
    i = torch.arange(n, device=device)
    z = torch.zeros_like(i)
    r = _philox([i, z + (step & 0xFFFFFFFF), z + (step >> 32), z + 0x64706D64], seed)
    out = []
    for a, b in ((r[0], r[1]), (r[2], r[3])):
        u = ((a.float() + 1.0) * 2.0**-32).clamp(max=1.0).double()
        v = (b.float() * 2.0**-32).double()
        rad = torch.sqrt(-2 * torch.log(u))
        out += [rad * torch.cos(2 * math.pi * v), rad * torch.sin(2 * math.pi * v)]
    return torch.stack(out[:dim], dim=1)


def _advance(x, v, box, mass, steps, terms, skin, dt, temperature, seed, nve, sample=None, first=0):
    """The trajectory: forces, G-JF or NVE update, wrap. ``seed``: the noise's;
    ``first``: the first particle's number in the noise stream's order."""
    images = torch.zeros_like(x)
    beta = torch.zeros_like(x)
    m = mass[:, None]
    alpha = m / 0.1
    a = (1 - alpha * dt / 2 / m) / (1 + alpha * dt / 2 / m)
    b = 1 / (1 + alpha * dt / 2 / m)
    width = torch.sqrt(2 * alpha * temperature * dt)
    ref, pairs = None, None
    for t in range(steps):
        if ref is not None:
            d = x - ref
            d -= box * torch.round(d / box)
        if ref is None or float((d * d).sum(1).max()) > (skin / 2) ** 2:
            ref, pairs = x.clone(), _pairs(x, box, terms.cut * terms.sigma_max + skin)
        if sample and (t + 1) % sample[0] == 0:
            f, _, u, w = _sums(x, box, pairs, terms, all_of=True)
        else:
            f = _sums(x, box, pairs, terms)
        if nve:
            v = v + f * dt / m
        else:
            new = width * _normals(seed, t, first + x.shape[0], x.shape[1], x.device)[first:]
            v = a * v + b * dt / m * f + b / (2 * m) * (beta + new)
            beta = new
        x = x + v * dt
        if sample and (t + 1) % sample[0] == 0:
            sample[1].append((u, w, float((m * v * v).sum())))
        shift = torch.floor(x / box)
        images = images + shift
        x = x - shift * box
    return x, v, images


def _noise_seed(seed):
    np.random.seed(seed)
    return int(np.random.randint(0, 2**62, dtype=np.int64))  # the first number a Simulation draws


def exact(case, seed):
    kind = case["kind"]
    dev = _dev()
    t = lambda v: torch.from_numpy(np.asarray(v)).to(dev)  # noqa: E731
    if kind == "train":
        return _exact_training(case, seed, dev)
    if kind == "replicas":
        return _exact_replicas(case, seed, dev)
    pos, vel, box, types, masses = _system(case, seed)
    n, dim = pos.shape
    x, v, box_t, mass = t(pos), t(vel), t(box), t(masses)
    if kind == "rdf":
        bins = np.linspace(0.5, float(np.min(box)) / 2, case["bins"] + 1)
        return _exact_rdf(case, x, box_t, types, bins)
    if kind == "surrogate":
        _, norm = _samples(seed, 4096)
        terms = _Terms(case, t(types).long(), _Net(_network(seed, norm, True), norm, dev))
        x, v, _ = _advance(x, v, box_t, mass, case["steps"], terms, 0.3, 0.004, 1.0, _noise_seed(seed), False)
        f, _, u, _ = _sums(x, box_t, _pairs(x, box_t, COSTLY_CUT), terms, all_of=True)
        return [x.float(), v.float(), f.float(), np.float32(u)]
    terms = _Terms(case, t(types).long())
    if kind == "run":
        if n * case["steps"] > (1.5e8 if case["potential"] == "harmonic" else 2.5e7):
            return None  # more than the time there is
        x, v, images = _advance(x, v, box_t, mass, case["steps"], terms, case["skin"], case["dt"],
                                case["temperature"], _noise_seed(seed), case["integrator"] == "nve")
        return [x, v, None]
    out = []
    for frame in _frames(case, seed):
        x = t(frame)
        f, lap, u, w = _sums(x, box_t, _pairs(x, box_t, terms.cut * terms.sigma_max), terms, all_of=True)
        volume = float(np.prod(box))
        kinetic = float((mass[:, None] * v * v).sum())
        out.append([f, lap, np.array([u, w, w / volume + kinetic / dim / volume])])
    return out


def _exact_rdf(case, x, box, types, bins):
    edges = torch.from_numpy(bins).to(x.device)
    r = bins[:-1] + np.diff(bins) / 2
    shell = 4 * np.pi * r**2 * np.diff(bins)
    groups = [(np.arange(len(types)),) * 2] if not case["types"] else [
        tuple(np.nonzero(types == g)[0] for g in pair) for pair in ((0, 0), (0, 1))]
    out = [] if case["types"] else [r]
    for a, b in groups:
        xa, xb = x[torch.from_numpy(a).to(x.device)], x[torch.from_numpy(b).to(x.device)]
        counts = torch.zeros(len(bins) - 1, dtype=torch.long, device=x.device)
        for k in range(0, len(a), 512):
            d = xa[k:k + 512, None] - xb[None]
            d -= box * torch.round(d / box)
            q = torch.sqrt((d * d).sum(-1)).reshape(-1)
            q = q[(q >= edges[0]) & (q <= edges[-1])]
            at = torch.bucketize(q, edges, right=True) - 1
            counts += torch.bincount(at.clamp(max=len(bins) - 2), minlength=len(bins) - 1)
        out.append(counts.double().cpu().numpy() / shell / (len(a) * len(b)) * float(torch.prod(box)))
    return out


def _exact_replicas(case, seed, dev):
    if _replica_particles(case) * case["steps"] > 2e6 or case["replicas"] * case["steps"] > 20000:
        return None  # more than the time there is
    specs = _replica_specs(case, seed)
    xs, vs, rows, first = [], [], [], 0
    terms = _Terms({}, None)
    for s in specs:
        t = lambda v: torch.from_numpy(np.asarray(v, dtype=np.float64)).to(dev)  # noqa: E731
        n = s.positions.shape[0]
        taken = []
        x, v, _ = _advance(t(s.positions), t(s.velocities), t(s.box), t(np.ones(n)), case["steps"], terms, 0.45,
                           0.005, s.temperature, seed, False,
                           (case["sample_every"], taken) if case["sample_every"] else None, first)
        xs.append(x)
        vs.append(v)
        first += n
        if taken:
            u, w, k = np.mean(np.array(taken), axis=0)
            volume = float(np.prod(s.box))
            rows.append((u / n, k / (3 * n), w / volume + k / 3 / volume))
    out = [torch.cat(xs), torch.cat(vs), None]
    return out + [np.array(c) for c in zip(*rows)] if rows else out


def _exact_training(case, seed, dev):
    """Adam on the framework's minibatches, the second layer's weights rounded
    to bf16 in the forward and backward products, everything else in 64 bits."""
    r, norm = _samples(seed, case["samples"])
    u, f = _costly_terms(r)
    t = lambda v: torch.from_numpy(np.asarray(v, dtype=np.float64)).to(dev)  # noqa: E731
    s = t((r * r).astype(np.float32))
    y = t(np.stack([u / norm[2], f * r / norm[3]], axis=1).astype(np.float32))
    p = t(_network(seed, norm, False))
    mo, ve = torch.zeros_like(p), torch.zeros_like(p)
    losses = []
    for k in range(case["steps"]):
        frac = k / (case["steps"] - 1) if case["steps"] > 1 else 1.0
        lr = 1e-6 + 0.5 * (2e-3 - 1e-6) * (1 + math.cos(math.pi * frac))
        b = torch.arange(case["batch"], device=dev)
        z = torch.zeros_like(b)
        w = _philox([b, z + k, z, z + 0x6D6C7031], seed)
        i = w[1] % case["samples"]  # a power of two: the upper word does not count
        q = p.clone()
        q[128:4224] = q[128:4224].float().bfloat16().double()
        q.requires_grad_(True)
        x = ((s[i] - float(norm[0])) * float(norm[1]))[:, None]
        h = torch.tanh(torch.tanh(x * q[0:64] + q[64:128]) @ q[128:4224].reshape(64, 64).T + q[4224:4288])
        e = (h @ q[4288:4416].reshape(2, 64).T + q[4416:4418] - y[i]) ** 2
        loss = e.sum()
        (g,) = torch.autograd.grad(loss / case["batch"], q)
        losses.append(float(loss))
        mo, ve = 0.9 * mo + 0.1 * g, 0.999 * ve + 0.001 * g * g
        p = p - lr * (mo / (1 - 0.9 ** (k + 1))) / (torch.sqrt(ve / (1 - 0.999 ** (k + 1))) + 1e-8)
    return [np.array(losses), p.cpu().numpy()]
