"""Cases of the evaluation path: structures in, energies / forces / stresses / magnetic moments out.

Every case goes through a public entry point (``MatRIS.predict``, ``MatRIS.forward`` on a graph in hand,
``GraphConverter.batch``, ``MatRISCalculator``, ``StructOptimizer``, ``MolecularDynamics``).  Structures are synthetic:
perturbed FCC Cu and BCC Fe supercells, random triclinic crystals of 8-64 atoms at 2-8 g/cm^3, 40-atom ABX3 cells and
amorphous Li6PS5Cl, i.e. the systems of ``matris_b200.workloads``; weights are seeded random ones of the 10-layer model
unless a case says otherwise.  What a user keeps between calls (the model, the calculator, the list of structures on the
host, the graph where the call takes one) is made in ``prepare``.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from matris_b200 import MatRIS, MatRISCalculator, MolecularDynamics, StructOptimizer, workloads
from matris_b200.applications import SimpleAtoms
from matris_b200.weights import random_checkpoint
from matris_b200.workloads import ATOMIC_WEIGHT, AMU_PER_A3_TO_G_PER_CM3, Crystal

_DEFAULTS = dict(count=1, lo=0, hi=0, nx=0, ny=0, nz=0, steps=0, layers=10, options="", task="efs")


def _case(name, call, system, **kw):
    return {**_DEFAULTS, "name": name, "call": call, "system": system, **kw}


def listed():
    return [
        # one small cell at a time: scripts and services that evaluate single structures; latency is all there is
        _case("cell-4", "predict", "fcc", nx=1, ny=1, nz=1),
        # a calculator on the host, one call per geometry, results read back (the 32-atom Cu configuration)
        _case("calculator-32", "calculator", "fcc", nx=2, ny=2, nz=2, task="efsm"),
        # relaxation of one ABX3 cell: a few FIRE steps with the decisions on the host
        _case("relax-40", "relax", "perovskite", steps=5),
        # molecular dynamics of a small amorphous cell
        _case("md-256", "md", "glass", lo=256, hi=256, steps=4),
        # a graph in hand, evaluated (the call a loop over prepared batches makes)
        _case("forward-12", "forward", "crystals", count=12, lo=8, hi=64, task="ef"),
        # a ragged batch with the optional terms of the model (biases, smoothed edge update), six layers
        _case("options-40", "predict", "crystals", count=40, lo=8, hi=64, task="efsm", layers=6, options="bias"),
        # energies and moments only: no backward pass
        _case("energies-96", "predict", "crystals", count=96, lo=8, hi=64, task="em"),
        # conversion of a list of structures into graphs, without the model
        _case("graphs-256", "graphs", "crystals", count=256, lo=8, hi=64, task=""),
        # the batched screen of random crystals
        _case("crystals-256", "predict", "crystals", count=256, lo=8, hi=64),
        # the batched screen of ABX3 cells: more than fits in memory at once, so it runs as sub-batches
        _case("perovskites-256", "predict", "perovskite", count=256, task="efsm"),
        # molecular dynamics of the 4096-atom amorphous electrolyte
        _case("md-4096", "md", "glass", lo=4096, hi=4096, steps=1),
        # one large structure (16,000 atoms)
        _case("iron-16000", "predict", "bcc", nx=20, ny=20, nz=20, task="efsm"),
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["cell", "calculator", "relax", "md", "forward", "options", "energies", "graphs", "crystals",
                       "perovskites", "metal"])
    if kind == "cell":
        c = _case("", "predict", "crystals", lo=log_int(3, 64), task=rng.choice(["ef", "efs", "efsm"]))
        c["hi"] = c["lo"]
    elif kind == "calculator":
        c = _case("", "calculator", "fcc", nx=rng.randint(1, 4), ny=rng.randint(1, 4), nz=rng.randint(1, 5),
                  task=rng.choice(["efs", "efsm"]), layers=rng.choice([6, 10]))
    elif kind == "relax":
        c = _case("", "relax", rng.choice(["perovskite", "crystals"]), lo=log_int(6, 90), steps=rng.randint(3, 7))
        c["hi"] = c["lo"]
    elif kind == "md":
        c = _case("", "md", "glass", lo=log_int(50, 4000), steps=rng.randint(1, 4), layers=rng.choice([6, 10]))
        c["hi"] = c["lo"]
    elif kind == "forward":
        c = _case("", "forward", "crystals", count=log_int(2, 120), lo=8, hi=rng.randint(20, 64),
                  task=rng.choice(["ef", "efs", "efsm"]))
    elif kind == "options":
        c = _case("", "predict", "crystals", count=log_int(4, 100), lo=8, hi=64, task=rng.choice(["efs", "efsm"]), layers=6,
                  options=rng.choice(["bias", "gaussian"]))
    elif kind == "energies":
        c = _case("", "predict", "crystals", count=log_int(3, 300), lo=8, hi=64, task=rng.choice(["e", "em"]))
    elif kind == "graphs":
        c = _case("", "graphs", "crystals", count=log_int(3, 600), lo=8, hi=64, task="")
    elif kind == "crystals":
        c = _case("", "predict", "crystals", count=log_int(8, 300), lo=rng.randint(4, 20), hi=rng.randint(30, 64))
    elif kind == "perovskites":
        c = _case("", "predict", "perovskite", count=log_int(4, 256), task=rng.choice(["efs", "efsm"]))
    else:
        c = _case("", "predict", "bcc", nx=rng.randint(3, 16), ny=rng.randint(3, 16), nz=rng.randint(4, 20),
                  task=rng.choice(["ef", "efsm"]))
    del c["name"]
    return c


# ------------------------------------------------------------------ structures
def _scatter(rng, n, lattice, spacing=1.7):
    """``n`` atoms on a random subset of the points of a grid of about ``spacing`` Angstrom, each moved a little."""
    g = np.maximum(1, np.floor(np.linalg.norm(lattice, axis=1) / spacing)).astype(int)
    while g.prod() < n:
        g = g + 1
    site = rng.choice(g.prod(), size=n, replace=False)
    frac = np.stack([site // (g[1] * g[2]), (site // g[2]) % g[1], site % g[2]], axis=1)
    return ((frac + rng.uniform(-0.15, 0.15, (n, 3))) / g) @ lattice


def _triclinic(rng, lo, hi):
    elements = np.array([z for z in range(1, 84) if z not in (2, 10, 18, 36, 54)])
    n = int(rng.integers(lo, hi + 1))
    numbers = rng.choice(elements, size=n)
    al, be, ga = np.deg2rad(rng.uniform(75.0, 105.0, 3))
    cx, cy = np.cos(be), (np.cos(al) - np.cos(be) * np.cos(ga)) / np.sin(ga)
    lat = np.array([[1.0, 0, 0], [np.cos(ga), np.sin(ga), 0], [cx, cy, np.sqrt(1.0 - cx * cx - cy * cy)]])
    lat = lat * rng.uniform(4.0, 12.0, 3)[:, None]
    mass = ATOMIC_WEIGHT[numbers].sum() * AMU_PER_A3_TO_G_PER_CM3
    lat = lat * (mass / rng.uniform(2.0, 8.0) / abs(np.linalg.det(lat))) ** (1.0 / 3.0)
    return Crystal(numbers.astype(np.int64), _scatter(rng, n, lat), lat)


def _connected(c, cutoff=5.5):
    """Whether every atom has a neighbour within ``cutoff`` (an isolated atom is an error of the graph)."""
    shifts = np.array([(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)], float) @ c.lattice
    d = c.cart[:, None, None, :] - c.cart[None, :, None, :] - shifts[None, None, :, :]
    d2 = (d * d).sum(-1)
    d2 = np.where(d2 < 1e-6, np.inf, d2)
    return bool((d2.min(axis=(1, 2)) < cutoff * cutoff).all())


def _glass(rng, n):
    fu = n // 13
    numbers = np.array([3] * (6 * fu + n - 13 * fu) + [15] * fu + [16] * (5 * fu) + [17] * fu, dtype=np.int64)
    rng.shuffle(numbers)
    box = (ATOMIC_WEIGHT[numbers].sum() * AMU_PER_A3_TO_G_PER_CM3 / 1.9) ** (1.0 / 3.0)
    lat = np.eye(3) * box
    return Crystal(numbers, _scatter(rng, n, lat, spacing=1.9), lat)


def _structures(case, seed):
    rng = np.random.default_rng(seed)
    s = case["system"]
    if s == "fcc":
        return [workloads.cu_fcc((case["nx"], case["ny"], case["nz"]), sigma=0.05, seed=seed)]
    if s == "bcc":
        return [workloads.fe_bcc((case["nx"], case["ny"], case["nz"]), seed=seed)]
    if s == "perovskite":
        return workloads.perovskites(case["count"], seed=seed)
    if s == "glass":
        return [_glass(rng, case["lo"])]
    # The geometries belong to the case, so that every seed gives graphs of the same size; the seed moves them rigidly, orders
    # their atoms and deals out the species.
    base = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    out = []
    while len(out) < case["count"]:
        c = _triclinic(base, case["lo"], max(case["lo"], case["hi"]))
        if _connected(c):
            order, turn = rng.permutation(len(c.numbers)), np.linalg.qr(rng.normal(size=(3, 3)))[0]
            turn = turn * np.sign(np.linalg.det(turn))
            out.append(Crystal(rng.permutation(c.numbers), (c.cart[order] + rng.uniform(0.0, 10.0, 3)) @ turn, c.lattice @ turn))
    return out


# ------------------------------------------------------------------ the calls
_OPTIONS = {"": {}, "bias": dict(use_bias=True, use_smoothed_for_delta_edge=True),
            "gaussian": dict(distance_expansion="Gaussian", three_body_expansion="fourier")}
_models = {}


def _model(case):
    """The model a program loads once and keeps (all states of a process share it)."""
    key = (case["layers"], case["options"])
    if key not in _models:
        ck = random_checkpoint(dict(num_layers=case["layers"], reference_energy="mpa", **_OPTIONS[case["options"]]), seed=0,
                               jitter=0.1)
        _models[key] = MatRIS.from_dict(ck).to("cuda")
    return _models[key]


def prepare(case, seed):
    model, structures = _model(case), _structures(case, seed)
    state = dict(call=case["call"], task=case["task"], steps=case["steps"], model=model)
    if case["call"] in ("predict", "graphs"):
        state["structures"] = structures
    elif case["call"] == "forward":
        state["graph"] = model.graph_converter.batch(structures)
    else:
        c = structures[0]
        atoms = state["atoms"] = SimpleAtoms(c.numbers, c.cart, c.lattice)
        if case["call"] == "calculator":
            state["driver"] = MatRISCalculator(model=model, task=case["task"], device=None)
        elif case["call"] == "relax":
            state["driver"] = StructOptimizer(model=model, task=case["task"], optimizer="FIRE", device=None)
        else:
            state["driver"] = MolecularDynamics(atoms, model=model, ensemble="nvt", thermostat="langevin", temperature=600,
                                                starting_temperature=600, timestep=1.0, task=case["task"], device=None,
                                                seed=seed % (1 << 30))
    return state


def run(state):
    call, task = state["call"], state["task"]
    if call == "graphs":
        g = state["model"].graph_converter.batch(state["structures"])
        return {k: getattr(g, k) for k in ("edge_ptr", "center", "neighbor", "image", "dist64", "rev", "d2u", "u2d", "trip_ptr",
                                           "trip_src_ptr", "line_graph", "trip_src_perm", "cart32")}
    if call in ("predict", "forward"):
        if call == "predict":
            out = state["model"].predict(state["structures"], task=task)
        else:
            out = state["model"](state["graph"], task=task)
        # one tensor per quantity, as for a table of results
        join = {"f": torch.cat, "s": torch.stack, "m": torch.cat}
        return {k: join[k](list(out[k])) if k in join else out[k] for k in task}
    atoms, driver = state["atoms"], state["driver"]
    if call == "calculator":
        driver.calculate(atoms)
        return {k: driver.results[k] for k in ("energy", "forces", "stress", "magmoms") if driver.results[k] is not None}
    if call == "relax":
        # a force threshold that is not reached: the run takes all its steps
        log = driver.relax(atoms, fmax=1e-9, steps=state["steps"], verbose=False)["trajectory"]
        return {"energies": np.array(log.energies), "forces": np.stack(log.forces), "stresses": np.stack(log.stresses),
                "positions": np.stack(log.atom_positions)}
    driver.run(state["steps"])
    r = driver.atoms.calc.results
    return {"positions": driver.atoms.positions, "momenta": driver.atoms.momenta, "energy": r["energy"], "forces": r["forces"],
            "stress": r["stress"]}


# ------------------------------------------------------------------ work and tolerance
# per atom: (directed edges within 6 A, triplets = ordered pairs of bonds within 4 A); measured means of the generators
_DENSITY = {"fcc": (78.0, 306.0), "bcc": (64.0, 260.0), "perovskite": (69.0, 322.0), "glass": (50.0, 215.0),
            "crystals": (28.0, 72.0)}


def _sizes(case):
    s = case["system"]
    if s in ("fcc", "bcc"):
        n = (4 if s == "fcc" else 2) * case["nx"] * case["ny"] * case["nz"]
    elif s == "perovskite":
        n = 40 * case["count"]
    else:
        n = case["count"] * (case["lo"] + max(case["lo"], case["hi"])) / 2.0
    e, t = _DENSITY[s]
    return n, n * e, n * t


def work(case):
    n, e, t = _sizes(case)
    graph = 26.0 * e + 20.0 * t + 28.0 * n  # the graph tensors written, positions and numbers read
    if case["call"] == "graphs":
        return {"bytes": graph + 24.0 * e, "flops": 30.0 * e}
    layers = case["layers"]
    # one 128 x 256 contraction of a row: 65,536 operations.  Terms of a node are formed once per node, those of a bond once
    # per bond, and only what differs from row to row per row: triplets 6 of them a layer (two gated MLPs of two layers,
    # attention logits, edge FFN), directed edges 3, bonds and atoms 12 each.
    forward = 65536.0 * layers * (6.0 * t + 3.0 * e + 12.0 * (e / 2.0 + n))
    both = 2.0 if ("f" in case["task"] or "s" in case["task"]) else 1.0
    weights = 4.0 * (1.03e6 * layers + 1e5)
    evaluations = case["steps"] + 1 if case["call"] in ("md", "relax") else 1
    return {"bytes": evaluations * (weights + 28.0 * n + 20.0 * n), "flops": evaluations * both * forward}


def tolerance(case):
    if case["call"] == "graphs":
        return "exact"
    # Features, weights and results are float32; the contractions carry 16 mantissa bits per operand and accumulate in
    # float32.  Forces and stresses are small sums of large terms (the smallest cells most): against exact float32 products
    # this arithmetic is off by up to 1.7e-4 (2-norm) in them, and two orders of the same sums by 3e-5.
    return {"rel": 5e-4, "max": 5e-3}
