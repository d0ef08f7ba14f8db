"""Energy, force and stress evaluations that users of this package run, as measurable cases.

Every case is one call of a public entry point (``B200PredictUnit.predict`` on device-resident inputs or
``B200Calculator.calculate`` on host atoms), on the systems of fairchem_b200/synthetic.py and the two model shapes of
fairchem_b200/weights.py, from a single molecule to the 100 000-atom water box.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from fairchem_b200 import synthetic, weights
from fairchem_b200.backbone import build_model
from fairchem_b200.calculator import B200Calculator
from fairchem_b200.predict import B200PredictUnit

MODELS = {"uma_s": weights.UMA_S, "escn_md_l4": weights.ESCN_MD_L4}
DEVICE = "cuda"


def _molecules(n_systems, nmin, nmax, **kw):
    return dict(system="molecules", systems=n_systems, nmin=nmin, nmax=nmax, model="uma_s", **kw)


def _crystal(system, nx, ny, nz, **kw):
    return dict(system=system, nx=nx, ny=ny, nz=nz, **kw)


def _water(atoms, **kw):
    return dict(system="water", atoms=atoms, model="uma_s", **kw)


def listed():
    return [
        # one small organic molecule behind an ASE-style calculator: an optimiser's step, latency only
        dict(_molecules(1, 21, 21, driver="calculator", wants="forces"), name="calculator_molecule_21"),
        # a batch of molecules of mixed sizes: dataset relabelling, batched relaxations
        dict(_molecules(64, 20, 60, driver="predict", wants="forces"), name="molecules_64"),
        # energies of a larger batch, nothing differentiated: screening, ranking of conformers
        dict(_molecules(257, 20, 60, driver="predict", wants="energy"), name="molecules_257_energy"),
        # bulk supercell of ordinary size, the usual single-point or MD step
        dict(_crystal("fcc_cu", 4, 4, 4, model="uma_s", driver="predict", wants="forces"), name="fcc_cu_256"),
        # cell relaxation of an alloy: energy, forces and stress from host atoms every step
        dict(_crystal("bcc_alloy", 7, 7, 7, model="uma_s", driver="calculator", wants="stress"), name="calculator_alloy_686_stress"),
        # random alloy of a few thousand atoms
        dict(_crystal("bcc_alloy", 10, 10, 10, model="uma_s", driver="predict", wants="forces"), name="bcc_alloy_2000"),
        # molecular dynamics of a liquid with positions on the device and a kept neighbour list
        dict(_water(1501, driver="md", wants="forces"), name="md_water_1501"),
        # mid-size liquids, atom counts that divide nothing
        dict(_water(5003, driver="predict", wants="forces"), name="water_5003"),
        dict(_water(24999, driver="predict", wants="forces"), name="water_24999"),
        # the largest system one GPU is asked for
        dict(_water(100_000, driver="predict", wants="forces"), name="water_100k"),
        # the larger model (10 layers, lmax 4) on a small and on a large supercell
        dict(_crystal("fcc_cu", 3, 3, 3, model="escn_md_l4", driver="predict", wants="forces"), name="l4_fcc_cu_108"),
        dict(_crystal("fcc_cu", 10, 20, 25, model="escn_md_l4", driver="predict", wants="forces"), name="l4_fcc_cu_20000"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["molecules", "molecules", "fcc_cu", "bcc_alloy", "water", "water", "l4"])
    wants = rng.choice(["forces", "forces", "forces", "stress", "energy"])
    if kind == "molecules":
        # batches from one molecule to a few hundred; sizes of the generator's own range
        n = _log_int(rng, 1, 300)
        nmin = rng.randint(8, 40)
        driver = "calculator" if n == 1 else "predict"
        return _molecules(n, nmin, rng.randint(nmin, 60), driver=driver, wants="forces" if wants == "stress" else wants)
    if kind == "water":
        driver = rng.choice(["predict", "predict", "md", "calculator"])
        if driver == "md" or (driver == "calculator" and wants == "energy"):
            wants = "forces"
        return _water(_log_int(rng, 300, 100_000), driver=driver, wants=wants)
    if kind == "l4":
        a = _log_int(rng, 2, 12)
        return _crystal("fcc_cu", a, rng.randint(2, a), rng.randint(2, min(2 * a, 20)), model="escn_md_l4", driver="predict", wants=wants)
    a = _log_int(rng, 2, 20)
    return _crystal(kind, a, rng.randint(2, a), rng.randint(2, 20), model="uma_s",
                    driver="predict" if wants == "energy" else rng.choice(["predict", "calculator"]), wants=wants)


def _system(case, seed):
    s = case["system"]
    if s == "molecules":
        # the sizes of the batch belong to the case, elements and positions to the seed
        span = case["nmax"] - case["nmin"] + 1
        sizes = [case["nmin"] + (17 * i) % span for i in range(case["systems"])]
        return synthetic.merge(synthetic.molecule_batch(1, n, n, seed=1000 * seed + i) for i, n in enumerate(sizes))
    if s == "water":
        return synthetic.water_box(case["atoms"], seed=seed)
    make = synthetic.fcc_cu if s == "fcc_cu" else synthetic.bcc_alloy
    return make((case["nx"], case["ny"], case["nz"]), seed=seed)


@functools.lru_cache(maxsize=2)
def _weights(model):
    return weights.random_init_state_dict(MODELS[model], 0)


def _build_unit(model, wants, skin=0.0):
    bb, head = build_model(MODELS[model], _weights(model), device=DEVICE, regress_forces=wants != "energy",
                           regress_stress=wants == "stress")
    return B200PredictUnit(bb, head, device=DEVICE, skin=skin)


@functools.lru_cache(maxsize=2)
def _unit(model, wants):
    # a program loads its model once and evaluates many systems with it
    return _build_unit(model, wants)


class _Atoms:
    """What a driver holds on the host: the fields of an ASE Atoms object that the calculator reads."""

    def __init__(self, data):
        self.positions = data.pos.numpy().astype(np.float64)
        self.numbers = data.atomic_numbers.numpy()
        self.pbc = data.pbc[0].numpy()
        self.cell = data.cell[0].numpy().astype(np.float64) if self.pbc.any() else np.zeros((3, 3))
        self.info = {"charge": int(data.charge[0]), "spin": int(data.spin[0])}

    def __len__(self):
        return len(self.numbers)


def prepare(case, seed):
    data = _system(case, seed)
    if case["driver"] == "calculator":
        task = data.dataset[0]
        return {"calculator": B200Calculator(_unit(case["model"], case["wants"]), task), "atoms": _Atoms(data)}
    data = data.to(DEVICE)
    if case["driver"] == "md":
        # a trajectory in progress: the neighbour list is some steps old and the atoms have moved since, by less
        # than half the skin
        unit = _build_unit(case["model"], case["wants"], skin=0.5)
        unit.predict(data)
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        step = 0.03 * torch.randn(data.pos.shape, generator=gen, device=DEVICE)
        with torch.no_grad():
            data["pos"] = data["pos"].detach() + step.clamp(-0.12, 0.12)
        return {"unit": unit, "data": data}
    return {"unit": _unit(case["model"], case["wants"]), "data": data}


def run(state):
    if "calculator" in state:
        calc = state["calculator"]
        calc.calculate(state["atoms"])
        return {k: calc.results[k] for k in ("energy", "forces", "stress") if k in calc.results}
    return state["unit"].predict(state["data"])


def _counts(case):
    """(atoms, edges) of a case; neighbours are capped at 30 per atom (31 with ties, in liquids)."""
    s = case["system"]
    if s == "molecules":
        per = 0.5 * (case["nmin"] + case["nmax"])
        n = case["systems"] * per
        return n, n * min(30.0, 0.75 * (per - 1))
    if s == "water":
        return case["atoms"], 31.0 * case["atoms"]
    n = case["nx"] * case["ny"] * case["nz"] * (4 if s == "fcc_cu" else 2)
    return n, 30.0 * n


def work(case):
    cfg = MODELS[case["model"]]
    c, h, r, lmax, nb = (cfg[k] for k in ("sphere_channels", "hidden_channels", "edge_channels", "lmax", "num_distance_basis"))
    atoms, edges = _counts(case)
    rows = [lmax + 1, lmax, lmax - 1]  # rows per |m|
    radial = nb * r + r * r
    conv1 = rows[0] * 2 * c * (rows[0] * h + lmax * h) + sum(4 * n * 2 * c * n * h for n in rows[1:])
    conv2 = rows[0] * h * rows[0] * c + sum(4 * n * h * n * c for n in rows[1:])
    wig = sum((2 * min(l, 2) + 1) * (2 * l + 1) for l in range(lmax + 1))
    nl = (lmax + 1) ** 2
    layer_edge = radial + r * 3 * lmax * 2 * c + conv1 + conv2 + wig * 3 * c
    layer_node = nl * c * h * 2 + c * lmax * h
    macs = edges * (cfg["num_layers"] * layer_edge + radial + r * rows[0] * c) + atoms * (cfg["num_layers"] * layer_node + c * h + h * h)
    passes = 1 if case["wants"] == "energy" else 2
    stored = rows[0] * 2 * c * (rows[0] * h + lmax * h) + rows[0] * h * rows[0] * c + sum(2 * n * n * 3 * c * h for n in rows[1:])
    weight = cfg["num_layers"] * (stored + radial + r * 3 * lmax * 2 * c + (lmax + 1) * 2 * c * h)
    return {"bytes": 4.0 * weight + 24.0 * atoms + (12.0 * atoms if passes == 2 else 8.0), "flops": 2.0 * macs * passes}


def tolerance(case):
    # 32-bit results of 4 (10) layers of 32-bit sums forwards and backwards
    return {"rel": 1e-5 if case["model"] == "uma_s" else 3e-5}
