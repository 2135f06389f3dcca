"""Energy-and-force evaluations that stand for the use of this package, each one call sequence of its public entry points.

A case names a model of the benchmark configurations, a structure, a precision and the way the evaluator is entered:

* ``calculate``: ``Symmetrix.calculate`` with positions in host memory, as an ASE-style driver calls it every step
  (neighbour list, evaluation, reduction and the copies of the results are all part of the pass);
* ``edges_host``: ``MACE.compute_node_energies_forces`` with a host-side neighbour list and ``reduce_forces`` to the host, as a
  LAMMPS run with a CPU neighbour list does;
* ``edges_device``: the same with edge arrays and results on the GPU, as a device-resident driver does;
* ``stages``: ``begin`` and the stage methods one by one, as the message-passing pair style does.

Every pass computes forward and backward (the forces are the reverse pass). Sizes run from one molecule to a box that fills the
GPU with work for some tens of milliseconds; boxes are anisotropic and their atom and edge counts odd where the structure allows.
"""
import json
import math
import os
import random
import tempfile

import numpy as np
import torch

from symmetrix_b200 import structures
from symmetrix_b200.calculator import Symmetrix
from symmetrix_b200.modelgen.gen_tp_code import tables
from symmetrix_b200.modelgen.generate import expand_contraction_weights, generate_model, named_spec, to_jsonable

# Models: the benchmark configurations, exported for the elements that the structures hold (as the benchmark does).
_MODELS = {
    "water64": ("water64", {}),                                                          # 64x0e, r_cut 5
    "organic128": ("organic128", {"atomic_numbers": [1, 6, 8]}),                         # 128x0e + 128x1o, r_cut 5
    "organic128_zd": ("organic128", {"atomic_numbers": [1, 8], "zbl": True, "density": True}),   # + ZBL, density normalisation
    "fcc128": ("fcc128", {}),                                                            # five metals, r_cut 6
    "deep256": ("deep256", {"atomic_numbers": [1, 6, 8]}),                               # 256x0e + 256x1o + 256x2e, three blocks
}


def listed():
    return [
        # one isolated molecule: a geometry optimisation or a scan, where latency is all
        {"name": "molecule_f64", "model": "organic128", "structure": "molecule", "n": 1, "dtype": "float64", "entry": "calculate"},
        # a conventional cell of a random alloy with its periodic images: phonons, equations of state
        {"name": "unit_cell_f64", "model": "fcc128", "structure": "fcc", "n": 1, "ny": 1, "nz": 1, "dtype": "float64", "entry": "calculate"},
        # configuration 0: 64 water molecules, the small model
        {"name": "water192_f64", "model": "water64", "structure": "water", "n": 4, "dtype": "float64", "entry": "calculate"},
        # a small MD box in single precision, through the calculator
        {"name": "fcc420_f32", "model": "fcc128", "structure": "fcc", "n": 5, "ny": 3, "nz": 7, "dtype": "float32", "entry": "calculate"},
        # pair-style stages with ZBL and density normalisation
        {"name": "water1029_zd_f64", "model": "organic128_zd", "structure": "water", "n": 7, "dtype": "float64", "entry": "stages"},
        # three interaction blocks, L_max = 2: double precision on a small liquid, single on a larger one
        {"name": "liquid207_deep_f64", "model": "deep256", "structure": "liquid", "n": 23, "dtype": "float64", "entry": "calculate"},
        {"name": "liquid2664_deep_f32", "model": "deep256", "structure": "liquid", "n": 296, "dtype": "float32", "entry": "edges_device"},
        # configuration 1: the 4,000-atom box in both precisions, device-resident and from a host neighbour list
        {"name": "fcc4000_f64", "model": "fcc128", "structure": "fcc", "n": 10, "ny": 10, "nz": 10, "dtype": "float64", "entry": "edges_device"},
        {"name": "fcc4000_f32", "model": "fcc128", "structure": "fcc", "n": 10, "ny": 10, "nz": 10, "dtype": "float32", "entry": "edges_host"},
        # configuration 2's construction at a quarter of its size, through the calculator
        {"name": "water24000_f32", "model": "organic128", "structure": "water", "n": 20, "dtype": "float32", "entry": "calculate"},
        # large boxes of configuration 3's construction
        {"name": "fcc30360_f64", "model": "fcc128", "structure": "fcc", "n": 15, "ny": 22, "nz": 23, "dtype": "float64", "entry": "edges_device"},
        {"name": "fcc87696_f32", "model": "fcc128", "structure": "fcc", "n": 29, "ny": 27, "nz": 28, "dtype": "float32", "entry": "edges_device"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    dtype = rng.choice(["float32", "float64"])
    entry = rng.choice(["calculate", "calculate", "edges_host", "edges_device", "stages"])
    model = rng.choice(["water64", "organic128", "organic128", "organic128_zd", "fcc128", "fcc128", "deep256"])
    case = {"model": model, "dtype": dtype, "entry": entry}
    if model == "fcc128":
        cells = math.exp(rng.uniform(math.log(2.0), math.log(20000 if dtype == "float32" else 7500)))
        side = cells ** (1.0 / 3.0)
        nx = max(1, round(side * rng.uniform(0.7, 1.4)))
        ny = max(1, round(side * rng.uniform(0.7, 1.4)))
        nz = max(2 if nx * ny == 1 else 1, round(cells / (nx * ny)))
        case.update(structure="fcc", n=nx, ny=ny, nz=nz)
        if rng.random() < 0.3:
            case["slab"] = True             # a surface: open along z
    elif model == "organic128" and rng.random() < 0.2:
        case.update(structure="molecule", n=_log_int(rng, 2, 16))
    elif model in ("organic128", "deep256") and (model == "deep256" or rng.random() < 0.5):
        top = {("organic128", "float32"): 5000, ("organic128", "float64"): 2500, ("deep256", "float32"): 400, ("deep256", "float64"): 150}
        case.update(structure="liquid", n=_log_int(rng, 2, top[(model, dtype)]))
    else:
        case.update(structure="water", n=_log_int(rng, 3, 22 if dtype == "float32" else 15))
    return case


# ------------------------------------------------------------------------------------------- inputs

def _spec(model):
    base, over = _MODELS[model]
    return named_spec(base, **over)


def _model_file(model):
    """The model file, written once per machine: the weights are seeded, so every process writes the same."""
    path = os.path.join(tempfile.gettempdir(), "smx_cases_%s_%d.json" % (model, os.getuid()))
    if not os.path.exists(path):
        text = json.dumps(to_jsonable(expand_contraction_weights(generate_model(_spec(model)))))
        part = "%s.%d" % (path, os.getpid())
        with open(part, "w") as f:
            f.write(text)
        os.replace(part, path)
    return path


_calculator = {}


def _calculator_for(model, dtype):
    """One calculator per model and precision, as a program keeps it over its structures; only the last one is held here."""
    key = (model, dtype)
    if key not in _calculator:
        _calculator.clear()
        _calculator[key] = Symmetrix(_model_file(model), dtype=dtype)
    return _calculator[key]


_liquid_cells = {}


def _liquid(n, rng):
    """A liquid of n molecules, rounded to copies of a cell of at most 40 (whose contacts are resolved), with thermal displacements."""
    copies = max(1, round((n / 30.0) ** (1.0 / 3.0)))
    reps = (copies, copies, max(1, round(n / (30.0 * copies * copies)))) if n > 40 else (1, 1, 1)
    count = max(1, round(n / (reps[0] * reps[1] * reps[2])))
    if count not in _liquid_cells:
        _liquid_cells[count] = structures.molecular_liquid(count, seed=count)
    s = structures.replicate(_liquid_cells[count], reps)
    s.positions = s.positions + rng.normal(0.0, 0.05, size=s.positions.shape)
    return s


def _structure(case, seed):
    spec = _spec(case["model"])
    rng = np.random.default_rng(seed)
    kind, n = case["structure"], case["n"]
    if kind == "fcc":
        s = structures.fcc_box((n, case["ny"], case["nz"]), 3.6, sorted(spec.atomic_numbers), seed=seed)
        if case.get("slab"):
            s.pbc = (True, True, False)
            s.cell[2, 2] += 12.0
    elif kind == "water":
        s = structures.water_box_density(n, 1.0, seed=seed)
    elif kind == "liquid":
        s = _liquid(n, rng)
    else:                                   # isolated molecules in a row, open boundaries
        one = structures.molecular_liquid(1, density_g_cm3=0.05, seed=1)
        d = one.positions - one.positions[0]
        d -= np.round(d / one.cell[0, 0]) * one.cell[0, 0]      # made whole
        pos = np.tile(d, (n, 1)) + np.repeat(np.arange(n), 9)[:, None] * np.array([6.0, 0.0, 0.0])
        s = structures.Structure(pos + rng.normal(0.0, 0.05, size=pos.shape), np.diag([6.0 * n, 12.0, 12.0]),
                                 np.tile(one.numbers, n), (False, False, False))
    return s


_KEYS = ["node_types", "num_neigh", "neigh_indices", "neigh_types", "xyz", "r"]


def prepare(case, seed):
    s = _structure(case, seed)
    calc = _calculator_for(case["model"], case["dtype"])
    state = {"case": case, "calc": calc, "structure": s}
    if case["entry"] == "calculate":
        return state
    ev = calc.evaluator
    zmap = {z: t for t, z in enumerate(ev.atomic_numbers)}
    types = np.array([zmap[int(z)] for z in s.numbers], dtype=np.int32)
    ev.build_neighbors(s.positions, types, s.cell, s.pbc)
    edges = dict(ev.get_edges(), node_types=types)
    edges["xyz"] = edges["xyz"].reshape(-1)
    if case["entry"] == "edges_device":
        state["edges"] = [torch.as_tensor(edges[k]).cuda() for k in _KEYS]
    else:
        state["edges"] = [np.ascontiguousarray(edges[k]) for k in _KEYS]
    return state


# ------------------------------------------------------------------------------------------- one pass

_FORWARD = ["A0", "A0_scaled", "M0", "H1", "Phi1", "A1", "A1_scaled", "M1", "H2", "readouts"]
_FORWARD_DEEP = ["A0", "M0", "H1", "Phim", "Am", "Mm", "Hm", "Phi1", "A1", "M1", "H2", "readouts"]


def _stages(ev, n, edges, case):
    """The sequence of the message-passing pair style on one rank."""
    ev.begin(n, *edges)
    ev.compute_ZBL()
    deep = ev.num_interactions == 3
    for name in (_FORWARD_DEEP if deep else _FORWARD):
        if name.endswith("_scaled") and not _MODELS[case["model"]][1].get("density"):
            continue
        getattr(ev, "compute_" + name)()
    ev.reverse_H2(zero_H1_adj=False)
    ev.reverse_M1()
    if _MODELS[case["model"]][1].get("density"):
        ev.reverse_A1_scaled(zero_dxyz=False)
    ev.reverse_A1()
    ev.reverse_Phi1(zero_dxyz=False, zero_H1_adj=False)
    if deep:
        ev.reverse_Hm()
        ev.reverse_Mm()
        ev.reverse_Am()
        ev.reverse_Phim(zero_dxyz=False, zero_H1_adj=False)
    ev.reverse_H1()
    ev.reverse_M0()
    if _MODELS[case["model"]][1].get("density"):
        ev.reverse_A0_scaled()
    ev.reverse_A0()


def run(state):
    case, calc, s = state["case"], state["calc"], state["structure"]
    if case["entry"] == "calculate":
        return calc.calculate(s.positions, s.cell, s.numbers, s.pbc)
    ev, n = calc.evaluator, s.num_atoms
    if case["entry"] == "stages":
        _stages(ev, n, state["edges"], case)
    else:
        ev.compute_node_energies_forces(n, *state["edges"])
    forces, virial, energy = ev.reduce_forces(device=case["entry"] == "edges_device")
    energies = ev.device_view("node_energies") if case["entry"] == "edges_device" else ev.node_energies
    return {"forces": forces, "virial": virial, "energy": energy, "energies": energies}


# ------------------------------------------------------------------------------------------- what a pass cannot do without

def _atoms_and_edges(case):
    """Atoms and expected neighbour pairs (density times the cutoff sphere) of a case."""
    spec, n = _spec(case["model"]), case["n"]
    sphere = 4.0 / 3.0 * math.pi * spec.r_cut ** 3
    if case["structure"] == "fcc":
        atoms, density = 4 * n * case["ny"] * case["nz"], 4 / 3.6 ** 3
    elif case["structure"] == "water":
        atoms, density = 3 * n ** 3, 3 * 0.602214076 / 18.01528
    elif case["structure"] == "liquid":
        atoms, density = 9 * n, 9 * 0.79 * 0.602214076 / 46.068
    else:
        return 9 * n, 9 * n * (8 if n == 1 else 11)
    return atoms, atoms * density * sphere


def work(case):
    spec = _spec(case["model"])
    atoms, edges = _atoms_and_edges(case)
    s = 8 if case["dtype"] == "float64" else 4
    K, L, E = spec.num_channels, spec.L_max, len(spec.atomic_numbers)
    paths, nz, _ = tables(L)
    P, Q, nLM = len(paths), sum(2 * p[0] + 1 for p in paths), (L + 1) ** 2
    T1, T2, nnz = sum(2 * p[1] + 1 for p in paths), sum(2 * p[2] + 1 for p in paths), len(nz)
    middle = spec.num_interactions - 2
    # in: positions (or edge arrays) and the model, of whose radial tables no more than one row per edge; out: energies and forces
    tables_per_row = (4 + P * (1 + middle)) * K * 4 * s
    rows = min(edges, E * (E + 1) / 2 * (spec.num_spline_points - 1))
    weights = (E * 4 + Q / 4.0 * (1 + middle) + 2 * nLM + E + 2) * K * K * s
    inputs = atoms * 32 if case["entry"] == "calculate" else edges * 40 + atoms * 8
    outputs = atoms * 32 + 56
    # multiply-adds count two: tensor products and layer 0 per edge and channel (both directions), channel mixes per atom
    tp = (len({(a, b) for (_, _, a, b, _) in nz}) + 2 * nnz + 2 * Q + 6 * P) + (5 * nnz + 2 * T1 + 4 * T2 + 13 * P)
    layer0 = 2 * 16 + 9 * 4 + 8 * 16 + 14 * 4
    mix = 2 * 2 * K * (nLM * (1 + 2 * middle) + Q * (1 + middle) + 2)
    return {"bytes": rows * tables_per_row + weights + inputs + outputs,
            "flops": edges * K * (tp * (1 + middle) + layer0) + atoms * K * mix}


def tolerance(case):
    # float64 sums in another order; float32 arithmetic (with 3xTF32 products) through the layers of a network and its adjoint
    return {"rel": 1e-11} if case["dtype"] == "float64" else {"rel": 1e-5}
