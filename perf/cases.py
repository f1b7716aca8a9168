"""The evaluations this framework is used for, as cases that can be timed and compared.

A case is one pass through `Calculator`'s public entry points, host arrays in and host arrays out, as a program calls
them: the model is loaded once and kept (the calculator below), the structures change. Four uses:

  compute   energy, forces and virial of a list of structures, neighbour search included (Calculator.compute)
  energy    energies alone: a screening run, the forward direction without the backward (compute_forces=False)
  md        an engine's own neighbour list, set once and stepped (set_neighbors + compute_step per step)
  relax     a batch staged once, moved and evaluated again and again (stage + update_staged / compute_staged / fetch)

Sizes, models and structures are the benchmark's own (64-, 648- and 1728-atom cells, batches of 64-atom mixtures, the xs,
s and l shapes, both featurizers, every GEMM mode) and what lies around them: molecules, cells with vacancies, ragged
batches. Weights are the seeded random ones of the benchmark definition; the inputs are made from the case's seed.
"""
import math
import os
import tempfile
from collections import OrderedDict

import numpy as np
import torch

from pet_kokkos_b200 import Calculator, EdgeListView
from pet_kokkos_b200 import checkpoint, structures

WEIGHT_SEED = 0
SPECIES = (6, 1, 7, 8, 14)
SKIN = 1.0  # what an engine's list reaches past the cutoff (Angstrom)

_DEFAULTS = {"use": "compute", "model": "s", "featurizer": "feedforward", "gemm": "native", "kind": "diamond", "nx": 1, "ny": 1,
             "nz": 1, "atoms": 0, "vacancies": 0, "structures": 1, "smallest": 0, "steps": 1}


def _case(name, **given):
    return dict(_DEFAULTS, name=name, **given)


def listed():
    return [
        # one molecule in vacuum, the smallest thing anybody evaluates: launches and latency
        _case("molecule21 xs native", model="xs", kind="molecule", atoms=21),
        # the benchmark's 64-atom cell at the small model, in the default precision
        _case("diamond64 xs native", model="xs", nx=2, ny=2, nz=2),
        # liquid water, the default precision at the ordinary size
        _case("water648 s native", kind="water", atoms=648),
        # the 1728-atom cell in the default precision
        _case("diamond1728 s native", nx=6, ny=6, nz=6),
        # the headline: the same cell in the fp32-accurate tensor-core mode
        _case("diamond1728 s 3xtf32", gemm="3xtf32", nx=6, ny=6, nz=6),
        # the two speed modes, on an odd cell of water and on a cell with vacancies
        _case("water1791 s tf32", gemm="tf32", kind="water", atoms=1791),
        _case("diamond1721 s bf16", gemm="bf16", nx=6, ny=6, nz=6, vacancies=7),
        # a batch of independent small structures
        _case("batch256x64 s 3xtf32", gemm="3xtf32", kind="mixture", atoms=64, structures=256),
        # screening: energies alone of molecules of all sizes
        _case("screen300 s tf32 energy", use="energy", gemm="tf32", kind="molecule", atoms=41, smallest=3, structures=300),
        # molecular dynamics driven by an engine's list, ten steps between rebuilds
        _case("md water648 s 3xtf32", use="md", gemm="3xtf32", kind="water", atoms=648, steps=10),
        # a batched relaxation with the residual featurizer, pairs kept between steps
        _case("relax 24x40 xs residual", use="relax", model="xs", featurizer="residual", kind="mixture", atoms=53, smallest=31,
              structures=24, steps=6),
        # the large model: 6 A cutoff, 158 neighbours, head size 64
        _case("diamond1000 l 3xtf32", model="l", gemm="3xtf32", nx=5, ny=5, nz=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_crystal(rng, lo, hi):
    """Cells along x, y, z of a diamond crystal with lo..hi conventional cells in all, and some vacancies."""
    total = _log_int(rng, lo, hi)
    nx = max(1, min(total, int(round(total ** (1 / 3) * math.exp(rng.uniform(-0.2, 0.2))))))
    ny = max(1, int(round((total / nx) ** 0.5)))
    nz = max(1, total // (nx * ny))
    return {"kind": "diamond", "nx": nx, "ny": ny, "nz": nz, "vacancies": rng.randint(0, max(1, nx * ny * nz // 4))}


def draw(rng):
    """One more case of the ranges above."""
    family = rng.choice(["small", "cell", "cell", "batch", "energy", "md", "relax", "large"])
    c = dict(_DEFAULTS)
    fast = rng.choice(["native", "3xtf32", "3xtf32", "tf32", "bf16"])
    if family == "small":  # molecules and unit cells
        c.update(model=rng.choice(["xs", "s"]), gemm=rng.choice(["native", "3xtf32"]))
        if rng.random() < 0.5:
            c.update(kind="molecule", atoms=_log_int(rng, 5, 80))
        else:
            c.update(_draw_crystal(rng, 1, 16))
    elif family == "cell":  # one periodic cell
        c.update(gemm=fast, model=rng.choice(["xs", "s", "s"]), featurizer=rng.choice(["feedforward"] * 3 + ["residual"]))
        if rng.random() < 0.5:
            c.update(kind="water", atoms=3 * _log_int(rng, 70, 600))
        else:
            c.update(_draw_crystal(rng, 16, 216))
    elif family == "batch":
        c.update(gemm=fast, kind="mixture", atoms=_log_int(rng, 33, 70), smallest=rng.randint(20, 33), structures=_log_int(rng, 8, 200))
    elif family == "energy":
        c.update(use="energy", gemm=fast, kind="molecule", atoms=_log_int(rng, 15, 60), smallest=rng.randint(2, 9),
                 structures=_log_int(rng, 16, 400))
    elif family == "md":
        c.update(use="md", gemm=rng.choice(["native", "3xtf32", "3xtf32", "tf32"]), model=rng.choice(["xs", "s"]), kind="water",
                 atoms=3 * _log_int(rng, 70, 300), steps=rng.randint(4, 12))
    elif family == "relax":
        c.update(use="relax", gemm=rng.choice(["native", "3xtf32"]), model="xs", featurizer=rng.choice(["residual", "feedforward"]),
                 kind="mixture", atoms=_log_int(rng, 33, 64), smallest=rng.randint(20, 33), structures=_log_int(rng, 4, 40),
                 steps=rng.randint(3, 8))
    else:
        c.update(model="l", gemm=rng.choice(["3xtf32", "3xtf32", "tf32", "bf16"]), **_draw_crystal(rng, 16, 110))
    return c


# ---- inputs ------------------------------------------------------------------------

def _molecule(n, seed):
    """n atoms of a compact molecule in vacuum: a random walk that keeps every pair more than 0.95 A apart."""
    rng = np.random.default_rng(seed)
    pos = np.zeros((1, 3))
    while len(pos) < n:
        step = rng.normal(size=3)
        c = pos[rng.integers(len(pos))] + step / np.linalg.norm(step) * rng.uniform(1.0, 1.6)
        if ((pos - c) ** 2).sum(1).min() > 0.95 ** 2:
            pos = np.vstack([pos, c])
    return structures.make_system(rng.choice(np.asarray(SPECIES), size=n), pos, np.zeros((3, 3)), (False, False, False))


def _crystal(c, seed):
    """nx x ny x nz conventional cells of diamond, jittered, `vacancies` atoms taken out."""
    a, rng = 3.567, np.random.default_rng(seed)
    dims = np.array([c["nx"], c["ny"], c["nz"]])
    basis = structures.diamond(1, a)["positions"]
    ijk = np.stack(np.meshgrid(*[np.arange(k) for k in dims], indexing="ij"), -1).reshape(-1, 1, 3) * a
    pos = (ijk + basis).reshape(-1, 3)
    pos = pos + rng.normal(0.0, 0.05, size=pos.shape)
    pos = np.delete(pos, rng.permutation(len(pos))[:c["vacancies"]], axis=0)
    return structures.make_system(np.full(len(pos), 6), pos, np.diag(dims * a))


def _structures(c, seed):
    rng = np.random.default_rng(seed + 1)
    if c["kind"] == "diamond":
        return [_crystal(c, seed)]
    if c["kind"] == "water":
        n = c["atoms"] // 3
        return [structures.water_box(n, 18.64 * (n / 216) ** (1 / 3), seed=seed)]
    top = c["atoms"]
    low = c["smallest"] or top
    sizes = rng.permutation(np.linspace(low, top, c["structures"]).round().astype(int))  # the same sizes, in the seed's order
    if c["kind"] == "molecule":
        return [_molecule(int(n), seed * 4099 + b) for b, n in enumerate(sizes)]
    return [structures.random_mixture(int(n), 9.0 * (n / 64) ** (1 / 3), seed=seed * 4099 + b) for b, n in enumerate(sizes)]


def _engine_list(system, reach):
    """Every pair within `reach` of a periodic cell, grouped by centre, with its cell shift: the list an engine keeps."""
    x = torch.tensor(system["positions"], device="cuda")
    cell = torch.tensor(system["cell"], device="cuda")
    widths = [1.0 / float(np.linalg.norm(np.linalg.inv(system["cell"])[:, d])) for d in range(3)]
    r = [range(-int(math.ceil(reach / w)) - 1, int(math.ceil(reach / w)) + 2) for w in widths]
    found = []
    for s in [(i, j, k) for i in r[0] for j in r[1] for k in r[2]]:
        shift = torch.tensor(s, dtype=torch.float64, device="cuda") @ cell
        d2 = ((x[None, :, :] + shift - x[:, None, :]) ** 2).sum(-1)
        i, j = torch.nonzero((d2 < reach * reach) & (d2 > 1e-12), as_tuple=True)
        if len(i):
            found.append(torch.cat([i[:, None], j[:, None], torch.tensor(s, device="cuda").expand(len(i), 3)], 1))
    pairs = torch.cat(found)
    pairs = pairs[torch.sort(pairs[:, 0], stable=True).indices].cpu().numpy()
    offsets = np.concatenate([[0], np.cumsum(np.bincount(pairs[:, 0], minlength=len(x)))])
    return EdgeListView(positions=system["positions"], atomic_numbers=system["atomic_numbers"], offsets=offsets.astype(np.int32),
                        neighbors=pairs[:, 1].astype(np.int32), shifts=pairs[:, 2:].astype(np.int32), cell=system["cell"])


_folder = None
_files = {}
_loaded = OrderedDict()


def _calculator(c):
    """The loaded model a program keeps: one per model and options, the latest two."""
    global _folder
    model = (c["model"], c["featurizer"])
    if model not in _files:
        _folder = _folder or tempfile.TemporaryDirectory(prefix="pet_cases_")
        _files[model] = checkpoint.write_random_checkpoint(os.path.join(_folder.name, "_".join(model)), c["model"], c["featurizer"],
                                                           seed=WEIGHT_SEED)
    key = model + (c["gemm"], c["use"] == "md", c["use"] == "relax")
    if key not in _loaded:
        while len(_loaded) >= 2:
            _loaded.popitem(last=False)
        _loaded[key] = Calculator(*_files[model], gemm=c["gemm"], md_fixed_shapes=c["use"] == "md", cache_neighbors=c["use"] == "relax")
    _loaded.move_to_end(key)
    return _loaded[key]


def prepare(case, seed):
    c = dict(_DEFAULTS, **case)
    calc = _calculator(c)
    systems = _structures(c, seed)
    state = {"use": c["use"], "calc": calc, "systems": systems}
    if c["use"] in ("md", "relax"):  # each step moves every atom a little along its own smooth path
        x = np.concatenate([s["positions"] for s in systems])
        rng = np.random.default_rng(seed + 2)
        a, b = rng.normal(0.0, 0.03, size=(2,) + x.shape)
        state["path"] = [x + a * math.sin(0.4 * k) + b * (1.0 - math.cos(0.4 * k)) for k in range(c["steps"])]
    if c["use"] == "md":
        state["list"] = _engine_list(systems[0], calc.cutoff + SKIN)
    return state


# ---- one pass ----------------------------------------------------------------------

def run(state):
    calc, use = state["calc"], state["use"]
    if use == "compute":
        r = calc.compute(state["systems"])
        return {"energy": r.energy, "per_atom_energy": r.per_atom_energy, "forces": r.forces, "virial": r.virial,
                "struct_id": r.struct_id}
    if use == "energy":
        r = calc.compute(state["systems"], compute_forces=False)
        return {"energy": r.energy, "per_atom_energy": r.per_atom_energy}
    steps = []
    if use == "md":
        calc.set_neighbors(state["list"])
        for x in state["path"]:
            steps.append(calc.compute_step(x, cell=state["list"].cell))
    else:
        calc.stage(state["systems"])
        for x in state["path"]:
            calc.update_staged(x)
            calc.compute_staged(True)
            steps.append(calc.fetch())
    return {what: np.stack([getattr(r, what) for r in steps]) for what in ("energy", "per_atom_energy", "forces", "virial")}


# ---- what a pass cannot do without --------------------------------------------------

def _sizes(c):
    """Atoms, directed edges within the cutoff and the sum over atoms of (tokens squared), as expected from densities."""
    h = checkpoint.make_hypers(c["model"], c["featurizer"])
    ball = 4.0 / 3.0 * math.pi * h["cutoff"] ** 3
    if c["kind"] == "diamond":
        n = 8 * c["nx"] * c["ny"] * c["nz"]
        atoms = n - c["vacancies"]
        per = ball * 8 / 3.567 ** 3 * atoms / n
    elif c["kind"] == "water":
        atoms = 3 * (c["atoms"] // 3)
        per = ball * 648 / 18.64 ** 3
    else:
        each = (c["atoms"] + (c["smallest"] or c["atoms"])) / 2
        atoms = each * c["structures"]
        per = ball * 64 / 9.0 ** 3 if c["kind"] == "mixture" else min(each - 1, ball * 0.1)
    return h, atoms, atoms * per, atoms * (per + 1) ** 2


def work(case):
    """Multiply-adds of the network's weight products and of the attention, forward and (with forces) with respect to the
    activations; bytes: the weights once, the structures in and the results out."""
    c = dict(_DEFAULTS, **case)
    h, n, e, s = _sizes(c)
    D, Dn, Dh, F = h["d_pet"], h["d_node"], h["d_head"], h["d_feedforward"]
    G, A, t = h["num_gnn_layers"], h["num_attention_layers"], n + e
    if h["featurizer_type"] == "feedforward":
        block = t * 4 * D * D + n * (2 * D * Dn + 6 * Dn * Dn) + e * 3 * D * F
        gemm = G * (A * block + e * (D * D + 6 * D * D)) + (G - 1) * e * D * D
        gemm += n * (Dn * Dh + Dh * Dh) + e * (D * Dh + Dh * Dh)
        if c["use"] != "energy":
            gemm *= 2
    else:
        block = t * (4 * D * D + 2 * D * F)
        gemm = G * (A * block + e * D * D + t * (D * Dh + Dh * Dh)) + (G - 1) * e * D * D
        if c["use"] != "energy":
            gemm *= 2
    attention = G * A * s * D * (2 if c["use"] == "energy" else 7)
    weights = sum(math.prod(v) for v in checkpoint.tensor_shapes(h, 85).values())
    per_atom = 28 + 8 if c["use"] == "energy" else 28 + 8 + 24
    return {"bytes": c["steps"] * (4 * weights + n * per_atom), "flops": 2 * c["steps"] * (gemm + attention)}


def tolerance(case):
    """Of forces, virials and energies against another correct implementation in the same mode: the fp32-class modes to fp32
    rounding through some thirty layers, the speed modes to their operands' 11 and 8 significant bits."""
    return {"native": {"rel": 1e-5}, "3xtf32": {"rel": 2e-5}, "tf32": {"rel": 1e-3}, "bf16": {"rel": 3e-3}}[case.get("gemm", "native")]
