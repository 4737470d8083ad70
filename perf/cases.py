"""What this framework is timed on: calls a user's program makes, over the
range of sizes, models and options it makes them with.

`listed()` names the cases, `draw(rng)` gives more of the same ranges,
`prepare(case, seed)` builds what a program holds before the call (the loaded
model, the structures, the buffers), `run(state)` is one pass through the
public entry points, `work(case)` the bytes and operations a pass cannot do
without and `exact(case, seed)` the pass's results in plain 64-bit torch.

Paths:
  evaluate   Batch.evaluateHost: positions in host memory to energies and
             forces in host memory (MD steps, batched prediction)
  values     symmetry functions alone, as nnp-scaling and descriptor
             analyses collect them
  adam       StudentTraining.step: a mini-batch of structures set, evaluated
             with stored derivatives, and one Adam step on energies and forces
  kalman     Training.update: a run of energy and of force updates of the
             Kalman filter
"""
import itertools
import math
import os

import numpy as np
import torch

from n2p2_b200 import Mode, Structure, read_structures, water
from n2p2_b200.student import StudentTraining
from n2p2_b200.training import ENERGY, FORCE, Training

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden")
MODELS = {
    "water40": "models/water40",              # 16 G2 + 24 narrow G3 per element, 25-25 networks
    "water56": "models/water56",              # the same + 16 wide G9, 64-64 networks (the teacher)
    "student": "models/student_water56",      # 8 G2 + 6 narrow G3 with a shorter angular cutoff, 16-16 networks
    "rpbe": "examples/H2O_RPBE-D3",           # 27-30 functions per element, shifted G2, tanh cutoff
    "anisole": "examples/Anisole_SCAN",       # 331-354 compact functions per element
    "qm9": "models/qm9_weighted",             # 45 weighted compact functions, five elements, open boundaries
}
EVALUATE = {"path": "evaluate", "precision": "fp64"}


def _directory(case):
    return os.path.join(GOLDEN, MODELS[case["model"]])


def listed():
    return [
        # one MD step of a small cell: host call, launches and short kernels count
        {"name": "md_64mol_fp64", **EVALUATE, "model": "water40", "boxes": 1, "smallest": 64, "largest": 64},
        # one MD step of a mid-size cell in the mixed form
        {"name": "md_512mol_mixed", **EVALUATE, "precision": "mixed", "model": "water40", "boxes": 1, "smallest": 512,
         "largest": 512},
        # batched prediction: boxes of uneven size, the plain and the mixed form
        {"name": "batch_256_fp64", **EVALUATE, "model": "water40", "boxes": 256, "smallest": 32, "largest": 512},
        {"name": "batch_256_mixed", **EVALUATE, "precision": "mixed", "model": "water40", "boxes": 256, "smallest": 32,
         "largest": 512},
        # a distilled model screening candidate boxes
        {"name": "student_256_fp64", **EVALUATE, "model": "student", "boxes": 256, "smallest": 32, "largest": 512},
        # one MD step of a large cell with the larger model (110,592 atoms)
        {"name": "md_36864mol_fp64", **EVALUATE, "model": "water56", "boxes": 1, "smallest": 36864, "largest": 36864},
        # frames of published potentials: shifted Gaussians with another cutoff function, compact functions,
        # and molecules of a data set (weighted functions, 9-29 atoms each)
        {"name": "rpbe_4_fp64", **EVALUATE, "model": "rpbe", "boxes": 4},
        {"name": "anisole_16_fp64", **EVALUATE, "model": "anisole", "boxes": 16},
        {"name": "qm9_1024_fp64", **EVALUATE, "model": "qm9", "boxes": 1024},
        # symmetry functions of a data set, for its scaling statistics
        {"name": "values_128_fp64", "path": "values", "precision": "fp64", "model": "water40", "boxes": 128,
         "smallest": 32, "largest": 512},
        # training: a mini-batch Adam step, and Kalman filter updates on a resident set
        {"name": "adam_32", "path": "adam", "model": "student", "boxes": 32, "smallest": 32, "largest": 256},
        {"name": "kalman_32_16", "path": "kalman", "model": "water40", "boxes": 32, "smallest": 32, "largest": 128,
         "energy_updates": 32, "force_updates": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "batch", "batch", "batch", "example", "values", "adam", "kalman"])
    water_model = rng.choice(["water40", "water40", "water56", "student"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    smallest = _log_int(rng, 32, 96)
    sizes = {"smallest": smallest, "largest": _log_int(rng, smallest, 512)}
    if kind == "single":
        n = _log_int(rng, 32, 16384)
        return {**EVALUATE, "precision": precision, "model": water_model, "boxes": 1, "smallest": n, "largest": n}
    if kind == "batch":
        return {**EVALUATE, "precision": precision, "model": water_model, "boxes": _log_int(rng, 2, 200), **sizes}
    if kind == "example":
        model, most = rng.choice([("rpbe", 5), ("anisole", 20), ("qm9", 1500)])
        return {**EVALUATE, "model": model, "boxes": _log_int(rng, 1, most)}
    if kind == "values":
        return {"path": "values", "precision": precision, "model": water_model, "boxes": _log_int(rng, 2, 160), **sizes}
    if kind == "adam":
        return {"path": "adam", "model": "student", "boxes": _log_int(rng, 4, 40), "smallest": smallest,
                "largest": _log_int(rng, smallest, 256)}
    return {"path": "kalman", "model": "water40", "boxes": _log_int(rng, 8, 48), "smallest": smallest,
            "largest": _log_int(rng, smallest, 128), "energy_updates": _log_int(rng, 4, 40),
            "force_updates": _log_int(rng, 4, 20)}


def _structures(case, seed):
    """Water boxes of sizes spread over the case's range (thermal
    displacements of 0.05-0.15 bohr), or displaced frames of the model's own
    structure file, in an order of the seed's."""
    rng = np.random.default_rng([seed, 7])
    n = case["boxes"]
    order = rng.permutation(n)
    if "smallest" in case:
        lo, hi = math.log(case["smallest"]), math.log(case["largest"])
        counts = np.rint(np.exp(lo + (order + 0.5) / n * (hi - lo))).astype(int)
        return [water.water_box(int(c), int(rng.integers(1 << 40)), sigma=rng.uniform(0.05, 0.15)) for c in counts]
    frames = read_structures(os.path.join(_directory(case), "input.data"))
    frames = [frames[k % len(frames)] for k in order]
    return [Structure(f.positions + rng.normal(scale=0.02, size=f.positions.shape), f.elements, box=f.box)
            for f in frames]


def _positions(structs):
    return np.ascontiguousarray(np.concatenate([s.positions for s in structs]))


def _pinned(*shape):
    t = torch.empty(shape, dtype=torch.float64)
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def _labels(structs, seed):
    """Energies and forces of the size a training set holds (hartree, bohr)."""
    rng = np.random.default_rng([seed, 11])
    n = sum(s.numAtoms for s in structs)
    return rng.normal(0.0, 1.0, len(structs)), rng.normal(0.0, 0.05, (n, 3))


def _kalman_order(case, structs, seed):
    rng = np.random.default_rng([seed, 13])
    es = rng.integers(0, len(structs), case["energy_updates"]).astype(np.int32)
    fs = rng.integers(0, len(structs), case["force_updates"]).astype(np.int32)
    fa = np.array([rng.integers(0, structs[k].numAtoms) for k in fs], dtype=np.int32)
    return es, fs, fa, rng.integers(0, 3, fs.size).astype(np.int32)


def _disturbed(weights, seed):
    return weights + np.random.default_rng([seed, 17]).normal(0.0, 0.02, weights.size)


class _State:
    """What a program holds between calls; `close` order: batch before mode."""

    def __init__(self, case):
        self.case = case
        self.mode = Mode(0).setupFromDirectory(_directory(case))
        self.batch = None
        self.trainer = None

    def __del__(self):
        for x in (self.trainer, self.batch, self.mode):
            if x is not None:
                x.close()


def prepare(case, seed):
    s = _State(case)
    structs = _structures(case, seed)
    if case["path"] == "kalman":
        # labels of the loaded networks, training from disturbed weights
        b = s.mode.batch(structs)
        b.setPositions(_positions(structs))
        b.evaluate()
        energies, forces = b.energies(), b.forces()
        b.close()
        s.trainer = Training(s.mode, structs, energies, forces)
        s.trainer.setWeights(_disturbed(s.trainer.weights(), seed))
        s.trainer.setupUpdaterKalman(0)
        s.trainer.setForceWeight(10.0)
        s.order = _kalman_order(case, structs, seed)
        return s
    if case["path"] == "adam":
        energies, forces = _labels(structs, seed)
        s.training = StudentTraining(s.mode, structs, energies, forces, batch_size=len(structs), seed=seed)
        s.trainer = s.training.trainer
        s.order = np.arange(len(structs))
        return s
    s.mode.setPrecision(case["precision"])
    s.batch = s.mode.batch(structs)
    n = sum(x.numAtoms for x in structs)
    s.positions, s.energies, s.forces = _pinned(n, 3), _pinned(len(structs)), _pinned(n, 3)
    s.positions[:] = _positions(structs)
    return s


def run(s):
    path = s.case["path"]
    if path == "evaluate":
        s.batch.evaluateHost(s.positions, s.energies, s.forces)
        if s.case["precision"] == "mixed":   # a program that takes the mixed form keeps single precision
            return {"energies": s.energies.astype(np.float32), "forces": s.forces.astype(np.float32)}
        return {"energies": s.energies, "forces": s.forces}
    if path == "values":
        s.batch.setPositions(s.positions)
        s.batch.evaluate(symmetryFunctionsOnly=True)
        g = s.batch.symmetryFunctions()
        return {"g": g.astype(np.float32) if s.case["precision"] == "mixed" else g}
    if path == "adam":
        loss, gradient = s.training.step(s.order, gradient=True)
        return {"loss": loss, "gradient": gradient, "weights": s.trainer.parameters()}
    es, fs, fa, fc = s.order
    ee = s.trainer.update(ENERGY, es)
    fe = s.trainer.update(FORCE, fs, fa, fc)
    return {"energy_errors": ee, "force_errors": fe, "weights": s.trainer.weights()}


# ---------------------------------------------------------------------------
# Work a pass cannot do without
# ---------------------------------------------------------------------------
# Per unordered neighbour pair (triplet) of an angular group and per member:
# geometry, cutoff and Gaussian of the pair (30 operations, exponential and
# root counted as one) and 4 per member for the value; the forces take the
# pair's three weighted sums (6 per member) and both neighbours' vectors (60).
def work(case):
    if "smallest" in case:
        lo, hi = case["smallest"], case["largest"]
        mean = lo if lo == hi else (hi - lo) / math.log(hi / lo)
        atoms = 3.0 * mean * case["boxes"]
        ang_rc = 8.0 if case["model"] == "student" else 12.0
        near = 3.0 * water.MOLECULE_DENSITY * 4.0 / 3.0 * math.pi * ang_rc ** 3
        all_near = 3.0 * water.MOLECULE_DENSITY * 4.0 / 3.0 * math.pi * 12.0 ** 3
        members, sfs, net = {"water40": (8, 40, 25), "water56": (8, 56, 64), "student": (4, 14, 16)}[case["model"]]
        pairs = 0.5 * near * near * 0.47                  # both neighbours within the cutoff of each other
        wide = 0.5 * 0.45 * near * near if case["model"] == "water56" else 0.0
        value = all_near * 8 * 4 + pairs * (30 + 4 * members) + wide * (12 + 4 * 16)
        force = all_near * 8 * 6 + pairs * (60 + 6 * members) + wide * (40 + 6 * 16)
    else:
        atoms, near, value_pair, sfs, net = {
            "rpbe": (1080.0, 109.0, 0.5 * 0.47 * (30 + 4 * 6), 30, 25),
            "anisole": (256.0, 210.0, 0.5 * (8 + 8 * 6 + 9 + 2 * 54), 354, 30),
            "qm9": (15.6, 14.6, 0.5 * (8 + 8 * 6 + 9 + 4 * 36), 45, 50)}[case["model"]]
        atoms *= case["boxes"]
        value, force = near * near * value_pair, near * near * value_pair * 2.0
    nets = 4.0 * (sfs * net + net * net)
    if case["path"] == "values":
        return {"bytes": atoms * (24 + 8 * sfs), "flops": atoms * value}
    if case["path"] == "adam":     # values and derivatives once, networks with their second-order pass
        return {"bytes": atoms * (24 + 24 + 8 * sfs), "flops": atoms * (value + force + 4 * nets)}
    if case["path"] == "kalman":   # the covariance's lower half is read and written by every update
        n = 2 * (40 * 25 + 25 + 25 * 25 + 25 + 25 + 1)
        updates = case["energy_updates"] + case["force_updates"]
        per_box = atoms / case["boxes"]
        return {"bytes": updates * (8.0 * n * n + 8.0 * per_box * sfs), "flops": updates * (4.0 * n * n + per_box * nets)}
    return {"bytes": atoms * (24 + 24 + 8), "flops": atoms * (value + force + nets)}


# ---------------------------------------------------------------------------
# The same results in plain 64-bit torch
# ---------------------------------------------------------------------------
_NUMBER = {"H": 1, "C": 6, "N": 7, "O": 8, "F": 9}
_ACTIVATION = {"t": torch.tanh, "p": lambda x: torch.nn.functional.softplus(x, threshold=35.0), "l": lambda x: x}


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Potential:
    """A model directory in torch: functions in the order the networks take
    them (by type, then cutoffs, widths and elements), scaling, networks."""

    def __init__(self, directory):
        rows = [line.split("#")[0].split() for line in open(os.path.join(directory, "input.nn"))]
        rows = [r for r in rows if r]
        key = {r[0]: r[1:] for r in reversed(rows)}
        self.symbols = sorted(key["elements"], key=_NUMBER.get)
        ne = len(self.symbols)
        at = {s: k for k, s in enumerate(self.symbols)}
        self.cutoff = int(key["cutoff_type"][0])
        self.length = float(key.get("conv_length", [1.0])[0])
        self.energy = float(key.get("conv_energy", [1.0])[0])
        self.mean = float(key.get("mean_energy", [0.0])[0])
        self.offset = torch.zeros(ne, dtype=torch.float64, device=_dev())
        for r in rows:
            if r[0] == "atom_energy":
                self.offset[at[r[1]]] = float(r[2])
        self.functions = [[] for _ in range(ne)]
        for r in rows:
            if r[0] != "symfunction_short":
                continue
            t, a = int(r[2]), r[3:]
            f = {"type": t}
            if t in (2, 20):
                pair, a = (at[a[0]], at[a[0]]), a[1:]
            elif t in (3, 9, 22):
                pair, a = tuple(sorted((at[a[0]], at[a[1]]))), a[2:]
            else:
                pair = (-1, -1)
            f["pair"] = pair
            if t == 2:
                eta, rs, rc = (float(x) for x in a[:3])
                order = (t, rc, eta, rs, pair)
                f.update(eta=eta / self.length ** 2, rs=rs * self.length, rc=rc * self.length)
            elif t in (3, 9):
                eta, lam, zeta, rc = (float(x) for x in a[:4])
                rs = float(a[4]) if len(a) > 4 else 0.0
                order = (t, rc, eta, rs, zeta, lam, pair)
                f.update(eta=eta / self.length ** 2, rs=rs * self.length, rc=rc * self.length, lam=lam, zeta=zeta)
            else:
                rl, rc = float(a[0]), float(a[1])
                angles = tuple(float(x) for x in a[2:4]) if t not in (20, 23) else ()
                f.update(rl=rl * self.length, rc=rc * self.length, angles=angles, asym=a[-1].endswith("a"))
                assert a[-1].rstrip("a") == "p2"
                order = (t, a[-1], pair, rc, rl, angles)
            self.functions[at[r[1]]].append((order, f))
        self.functions = [[f for _, f in sorted(fs, key=lambda x: x[0])] for fs in self.functions]
        self.rc = max(f["rc"] for fs in self.functions for f in fs)
        table = [line.split() for line in open(os.path.join(directory, "scaling.data")) if not line.startswith("#")]
        table = np.array([[float(x) for x in r[2:6]] for r in table[:sum(len(f) for f in self.functions)]])
        lo, hi = (float(key[k][0]) for k in ("scale_min_short", "scale_max_short"))
        if "scale_symmetry_functions_sigma" in key:
            factor, shift = (hi - lo) / table[:, 3], table[:, 2]
        else:
            factor, shift = (hi - lo) / (table[:, 1] - table[:, 0]), table[:, 2]
            assert "center_symmetry_functions" in key
        begin = np.cumsum([0] + [len(f) for f in self.functions])
        self.scaling = [(torch.tensor(factor[a:b], device=_dev()), torch.tensor(shift[a:b], device=_dev()), lo)
                        for a, b in zip(begin[:-1], begin[1:])]
        nodes = [int(x) for x in key["global_nodes_short"]]
        self.activations = key["global_activation_short"]
        self.sizes = [[len(f)] + nodes + [1] for f in self.functions]
        self.weights = torch.cat([torch.tensor(np.loadtxt(os.path.join(directory, "weights.%03d.data" % _NUMBER[s]),
                                                          usecols=0, ndmin=1)) for s in self.symbols]).to(_dev())
        self.counts = [sum((a + 1) * b for a, b in zip(z[:-1], z[1:])) for z in self.sizes]

    def network(self, e, g, weights):
        p = sum(self.counts[:e])
        for nin, nout, act in zip(self.sizes[e][:-1], self.sizes[e][1:], self.activations):
            w, b = weights[p:p + nin * nout].reshape(nin, nout), weights[p + nin * nout:p + (nin + 1) * nout]
            g = _ACTIVATION[act](g @ w + b)
            p += (nin + 1) * nout
        return g[:, 0]

    def fc(self, r, rc):
        x = r / rc
        y = torch.tanh(1.0 - x) ** 3 if self.cutoff == 2 else ((15.0 - 6.0 * x) * x - 10.0) * x ** 3 + 1.0
        return torch.where(r < rc, y, torch.zeros_like(y))

    @staticmethod
    def compact(x, lo, hi, asym):
        y = (x - 0.5 * (lo + hi)).abs() / (0.5 * (hi - lo))
        inside = y < 1.0
        y = torch.where(inside, y, torch.ones_like(y))
        if asym:
            y = (2.0 - y) * y
        return torch.where(inside, ((15.0 - 6.0 * y) * y - 10.0) * y ** 3 + 1.0, torch.zeros_like(y))

    def values(self, e, d, other):
        """Scaled functions [A, n] of A atoms of element e from their
        neighbours' vectors d [A, M, 3] and elements [A, M] (-1: none)."""
        real = other >= 0
        r = torch.sqrt(torch.where(real, (d * d).sum(2), torch.full_like(d[:, :, 0], 4.0 * self.rc ** 2)))
        fs = self.functions[e]
        masks = [(other == k).to(d.dtype) for k in range(len(self.symbols))]
        charge = real.to(d.dtype)
        for k, s in enumerate(self.symbols):
            charge = charge + (_NUMBER[s] - 1) * masks[k]
        if any(f["type"] not in (2, 20, 23) for f in fs):
            m = d.shape[1]
            both = real[:, :, None] & real[:, None, :] & ~torch.eye(m, dtype=torch.bool, device=d.device)
            dd = d[:, :, None, :] - d[:, None, :, :]
            rjk = torch.sqrt(torch.where(both, (dd * dd).sum(3), torch.full_like(dd[:, :, :, 0], 4.0 * self.rc ** 2)))
            cos = (d[:, :, None, :] * d[:, None, :, :]).sum(3) / (r[:, :, None] * r[:, None, :])
            both = both.to(d.dtype)
            angle = None
        parts, out = {}, []

        def once(name, make):
            if name not in parts:
                parts[name] = make()
            return parts[name]

        for f in fs:
            t, (e1, e2) = f["type"], f["pair"]
            if t in (2, 3, 9):
                w = once(("w", f["eta"], f["rs"], f["rc"]), lambda: torch.exp(-f["eta"] * (r - f["rs"]) ** 2) * self.fc(r, f["rc"]))
                if t == 2:
                    out.append((w * masks[e1]).sum(1))
                    continue
                k = torch.clamp(1.0 + f["lam"] * cos, min=0.0) ** f["zeta"] * both
                if t == 3:
                    k = k * once(("k", f["eta"], f["rs"], f["rc"]),
                                 lambda: torch.exp(-f["eta"] * (rjk - f["rs"]) ** 2) * self.fc(rjk, f["rc"]))
                scale = 2.0 ** (1.0 - f["zeta"])
            else:
                w = once(("w", f["rl"], f["rc"], f["asym"]), lambda: self.compact(r, f["rl"], f["rc"], f["asym"]))
                if t in (20, 23):
                    out.append((w * (masks[e1] if t == 20 else charge)).sum(1))
                    continue
                if angle is None:
                    angle = torch.acos(torch.clamp(cos * both, -1.0 + 1e-15, 1.0 - 1e-15))
                k = once(("a",) + f["angles"],
                         lambda: self.compact(angle, *(math.radians(x) for x in f["angles"]), False) * both)
                if t == 24:
                    k = k * once(("k", f["rl"], f["rc"], f["asym"]),
                                 lambda: self.compact(rjk, f["rl"], f["rc"], f["asym"]))
                scale = 1.0
            wj, wk = (w * charge, w * charge) if e1 < 0 else (w * masks[e1], w * masks[e2])
            pairs = (torch.matmul(k, wk[:, :, None])[:, :, 0] * wj).sum(1)
            out.append(pairs * scale * (0.5 if e1 == e2 else 1.0))
        factor, shift, lo = self.scaling[e]
        return lo + factor * (torch.stack(out, 1) - shift)


class _Set:
    """Structures with their neighbour lists: internal positions x [N, 3],
    elements, structure of each atom, and per atom the neighbours' indices
    [N, M] (-1: none) and lattice shifts [N, M, 3]."""

    def __init__(self, pot, structs):
        dev = _dev()
        at = {s: k for k, s in enumerate(pot.symbols)}
        self.pot = pot
        self.x = torch.tensor(_positions(structs), device=dev) * pot.length
        self.element = torch.tensor([at[y] for s in structs for y in s.elements], device=dev)
        self.number = len(structs)
        self.begin = np.cumsum([0] + [s.numAtoms for s in structs])
        self.of = torch.repeat_interleave(torch.arange(len(structs), device=dev),
                                          torch.tensor([s.numAtoms for s in structs], device=dev))
        found = []
        for k, s in enumerate(structs):
            x = self.x[self.begin[k]:self.begin[k + 1]]
            shifts = torch.zeros(1, 3, dtype=torch.float64, device=dev)
            if s.box is not None:
                box = torch.tensor(np.asarray(s.box, dtype=np.float64), device=dev) * pot.length
                x = x - torch.floor(x @ torch.linalg.inv(box)) @ box     # the cell's own copy of every atom
                self.x[self.begin[k]:self.begin[k + 1]] = x
                height = 1.0 / torch.linalg.norm(torch.linalg.inv(box), dim=0)
                n = [int(math.ceil(pot.rc / float(h))) for h in height]
                shifts = torch.tensor(list(itertools.product(*[range(-c, c + 1) for c in n])), dtype=torch.float64,
                                      device=dev) @ box
            home = int((shifts.abs().sum(1) == 0).nonzero()[0, 0])
            images = (x[None] + shifts[:, None]).reshape(-1, 3)
            near = ((images > x.min(0).values - pot.rc) & (images < x.max(0).values + pot.rc)).all(1).nonzero()[:, 0]
            images = images[near]
            step = max(1, int(1.5e8 // max(1, near.numel())))
            for a in range(0, x.shape[0], step):
                y = x[a:a + step]
                r2 = sum((images[None, :, c] - y[:, None, c]) ** 2 for c in range(3))
                own = torch.arange(a, a + y.shape[0], device=dev)[:, None] + home * x.shape[0]
                i, j = ((r2 < pot.rc ** 2) & (near[None] != own)).nonzero(as_tuple=True)
                j = near[j]
                found.append((i + a + self.begin[k], j % x.shape[0] + self.begin[k], shifts[j // x.shape[0]]))
        i, j, shift = (torch.cat(v) for v in zip(*found))
        count = torch.bincount(i, minlength=self.x.shape[0])
        slot = torch.arange(i.numel(), device=dev) - (torch.cumsum(count, 0) - count)[i]
        most = max(1, int(count.max()))
        self.neighbor = torch.full((self.x.shape[0], most), -1, device=dev)
        self.neighbor[i, slot] = j
        self.shift = torch.zeros(self.x.shape[0], most, 3, dtype=torch.float64, device=dev)
        self.shift[i, slot] = shift
        self.count = count

    def chunks(self, most=1.2e7, only=None):
        """(element, atoms) pieces whose pair arrays stay small."""
        for e in range(len(self.pot.symbols)):
            mine = (self.element == e) if only is None else ((self.element == e) & only)
            mine = mine.nonzero()[:, 0]
            mine = mine[torch.argsort(self.count[mine])]
            a = 0
            while a < mine.numel():
                b = min(mine.numel(), a + 4096)
                while b > a + 1 and (b - a) * int(self.count[mine[b - 1]]) ** 2 > most:
                    b = a + max(1, (b - a) * 3 // 4)
                yield e, mine[a:b]
                a = b

    def values(self, e, atoms, x):
        m = max(1, int(self.count[atoms].max()))
        j = self.neighbor[atoms, :m]
        d = x[j.clamp(min=0)] + self.shift[atoms, :m] - x[atoms][:, None]
        return self.pot.values(e, d, torch.where(j >= 0, self.element[j.clamp(min=0)], j))

    def evaluate(self, weights):
        """Energy per structure and forces, physical units."""
        x = self.x.clone().requires_grad_(True)
        energy = torch.zeros(self.number, dtype=torch.float64, device=x.device)
        for e, atoms in self.chunks():
            each = self.pot.network(e, self.values(e, atoms, x), weights)
            each.sum().backward()
            energy.index_add_(0, self.of[atoms], each.detach())
        atoms = torch.bincount(self.of, minlength=self.number)
        offset = torch.zeros_like(energy).index_add_(0, self.of, self.pot.offset[self.element])
        return (energy / self.pot.energy + atoms.double() * self.pot.mean + offset,
                -x.grad * (self.pot.length / self.pot.energy))

    def tangents(self, direction, only=None):
        """(element, atoms, functions, their derivative along `direction`)."""
        out = []
        with torch.no_grad():
            for e, atoms in self.chunks(4e6, only):
                g, dg = torch.func.jvp(lambda x: self.values(e, atoms, x), (self.x,), (direction,))
                out.append((e, atoms, g, dg))
        return out


def _numpy(t):
    return t.detach().cpu().numpy()


def _exact_adam(pot, data, structs, seed):
    energies, forces = (torch.tensor(v, device=_dev()) for v in _labels(structs, seed))
    e, f = data.evaluate(pot.weights)
    atoms = torch.bincount(data.of, minlength=data.number)
    de, df = (e - energies) / atoms, f - forces
    loss_e, loss_f = (de * de).sum() / len(structs), 10.0 * (df * df).sum() / df.numel()
    # d loss / d weights with the adjoints of the energies and of the forces held fixed
    a, u = 2.0 * de / atoms / len(structs), 20.0 * df / df.numel()
    weights = pot.weights.clone().requires_grad_(True)
    for el, at, g, dg in data.tangents(u):
        g = g.requires_grad_(True)
        each = pot.network(el, g, weights)
        slope, = torch.autograd.grad(each.sum(), g, create_graph=True)
        ((a[data.of[at]] * each).sum() - (slope * dg).sum()).backward()
    g = weights.grad
    step = 1e-3 * math.sqrt(1.0 - 0.999) / (1.0 - 0.9) * (0.1 * g) / (torch.sqrt(0.001 * g * g) + 1e-8)
    return {"loss": _numpy(torch.stack([loss_e + loss_f, loss_e, loss_f])), "gradient": _numpy(g),
            "weights": _numpy(weights - step)}


def _exact_kalman(pot, data, case, structs, seed):
    energies, forces = data.evaluate(pot.weights)
    es, fs, fa, fc = _kalman_order(case, structs, seed)
    n = pot.weights.numel()
    w = torch.tensor(_disturbed(_numpy(pot.weights), seed), device=_dev())
    p = torch.eye(n, dtype=torch.float64, device=_dev()) / 1e-2
    q, eta = 0.01, 0.01
    errors = {ENERGY: [], FORCE: []}
    still = data.tangents(torch.zeros_like(data.x), only=torch.isin(data.of, torch.tensor(es, device=_dev()).long()))
    for prop, k, atom, comp in [(ENERGY, s, 0, 0) for s in es] + [(FORCE, *o) for o in zip(fs, fa, fc)]:
        x = w.clone().requires_grad_(True)
        if prop == ENERGY:
            pred = sum(pot.network(el, g[data.of[at] == int(k)], x).sum() for el, at, g, _ in still)
            miss = energies[int(k)] - pred
        else:
            unit = torch.zeros_like(data.x)
            unit[data.begin[k] + atom, comp] = 1.0
            pred = 0.0
            for el, at, g, dg in data.tangents(unit, only=data.of == int(k)):
                g = g.requires_grad_(True)
                slope, = torch.autograd.grad(pot.network(el, g, x).sum(), g, create_graph=True)
                pred = pred - (slope * dg).sum()
            miss = forces[data.begin[k] + atom, comp] - pred
        h, = torch.autograd.grad(pred, x)
        miss = float(miss.detach())
        errors[prop].append(miss)
        if prop == FORCE:
            h, miss = 10.0 * h, 10.0 * miss
        v = p @ h
        if eta < 1.0:
            eta *= math.exp(2.302)
        gain = v / (float(h @ v) + 1.0 / eta)
        p -= torch.outer(gain, v)
        p.diagonal().add_(q)
        w = w + gain * miss
        if q > 1e-6:
            q *= math.exp(-2.302)
    return {"energy_errors": np.array(errors[ENERGY]), "force_errors": np.array(errors[FORCE]), "weights": _numpy(w)}


def exact(case, seed):
    structs = _structures(case, seed)
    pot = _Potential(_directory(case))
    data = _Set(pot, structs)
    if case["path"] == "adam":
        return _exact_adam(pot, data, structs, seed)
    if case["path"] == "kalman":
        return _exact_kalman(pot, data, case, structs, seed)
    if case["path"] == "values":
        rows = [None] * data.x.shape[0]
        with torch.no_grad():
            for e, atoms in data.chunks():
                g = _numpy(data.values(e, atoms, data.x))
                for k, a in enumerate(atoms.tolist()):
                    rows[a] = g[k]
        return {"g": np.concatenate(rows)}
    energy, forces = data.evaluate(pot.weights)
    return {"energies": _numpy(energy), "forces": _numpy(forces)}
