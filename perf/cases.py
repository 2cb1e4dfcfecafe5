"""Performance cases: what a user of this framework has it compute, with the
inputs, the call and the algorithmic work of each.

A case is a dict of plain values; ``kind`` names the entry point:

  md       one periodic configuration per call, as an MD or relaxation loop makes
           it: the drop-in serial wrapper (``api = "serial"``) or Calculator.evaluate
  batch    many configurations of uneven size in one call (training-set
           evaluation, ensembles): stage / launch / collect on packed arrays, or
           evaluate_batch on a list of configurations
  serve    a burst of single-point requests through the continuous-batching Server
  lammps   the pair style on a caller's neighbour list with ghost atoms
  clusters the per-cluster entry point (the caller owns the cluster loop)
  hist     the all-pairs histogram of the fingerprint tool

Parameter sets are seeded synthetic ones of the 12/8/4 and 12/10/4 recipes
(``synth.spec_c1`` .. ``spec_c5``); positions are uniform with a hard core, at the
densities of the benchmark's workloads.
"""

import atexit
import itertools
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from chimes_calculator_gb300 import FP64, MIXED, Calculator, ChimesError
from chimes_calculator_gb300 import chimescalc_serial_py as serial
from chimes_calculator_gb300 import synth
from chimes_calculator_gb300.serving import Server

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F8 = torch.float64
PRECISION = {"fp64": FP64, "mixed": MIXED}


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # an MD step of a small one-element cell through the drop-in wrapper: launches and latency
        {"name": "md-64-serial", "kind": "md", "api": "serial", "n": 64, "rho": 0.0878, "set": "c1", "tilt": 0.0,
         "precision": "fp64"},
        # an MD step of the benchmark's 1024-atom two-element box, plain FP64
        {"name": "md-1024-fp64", "kind": "md", "api": "calc", "n": 1024, "rho": 0.0962, "set": "c2", "tilt": 0.0,
         "precision": "fp64"},
        # single points on an odd-sized triclinic three-element cell
        {"name": "md-333-triclinic", "kind": "md", "api": "calc", "n": 333, "rho": 0.075, "set": "c5-3", "tilt": 0.3,
         "precision": "fp64"},
        # an MD step of a large cell, plain FP64, a size that is no multiple of anything
        {"name": "md-8191-fp64", "kind": "md", "api": "calc", "n": 8191, "rho": 0.0929, "set": "c3", "tilt": 0.0,
         "precision": "fp64"},
        # the 32768-atom box of the precision-form workload
        {"name": "md-32768-mixed", "kind": "md", "api": "calc", "n": 32768, "rho": 0.0929, "set": "c3", "tilt": 0.0,
         "precision": "mixed"},
        # energies, forces and stresses of a training set, FP64, a list of configurations
        {"name": "batch-384-fp64", "kind": "batch", "api": "list", "configs": 384, "n_max": 512, "precision": "fp64"},
        # the same at volume in the mixed form, packed arrays
        {"name": "batch-2000-mixed", "kind": "batch", "api": "packed", "configs": 2000, "n_max": 512,
         "precision": "mixed"},
        # a burst of requests of 16-4096 atoms on three parameter sets
        {"name": "serve-64-mixed", "kind": "serve", "requests": 64, "n_max": 4096, "precision": "mixed"},
        # a LAMMPS step between re-neighbourings, and one that re-neighbours
        {"name": "lammps-1024-step", "kind": "lammps", "n": 1024, "rho": 0.0962, "set": "c2", "rebuild": False,
         "precision": "fp64"},
        {"name": "lammps-2999-rebuild", "kind": "lammps", "n": 2999, "rho": 0.0962, "set": "c2", "rebuild": True,
         "precision": "fp64"},
        # a caller that owns its cluster loop: quadruplets of one configuration
        {"name": "clusters4-9001", "kind": "clusters", "body": 4, "count": 9001, "set": "c2"},
        # the 3-body self-histogram of a frame's fingerprints
        {"name": "hist3-40001", "kind": "hist", "body": 3, "count": 40001, "set": "c2"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "md", "batch", "batch", "serve", "lammps", "clusters", "hist"])
    if kind == "md":
        precision = rng.choice(["fp64", "fp64", "mixed"])
        n = _log(rng, 8, 8191 if precision == "fp64" else 32768)
        return {"kind": "md", "api": "serial" if n <= 512 and precision == "fp64" and rng.random() < 0.5 else "calc",
                "n": n, "rho": round(rng.uniform(0.05, 0.1), 4), "set": rng.choice(["c1", "c2", "c3", "c5-3"]),
                "tilt": rng.choice([0.0, 0.0, 0.3]), "precision": precision}
    if kind == "batch":
        precision = rng.choice(["fp64", "mixed"])
        return {"kind": "batch", "api": rng.choice(["list", "packed"]),
                "configs": _log(rng, 2, 384 if precision == "fp64" else 2000), "n_max": _log(rng, 32, 512),
                "precision": precision}
    if kind == "serve":
        return {"kind": "serve", "requests": _log(rng, 4, 64), "n_max": _log(rng, 128, 4096),
                "precision": rng.choice(["fp64", "mixed"])}
    if kind == "lammps":
        return {"kind": "lammps", "n": _log(rng, 300, 3000), "rho": round(rng.uniform(0.06, 0.1), 4),
                "set": rng.choice(["c1", "c2", "c3"]), "rebuild": rng.random() < 0.5,
                "precision": rng.choice(["fp64", "mixed"])}
    body = rng.choice([2, 3, 4])
    if kind == "clusters":
        return {"kind": "clusters", "body": body, "count": _log(rng, 1, 50000 if body < 4 else 9001), "set": "c2"}
    return {"kind": "hist", "body": body, "count": _log(rng, 300, 40001 if body < 4 else 9001), "set": "c2"}


# ---------------------------------------------------------------------------
# Parameter sets
# ---------------------------------------------------------------------------
_tmp = None
_sets = {}


def _spec(key):
    if key == "c1":
        return synth.spec_c1()
    if key.startswith("c5-"):
        return synth.specs_c5()[int(key[3:]) - 1]
    return {"c2": synth.spec_c2, "c3": synth.spec_c3, "c4": synth.spec_c4}[key]()


def _param_set(key):
    """(path of the parameter file, its contents as _read_params gives them)."""
    global _tmp
    if key not in _sets:
        if _tmp is None:
            _tmp = tempfile.mkdtemp(prefix="chimes_cases_")
            atexit.register(shutil.rmtree, _tmp, True)
        text = synth.build_param_text(_spec(key))
        path = os.path.join(_tmp, key + ".txt")
        with open(path, "w") as f:
            f.write(text)
        _sets[key] = (path, _read_params(text))
    return _sets[key]


def _read_params(text):
    """The parts of a ChIMES parameter file that define the model, as plain values."""
    p = {"pairs": [], "c2": [], "cl": {3: [], 4: []}, "cut": {3: None, 4: None}}
    lines = [ln.split() for ln in text.split("\n")]
    k = 0
    while k < len(lines):
        t = lines[k]
        if t[:1] == ["PAIRTYP:"]:
            p["orders"] = [int(v) for v in t[2:5]]
        elif t[:2] == ["ATOM", "TYPES:"]:
            nt = int(t[2])
            p["el"] = [lines[k + 3 + a][1] for a in range(nt)]
        elif t[:2] == ["#", "PAIRIDX"]:
            while len(lines[k + 1]) == 8:
                k += 1
                w = lines[k]
                p["pairs"].append((w[1], w[2], float(w[3]), float(w[4]), float(w[7])))
        elif t[:2] == ["FCUT", "TYPE:"]:
            p["offset"] = float(t[3])
        elif t[:1] == ["SPECIAL"]:
            p["cut"][int(t[1][0])] = float(t[4])
        elif t[:2] == ["PAIRTYPE", "PARAMS:"]:
            p["c2"].append([float(lines[k + 2 + c][1]) for c in range(p["orders"][0])])
        elif t[:1] in (["TRIPLETTYPE"], ["QUADRUPLETYPE"]):
            body = 3 if t[0] == "TRIPLETTYPE" else 4
            atoms = lines[k + 1][3:]
            npair = body * (body - 1) // 2
            total = int(lines[k + 2][-1])
            rows = [([int(v) for v in r[1:1 + npair]], float(r[-1])) for r in lines[k + 5:k + 5 + total]]
            p["cl"][body].append((atoms, rows))
            k += 4 + total
        k += 1
    return p


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _place(counts, cells, rmin, seed):
    """Uniform positions with a hard core in many periodic cells at once: atoms
    closer than rmin to a lower-numbered one are drawn again until none is.
    counts[S], cells[S][3][3]; returns [sum counts][3] Cartesian positions."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    out = [None] * len(counts)
    order = np.argsort(counts, kind="stable")
    a = 0
    while a < len(order):
        # configurations of similar size together, at most 2^28 distances at a time
        b = a + 1
        while b < len(order) and (b + 1 - a) * counts[order[b]] ** 2 <= 1 << 28:
            b += 1
        ids = order[a:b]
        a = b
        n = int(counts[ids[-1]])
        cell = torch.tensor(np.stack([cells[i] for i in ids]), device=DEV, dtype=torch.float32)
        real = torch.arange(n, device=DEV)[None, :] < torch.tensor([int(counts[i]) for i in ids], device=DEV)[:, None]
        frac = torch.rand((len(ids), n, 3), generator=g, device=DEV, dtype=F8)
        step = max(1, min(n, (1 << 28) // (len(ids) * n)))
        while True:
            f4 = frac.float()
            bad = torch.zeros_like(real)
            for r in range(0, n, step):
                d = f4[:, r:r + step, None, :] - f4[:, None, :, :]
                d -= d.round()
                d = torch.matmul(d.reshape(len(ids), -1, 3), cell).square().sum(-1).reshape(len(ids), -1, n)
                lower = torch.arange(n, device=DEV)[None, :] < torch.arange(r, min(n, r + step), device=DEV)[:, None]
                bad[:, r:r + step] = ((d < (1.001 * rmin) ** 2) & lower & real[:, None, :]).any(-1)
            bad &= real
            if not bool(bad.any()):
                break
            new = torch.rand(frac.shape, generator=g, device=DEV, dtype=F8)
            frac = torch.where(bad[..., None], new, frac)
        pos = torch.matmul(frac, torch.tensor(np.stack([cells[i] for i in ids]), device=DEV, dtype=F8)).cpu().numpy()
        for k, i in enumerate(ids):
            out[i] = pos[k, :counts[i]]
    return np.ascontiguousarray(np.concatenate(out))


def _cell(n, rho, tilt=0.0):
    side = (n / rho) ** (1.0 / 3.0)
    return np.array([[side, 0.0, 0.0], [tilt * side, side, 0.0], [0.5 * tilt * side, -tilt * side, side]])


def _config(n, rho, tilt, nt, seed):
    """(positions, type indices, cell) of one configuration."""
    cell = _cell(n, rho, tilt)
    pos = _place(np.array([n]), [cell], 1.2 if nt == 1 else 1.0, seed)
    types = np.random.default_rng(seed + 1).integers(0, nt, n).astype(np.int32)
    return pos, types, cell


def _many(count, n_min, n_max, elements, seed):
    """count configurations: sizes log-uniform, densities 0.05 - 0.12 (the same
    for every seed), elements[s] of them; positions and types from the seed."""
    rng = np.random.default_rng(count + n_max)
    n = np.maximum(n_min, np.round(np.exp(rng.uniform(math.log(n_min), math.log(n_max), count)))).astype(int)
    cells = [_cell(a, r) for a, r in zip(n, rng.uniform(0.05, 0.12, count))]
    ne = elements(rng, count)
    pos = _place(n, cells, 1.0, seed)
    rng = np.random.default_rng(seed)
    types = [rng.integers(0, e, a).astype(np.int32) for a, e in zip(n, ne)]
    ends = np.cumsum(n)
    return [(pos[e - a:e], t, c) for a, e, t, c in zip(n, ends, types, cells)]


_handles = {}


def _handle(key, make):
    """What a program opens once and keeps: a calculator or server with its parameter sets."""
    if key not in _handles:
        _handles[key] = make()
    return _handles[key]


def _calculator(sets, precision):
    c = Calculator(precision=PRECISION[precision], graph=True)
    for s in sets:
        c.load_params(_param_set(s)[0])
    return c


def _tuned(key, sets, precision, packed_of):
    """A calculator, autotuned once on the first inputs of its workload."""
    def make():
        c = _calculator(sets, precision)
        c.autotune(packed_of(c))
        return c
    return _handle(key, make)


def _case_key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


_serial_set = None


def _serial(key):
    """The wrapper module's static instance with this parameter set."""
    global _serial_set
    if _serial_set != key:
        if serial.chimes_wrapper is None:
            serial.chimes_wrapper = serial.init_chimes_wrapper()
        serial.set_chimes(small=False)
        serial.init_chimes(_param_set(key)[0])
        _serial_set = key
    return serial


SKIN = 0.3
SERVE_SETS = ("c5-1", "c5-2", "c5-3")


def _inputs(case, seed):
    """Plain numpy inputs of a case, from the seed alone."""
    kind = case["kind"]
    if kind == "md":
        nt = len(_spec(case["set"]).elements)
        return _config(case["n"], case["rho"], case["tilt"], nt, seed)
    if kind == "batch":
        return _many(case["configs"], 8, case["n_max"], lambda r, k: r.integers(1, 4, k), seed)
    if kind == "serve":
        slots = np.random.default_rng(case["requests"]).integers(0, 3, case["requests"])
        return slots, _many(case["requests"], 16, case["n_max"], lambda r, k: slots + 1, seed)
    if kind == "lammps":
        # one frame's ghosts and list; the seed moves the atoms less than half the skin since
        nt = len(_spec(case["set"]).elements)
        cell = _cell(case["n"], case["rho"])
        base = synth.Config(["X"] * case["n"], _place(np.array([case["n"]]), [cell], 1.3, case["n"]), cell)
        types = np.random.default_rng(case["n"]).integers(0, nt, case["n"]).astype(np.int32)
        cut = max(p[3] for p in _param_set(case["set"])[1]["pairs"])
        nl = synth.lammps_neighbors(base, types, cut + SKIN, seed=case["n"])
        nl.x = nl.x + np.random.default_rng(seed).uniform(-0.08, 0.08, (case["n"], 3))[nl.owner]
        return nl
    # clusters of one configuration, those the model evaluates, in a seeded order
    p = _param_set(case["set"])[1]
    body, count = case["body"], case["count"]
    per_atom = {2: 20.0, 3: 40.0, 4: 7.5}[body]
    n = max(64, int(1.1 * count / per_atom))
    while True:
        pos, types, cell = _config(n, 0.0962, 0.0, len(p["el"]), seed)
        nodes = _periodic(p, [(pos, types, cell)])
        cl = _clusters(p, nodes, body)
        if len(cl["node"]) >= count:
            break
        n = int(1.3 * n)
    g = torch.Generator(device="cpu")
    g.manual_seed(seed)
    pick = torch.randperm(len(cl["node"]), generator=g)[:count].to(cl["node"].device)
    dr = cl["dr"][pick]
    return (dr.norm(dim=-1).cpu().numpy(), dr.cpu().numpy(),
            nodes["type"][cl["node"][pick]].to(torch.int32).cpu().numpy())


def prepare(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    st = {"case": case, "x": x}
    if kind == "md" and case["api"] == "serial":
        pos, types, cell = x
        el = _param_set(case["set"])[1]["el"]
        st["args"] = (len(pos), *(list(pos[:, k]) for k in range(3)), [el[t] for t in types],
                      *(list(cell[k]) for k in range(3)))
        _serial(case["set"])
    elif kind == "md":
        st["calc"] = _tuned(_case_key(case), [case["set"]], case["precision"], lambda c: c.pack([x]))
    elif kind == "batch":
        st["calc"] = _tuned(_case_key(case), ["c4"], case["precision"], lambda c: c.pack(x))
        if case["api"] == "packed":
            st["packed"] = st["calc"].pack(x)
    elif kind == "serve":
        def make():
            s = Server(workers=4, max_batch_atoms=16384, precision=PRECISION[case["precision"]])
            for k in SERVE_SETS:
                s.load_params(_param_set(k)[0])
            s.autotune(x[1], [int(v) for v in x[0]])
            return s
        st["server"] = _handle(_case_key(case), make)
    elif kind == "lammps":
        # the lists belong to one simulation: a calculator of its own
        st["calc"] = _calculator([case["set"]], case["precision"])
        st["calc"].nl_compute(x, SKIN, rebuild=True)
    else:
        st["calc"] = _handle(("direct", case["set"]), lambda: _calculator([case["set"]], "fp64"))
    return st


def run(state):
    case, x = state["case"], state["x"]
    kind = case["kind"]
    if kind == "md" and case["api"] == "serial":
        n = len(x[0])
        zero = [0.0] * n
        fx, fy, fz, stress, energy = _serial(case["set"]).calculate_chimes(*state["args"], 0.0, zero, zero, zero,
                                                                           [0.0] * 9)
        return {"energy": np.float64(energy), "force": np.stack([np.frombuffer(f) for f in (fx, fy, fz)], axis=1),
                "stress": np.frombuffer(stress)}
    calc = state.get("calc")
    if kind == "md":
        return calc.evaluate(*x)
    if kind == "batch" and case["api"] == "list":
        res = calc.evaluate_batch(x)
        return {"energy": np.array([r["energy"] for r in res]), "force": np.concatenate([r["force"] for r in res]),
                "stress": np.stack([r["stress"] for r in res])}
    if kind == "batch":
        for attempt in range(6):     # a list that outgrows its buffer is reported by collect
            calc.stage(state["packed"])
            calc.launch()
            try:
                energy, force, stress = calc.collect()
                break
            except ChimesError:
                if attempt == 5:
                    raise
        return {"energy": energy, "force": force, "stress": stress.reshape(-1, 9)}
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(p, t, c, slot=int(s)) for s, (p, t, c) in zip(*x)]
        res = [server.take(i) for i in ids]
        return {"energy": np.array([r["energy"] for r in res]), "force": np.concatenate([r["force"] for r in res]),
                "stress": np.stack([r["stress"] for r in res])}
    if kind == "lammps":
        res = calc.nl_compute(x, SKIN, rebuild=case["rebuild"])
        return dict(res, energy=np.float64(res["energy"]))
    if kind == "clusters":
        return calc.clusters(case["body"], *x)
    counts, samples = calc.fp_histogram(case["body"], x[0], x[2])
    return {"counts": counts, "samples": samples}


# ---------------------------------------------------------------------------
# Algorithmic work
# ---------------------------------------------------------------------------
def _cluster_flops(key):
    """(flops per pair, per triplet, per quadruplet): tables, two multiply-adds
    per coefficient (energy side and gradient side) and the force scalars."""
    p = _param_set(key)[1]
    o2, o3, o4 = p["orders"]
    out = [12.0 * o2 + 36.0]
    for body, order, npair in ((3, o3, 3), (4, o4, 6)):
        rows = [len(r) for _, r in p["cl"][body]]
        out.append(npair * (6.0 * order + 36.0) + 4.0 * sum(rows) / len(rows) if rows else 0.0)
    return out


def _model_work(key, n, rho):
    """Flops of one configuration at density rho: list entries, triplets and
    quadruplets per atom of the 5.0 / 4.0 / 3.2 A cutoffs, measured on the
    1024-atom workload (25.3, 46.2 and 9.07 at 0.0962) and scaled by density."""
    f2, f3, f4 = _cluster_flops(key)
    x = rho / 0.0962
    return n * (25.3 * x * f2 + 46.2 * x * x * f3 + 9.07 * x ** 3 * f4)


def work(case):
    kind = case["kind"]
    if kind in ("md", "lammps"):
        n = case["n"]
        rows = sum(len(r) for b in (3, 4) for _, r in _param_set(case["set"])[1]["cl"][b])
        by = 52.0 * n + 12.0 * rows + 152
        if kind == "lammps":
            ghosts = ((n / case["rho"]) ** (1 / 3) + 10.6) ** 3 * case["rho"]
            by = 60.0 * ghosts + 12.0 * rows + (n * 4.19 * 5.3 ** 3 * case["rho"] * 4 if case["rebuild"] else 0)
        return {"bytes": by, "flops": _model_work(case["set"], n, case["rho"])}
    if kind in ("batch", "serve"):
        lo = 8 if kind == "batch" else 16
        mean = (case["n_max"] - lo) / math.log(case["n_max"] / lo)
        n = mean * (case["configs"] if kind == "batch" else case["requests"])
        # the second and third moments of a density uniform in 0.05 - 0.12
        f2, f3, f4 = _cluster_flops("c4" if kind == "batch" else "c5-2")
        flops = n * (25.3 * 0.085 / 0.0962 * f2 + 46.2 * 0.00763 / 0.0962 ** 2 * f3
                     + 9.07 * 0.000718 / 0.0962 ** 3 * f4)
        return {"bytes": 52.0 * n, "flops": flops}
    body, c = case["body"], case["count"]
    npair = body * (body - 1) // 2
    if kind == "clusters":
        return {"bytes": c * (32.0 * npair + 4 * body + 24 * body + 56 + 8 * npair),
                "flops": c * _cluster_flops(case["set"])[body - 2]}
    return {"bytes": c * (8.0 * npair + 4 * body) + 800, "flops": 0.5 * c * c * (3.0 * npair + 3)}


# ---------------------------------------------------------------------------
# 64-bit reference: the ChIMES model on explicit cluster lists, in plain torch
# ---------------------------------------------------------------------------
SLOTS = {2: [(0, 1)], 3: [(0, 1), (0, 2), (1, 2)], 4: [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]}


def _t(a, dtype=None):
    return torch.as_tensor(a, device=DEV, dtype=dtype)


def _ranges(count):
    """For count[k] items in group k: (group of each item, its number within the group)."""
    grp = torch.repeat_interleave(torch.arange(len(count), device=DEV), count)
    first = torch.cumsum(count, 0) - count
    return grp, torch.arange(len(grp), device=DEV) - first[grp]


def _periodic(p, configs):
    """Atoms and the periodic images near them, and each atom's neighbours
    within the longest cutoff whose parent is not numbered below it."""
    rc = max(q[3] for q in p["pairs"])
    sizes = [len(c[0]) for c in configs]
    cfg = torch.repeat_interleave(torch.arange(len(configs), device=DEV), _t(sizes))
    cells = np.stack([c[2] for c in configs])
    inv = np.linalg.inv(cells)
    frac = _t(np.concatenate([c[0] @ i for c, i in zip(configs, inv)]), F8)
    frac = frac - torch.floor(frac)
    vol = np.abs(np.linalg.det(cells))
    cross = np.stack([np.cross(cells[:, (k + 1) % 3], cells[:, (k + 2) % 3]) for k in range(3)], axis=1)
    margin = rc / (vol[:, None] / np.linalg.norm(cross, axis=2)) + 1e-9
    reach = np.ceil(margin.max(axis=0)).astype(int)
    H, mg = _t(cells, F8)[cfg], _t(margin, F8)[cfg]
    n = len(frac)
    xs, parent = [torch.bmm(frac[:, None], H)[:, 0]], [torch.arange(n, device=DEV)]
    for s in itertools.product(*(range(-r, r + 1) for r in reach)):
        if s == (0, 0, 0):
            continue
        f = frac + _t(s, F8)
        keep = ((f >= -mg) & (f < 1.0 + mg)).all(1).nonzero()[:, 0]
        xs.append(torch.bmm(f[keep][:, None], H[keep])[:, 0])
        parent.append(keep)
    x, parent = torch.cat(xs), torch.cat(parent)
    # bins of the cutoff's size, numbered per configuration with an empty rim
    gc = cfg[parent]
    lo = torch.full((len(configs), 3), math.inf, device=DEV, dtype=F8).scatter_reduce(
        0, gc[:, None].expand(-1, 3), x, "amin")
    b = torch.floor((x - lo[gc]) / rc).long() + 1
    dim = torch.zeros((len(configs), 3), device=DEV, dtype=torch.long).scatter_reduce(
        0, gc[:, None].expand(-1, 3), b, "amax") + 2
    first = torch.cumsum(dim.prod(1), 0) - dim.prod(1)
    key = first[gc] + (b[:, 0] * dim[gc, 1] + b[:, 1]) * dim[gc, 2] + b[:, 2]
    skey, order = torch.sort(key)
    off = _t(list(itertools.product((-1, 0, 1), repeat=3)))
    nk = (first[cfg][:, None] + ((b[:n, None, 0] + off[:, 0]) * dim[cfg, 1][:, None] + b[:n, None, 1] + off[:, 1])
          * dim[cfg, 2][:, None] + b[:n, None, 2] + off[:, 2]).reshape(-1)
    start = torch.searchsorted(skey, nk)
    grp, k = _ranges(torch.searchsorted(skey, nk, right=True) - start)
    i, j = grp // 27, order[start[grp] + k]
    d = x[j] - x[i]
    keep = (parent[j] >= i) & (j != i) & (d.square().sum(1) < rc * rc)
    return {"i": i[keep], "j": j[keep], "d": d[keep], "parent": parent, "n": n, "nodes": len(x),
            "type": torch.cat([_t(c[1]).long() for c in configs])[parent], "cfg": cfg, "vol": vol, "strict": False}


def _from_list(nl):
    """The same for a caller's neighbour list with ghost atoms."""
    i = _t(np.repeat(nl.ilist, nl.numneigh)).long()
    j, x, tag = _t(nl.neigh).long(), _t(nl.x, F8), _t(nl.tag).long()
    keep = tag[j] >= tag[i]
    i, j = i[keep], j[keep]
    order = torch.sort(i, stable=True).indices
    i, j = i[order], j[order]
    return {"i": i, "j": j, "d": x[j] - x[i], "parent": tag, "n": nl.nlocal, "nodes": len(x),
            "type": _t(nl.type).long(), "strict": True}


def _pick(lists, sel):
    return [v[sel] for v in lists]


def _clusters(p, nodes, body):
    """Clusters of one body order: node[M][body] and dr[M][P][3], each oriented
    as the neighbour lists give it (first atom i, members with parents not
    below the earlier members')."""
    par, cut = nodes["parent"], p["cut"].get(body)
    i, j, d = nodes["i"], nodes["j"], nodes["d"]
    if body == 2:
        if nodes["strict"]:
            i, j, d = _pick((i, j, d), par[j] > par[i])
        rout = _t([[q[3] for q in p["pairs"]]], F8)[0]
        pt = _pair_type(p, nodes["type"][i], nodes["type"][j])
        i, j, d = _pick((i, j, d), d.norm(dim=1) < rout[pt])
        return {"node": torch.stack([i, j], 1), "dr": d[:, None]}
    i, j, d = _pick((i, j, d), d.norm(dim=1) < cut)
    count = torch.bincount(i, minlength=nodes["nodes"])
    first = torch.cumsum(count, 0) - count
    e, k = _ranges(count[i])
    f = first[i[e]] + k
    e, f = _pick((e, f), (e != f) & (par[j[e]] <= par[j[f]]))
    e, f = _pick((e, f), (d[f] - d[e]).norm(dim=1) < cut)
    if body == 3:
        return {"node": torch.stack([i[e], j[e], j[f]], 1), "dr": torch.stack([d[e], d[f], d[f] - d[e]], 1)}
    t, k = _ranges(count[i[e]])
    g = first[i[e[t]]] + k
    e, f = e[t], f[t]
    e, f, g = _pick((e, f, g), (g != e) & (g != f) & (par[j[f]] <= par[j[g]]))
    e, f, g = _pick((e, f, g), ((d[g] - d[e]).norm(dim=1) < cut) & ((d[g] - d[f]).norm(dim=1) < cut))
    return {"node": torch.stack([i[e], j[e], j[f], j[g]], 1),
            "dr": torch.stack([d[e], d[f], d[g], d[f] - d[e], d[g] - d[e], d[g] - d[f]], 1)}


def _pair_index(p):
    nt = len(p["el"])
    out = np.zeros((nt, nt), dtype=int)
    for k, q in enumerate(p["pairs"]):
        a, b = p["el"].index(q[0]), p["el"].index(q[1])
        out[a, b] = out[b, a] = k
    return out


def _pair_type(p, a, b):
    return _t(_pair_index(p))[a, b]


def _tuple_map(p, types, body):
    """(cluster type, pair map) of an ordered type tuple: the cluster's pair q
    takes power map[q] of the type's list, from the first permutation of the
    atoms whose pair types are the list's."""
    pi, slots = _pair_index(p), SLOTS[body]
    ci = next(k for k, (atoms, _) in enumerate(p["cl"][body])
              if sorted(p["el"].index(a) for a in atoms) == sorted(types))
    at = [p["el"].index(a) for a in p["cl"][body][ci][0]]
    want = [pi[at[a], at[b]] for a, b in slots]
    for perm in itertools.permutations(range(body)):
        if [pi[types[perm[a]], types[perm[b]]] for a, b in slots] == want:
            run_pairs = [tuple(sorted((perm[a], perm[b]))) for a, b in slots]
            return ci, [run_pairs.index(s) for s in slots]
    raise ValueError("no permutation matches")


def _tables(p, pt, r, rout, order):
    """T[n], dT/dr[n] for n = 0..order and the cutoff and its slope, per distance."""
    lam, rin = (_t([q[k] for q in p["pairs"]], F8)[pt] for k in (4, 2))
    lo, hi = torch.exp(-rout / lam), torch.exp(-rin / lam)
    s = torch.exp(-r / lam)
    x = (s - 0.5 * (hi + lo)) / (0.5 * (hi - lo))
    g = -s / lam / (0.5 * (hi - lo))
    T, U = [torch.ones_like(x), x], [torch.ones_like(x), 2 * x]
    for _ in range(2, order + 1):
        T.append(2 * x * T[-1] - T[-2])
        U.append(2 * x * U[-1] - U[-2])
    D = [torch.zeros_like(x)] + [n * U[n - 1] * g for n in range(1, order + 1)]
    th = rout - p["offset"] * rout
    pi = 3.14159265359
    ph = (r - th) / (rout - th) * pi + pi / 2
    fc = torch.where(r < th, torch.ones_like(r), 0.5 + 0.5 * torch.sin(ph))
    fcd = torch.where(r < th, torch.zeros_like(r), 0.5 * torch.cos(ph) * pi / (rout - th))
    return torch.stack(T[:order + 1], 1), torch.stack(D[:order + 1], 1), fc, fcd


def _evaluate(p, types, dr, body):
    """Per cluster: energy, force scalar of each pair (force on its first atom
    is scalar * dr), and the last coefficient's own force scalars."""
    M, slots = len(dr), SLOTS[body]
    r = dr.norm(dim=-1)
    E, fs, last = torch.zeros(M, device=DEV, dtype=F8), torch.zeros_like(r), torch.zeros_like(r)
    if body == 2:
        pt = _pair_type(p, types[:, 0], types[:, 1])
        rout = _t([q[3] for q in p["pairs"]], F8)[pt]
        T, D, fc, fcd = _tables(p, pt, r[:, 0], rout, p["orders"][0])
        a = _t(p["c2"], F8)[pt]
        S, G = (a * T[:, 1:]).sum(1), (a * D[:, 1:]).sum(1)
        return fc * S, ((fc * G + fcd * S) / r[:, 0])[:, None], torch.ones_like(r)
    R, P = p["orders"][body - 2], len(slots)
    nt = len(p["el"])
    u = torch.zeros(M, device=DEV, dtype=torch.long)
    for k in range(body):
        u = u * nt + types[:, k]
    for tup in itertools.product(range(nt), repeat=body):
        sel = (u == sum(t * nt ** (body - 1 - k) for k, t in enumerate(tup))).nonzero()[:, 0]
        if not len(sel):
            continue
        ci, mp = _tuple_map(p, tup, body)
        rows = p["cl"][body][ci][1]
        A = np.zeros((R,) * P)
        for pw, c in rows:
            A[tuple(pw[m] for m in mp)] += c
        A = _t(A, F8).reshape(R if body == 3 else R ** 3, -1)
        lp, lc = [rows[-1][0][m] for m in mp], rows[-1][1]
        for sub in torch.split(sel, 1 << 18):
            tabs = []
            for q, (a, b) in enumerate(slots):
                pt = torch.full((len(sub),), int(_pair_index(p)[tup[a], tup[b]]), device=DEV)
                tabs.append(_tables(p, pt, r[sub, q], torch.full_like(r[sub, q], p["cut"][body]), R - 1))
            T, D = [t[0] for t in tabs], [t[1] for t in tabs]

            def outer(v):
                o = v[0]
                for w in v[1:]:
                    o = (o[:, :, None] * w[:, None, :]).reshape(len(o), -1)
                return o

            K = 1 if body == 3 else 3
            X, Y = outer(T[:K]), outer(T[K:])
            AY, XA = Y @ A.T, X @ A
            S = (X * AY).sum(1)
            G = []
            for q in range(P):
                v = [D[q] if m == q else T[m] for m in range(P)]
                G.append((outer(v[:K]) * AY).sum(1) if q < K else (XA * outer(v[K:])).sum(1))
            fc = torch.stack([t[2] for t in tabs], 1)
            fcd = torch.stack([t[3] for t in tabs], 1)
            E[sub] = fc.prod(1) * S
            for q in range(P):
                rest = torch.cat([fc[:, :q], fc[:, q + 1:]], 1).prod(1) / r[sub, q]
                fs[sub, q] = rest * (fc[:, q] * G[q] + fcd[:, q] * S)
                tl = torch.stack([T[m][:, lp[m]] for m in range(P) if m != q], 1).prod(1)
                last[sub, q] = lc * (fc[:, q] * D[q][:, lp[q]] + fcd[:, q] * T[q][:, lp[q]]) * rest * tl
    return E, fs, last


def _forces(fs, dr, body):
    f = torch.zeros((len(dr), body, 3), device=DEV, dtype=F8)
    for q, (a, b) in enumerate(SLOTS[body]):
        v = fs[:, q, None] * dr[:, q]
        f[:, a] += v
        f[:, b] -= v
    return f, -(fs[:, :, None, None] * dr[:, :, :, None] * dr[:, :, None, :]).sum(1)


def _model(p, nodes):
    """Energy and virial per configuration (one when none is given) and the force on every node."""
    ncfg = len(nodes["vol"]) if "vol" in nodes else 1
    E = torch.zeros(ncfg, device=DEV, dtype=F8)
    V = torch.zeros((ncfg, 3, 3), device=DEV, dtype=F8)
    F = torch.zeros((nodes["nodes"], 3), device=DEV, dtype=F8)
    for body in (2, 3, 4):
        if p["orders"][body - 2] <= 0:
            continue
        cl = _clusters(p, nodes, body)
        if not len(cl["node"]):
            continue
        e, fs, _ = _evaluate(p, nodes["type"][cl["node"]], cl["dr"], body)
        f, v = _forces(fs, cl["dr"], body)
        c = nodes["cfg"][cl["node"][:, 0]] if "cfg" in nodes else torch.zeros_like(cl["node"][:, 0])
        E.index_add_(0, c, e)
        V.index_add_(0, c, v)
        F.index_add_(0, cl["node"].reshape(-1), f.reshape(-1, 3))
    return E, V, F


def _exact_configs(p, configs):
    nodes = _periodic(p, configs)
    E, V, F = _model(p, nodes)
    f = torch.zeros((nodes["n"], 3), device=DEV, dtype=F8).index_add_(0, nodes["parent"], F)
    return E.cpu().numpy(), f.cpu().numpy(), (V.reshape(-1, 9).cpu().numpy() / nodes["vol"][:, None])


def exact(case, seed):
    kind = case["kind"]
    if kind == "hist":
        return None              # whole numbers
    x = _inputs(case, seed)
    if kind in ("md", "batch"):
        p = _param_set("c4" if kind == "batch" else case["set"])[1]
        e, f, s = _exact_configs(p, x if kind == "batch" else [x])
        if kind == "md":
            return {"energy": e[0], "force": f, "stress": s[0]}
        return {"energy": e, "force": f, "stress": s}
    if kind == "serve":
        slots, configs = x
        e, s, f = np.zeros(len(configs)), np.zeros((len(configs), 9)), [None] * len(configs)
        for k, name in enumerate(SERVE_SETS):
            ids = np.nonzero(slots == k)[0]
            if not len(ids):
                continue
            ek, fk, sk = _exact_configs(_param_set(name)[1], [configs[i] for i in ids])
            e[ids], s[ids] = ek, sk
            ends = np.cumsum([len(configs[i][0]) for i in ids])
            for i, b in zip(ids, ends):
                f[i] = fk[b - len(configs[i][0]):b]
        return {"energy": e, "force": np.concatenate(f), "stress": s}
    p = _param_set(case["set"])[1]
    if kind == "lammps":
        E, V, F = _model(p, _from_list(x))
        v = V[0].cpu().numpy()
        return {"energy": E[0].cpu().numpy(), "force": F.cpu().numpy(),
                "virial": np.array([v[0, 0], v[1, 1], v[2, 2], v[0, 1], v[0, 2], v[1, 2]])}
    dr, types = _t(x[1], F8), _t(x[2]).long()
    e, fs, last = _evaluate(p, types, dr, case["body"])
    f, v = _forces(fs, dr, case["body"])
    s = torch.stack([v[:, a, b] for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))], 1)
    return {"energy": e.cpu().numpy(), "force": f.cpu().numpy(), "stress": s.cpu().numpy(),
            "fscal": last.cpu().numpy()}
