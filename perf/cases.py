"""The calls a user of the correlation scan makes, as measurable cases.

Three kinds of work reach this library:

* ``scan``: ``FFTScan.scan`` over a rotation set with the receptor and ligand
  already set (host rotations in, host peaks out) -- the rot-scan worker's
  loop, at cubic and per-axis grid sizes, for each term set, from a handful of
  rotations to a whole set;
* ``pair`` / ``pairs``: a new receptor/ligand pair on an open context
  (receptor grids and transforms, ligand tables, then a scan), and a list of
  uneven pairs in one call with a tuned plan;
* ``predict`` / ``train``: the learned rotation proposal's inference over a
  rotation set and its training steps.

Molecules are seeded random-walk globules at protein density, as the
benchmark workloads use; rotations are uniform quaternions.
"""
import math

import numpy as np
import torch

from proddl2_gb300 import FFTScan, ScanConfig
from proddl2_gb300.pairs import PairInput, scan_pairs
from proddl2_gb300.proposal import Proposal

STEP = 1.2          # grid step, Angstrom
DENSITY = 0.05      # heavy atoms per cubic Angstrom
N_TYPES = 18
LJ_CUT = 9.0
DESC = 128
# the tuned plan of the uneven-pairs workload (streams; per grid edge the
# rotations per launch and the pencil-stage form)
PAIR_PLAN = {"n_streams": 4,
             "rot_batch": {48: 256, 64: 256, 80: 256, 96: 256, 112: 128, 128: 128, 144: 64},
             "pencil_form": {48: "fft", 64: "fft", 80: "tensor", 96: "tensor", 112: "tensor", 128: "tensor",
                             144: "fft"}}


def _scan(name, dims, terms, n_rec, n_lig, n_rot, peaks=4):
    return {"name": name, "kind": "scan", "nx": dims[0], "ny": dims[1], "nz": dims[2], "terms": terms,
            "n_rec": n_rec, "n_lig": n_lig, "n_rot": n_rot, "peaks": peaks}


def listed():
    return [
        # a handful of poses of a small pair: launches and host calls count
        _scan("few_ace48", (48, 48, 48), "shape_ace", 700, 150, 8),
        # plain shape search of a small complex, the whole rotation set
        _scan("shape64", (64, 64, 64), "shape", 1800, 450, 2000),
        # one worker task of the large pair: a short rotation range that does
        # not fill a launch group
        _scan("ace128_task", (128, 128, 128), "shape_ace", 4000, 1500, 100),
        # the exhaustive search of the large pair (~6 degree rotation set)
        _scan("ace128_full", (128, 128, 128), "shape_ace", 4000, 1500, 9000),
        # the same molecules on a grid sized per axis
        _scan("ace_box112x120x126", (112, 120, 126), "shape_ace", 4000, 1500, 1024),
        # the soft-core Lennard-Jones potential (the default potentialName)
        _scan("lj128", (128, 128, 128), "lj_comp", 4000, 1500, 2000),
        # the default potential on the default grid rule: sizes per axis
        _scan("lj_box90x96x100", (90, 96, 100), "lj_comp", 2500, 800, 1000),
        # many translations kept per rotation (for a later refinement)
        _scan("deep80", (80, 80, 80), "shape_ace", 1500, 400, 1000, peaks=32),
        # a new pair on an open context: set-up and scan
        {"name": "new_pair96", "kind": "pair", "nx": 96, "ny": 96, "nz": 96, "terms": "shape_ace", "n_rec": 2500,
         "n_lig": 700, "n_rot": 512, "peaks": 4},
        # uneven pairs in one call
        {"name": "pairs8", "kind": "pairs", "n_pairs": 8, "n_rot": 400, "peaks": 4},
        # ranking a rotation set with the trained proposal
        {"name": "predict9000", "kind": "predict", "n_lig": 450, "n_rot": 9000},
        # training steps of the proposal
        {"name": "train20", "kind": "train", "n_pairs": 4, "n_lig": 450, "n_samples": 2000, "steps": 20,
         "batch": 256},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _atoms(radius):
    return int(4.0 / 3.0 * math.pi * radius ** 3 * DENSITY)


# FFT sizes per axis: the sizes findBestSize gives between 40 and 150
_BOX = [n for n in range(40, 151)
        if any(2 ** a * 3 ** b * 5 ** c * 7 ** d * e == n for a in range(8) for b in range(5) for c in range(4)
               for d in range(3) for e in (1, 11, 13))]
_CUBIC = (48, 64, 80, 96, 112, 128, 144)


def draw(rng):
    kind = rng.choice(["scan", "scan", "scan", "scan", "scan", "scan", "pair", "pairs", "predict", "train"])
    if kind == "pairs":
        return {"kind": "pairs", "n_pairs": rng.randint(2, 9), "n_rot": int(_log(rng, 60, 400)), "peaks": 4}
    if kind == "predict":
        return {"kind": "predict", "n_lig": int(_log(rng, 150, 2000)), "n_rot": int(_log(rng, 40, 20000))}
    if kind == "train":
        return {"kind": "train", "n_pairs": rng.randint(1, 6), "n_lig": int(_log(rng, 150, 1500)),
                "n_samples": int(_log(rng, 300, 4000)), "steps": rng.randint(2, 24),
                "batch": rng.choice([64, 100, 128, 200, 256, 512])}
    terms = rng.choice(["shape_ace", "shape_ace", "shape", "lj_comp", "lj_comp", "lj_avg"])
    if kind == "pair" and terms == "lj_avg":
        terms = "shape_ace"
    if rng.random() < 0.5:
        n = rng.choice(_CUBIC)
        dims = (n, n, n)
    else:
        c = rng.choice([n for n in _BOX if 48 <= n <= 128])
        near = [n for n in _BOX if abs(n - c) <= 22]
        dims = (rng.choice(near), rng.choice(near), rng.choice(near))
    half = min(dims) * STEP / 2
    n_rec = max(60, min(6000, _atoms(rng.uniform(0.30, 0.45) * half)))
    n_lig = max(20, min(2000, _atoms(rng.uniform(0.16, 0.28) * half)))
    if terms == "shape":
        n_lig = max(n_lig, 200)  # whole-number scores: a tiny ligand's best cells are mostly ties
    k = {"shape_ace": N_TYPES, "shape": 1, "lj_comp": 2, "lj_avg": 1}[terms]
    # the cost of a drawn pass stays below the exhaustive search's
    most = 1.5e10 / (dims[0] * dims[1] * dims[2] * (0.3 * k + 1.0))
    n_rot = max(4, int(min(_log(rng, 6, 6000), most)))
    peaks = 4
    if dims in [(n, n, n) for n in _CUBIC] and kind == "scan" and terms == "shape_ace":
        peaks = rng.choice([1, 4, 4, 8, 24, 48])
    return {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "terms": terms, "n_rec": n_rec,
            "n_lig": n_lig, "n_rot": n_rot, "peaks": peaks}


# ---------------------------------------------------------------------------
# seeded inputs
# ---------------------------------------------------------------------------
def _globule(n, rng):
    """Chain of n atoms, 3.8 A steps, kept inside a sphere of matching density."""
    radius2 = (3.0 * n / (4.0 * math.pi * DENSITY)) ** (2.0 / 3.0)
    steps = rng.normal(size=(4 * n + 64, 3))
    steps *= 3.8 / np.linalg.norm(steps, axis=1)[:, None]
    steps = steps.tolist()
    x = y = z = 0.0
    pts, at = [(x, y, z)], 0
    while len(pts) < n:
        for _ in range(64):
            dx, dy, dz = steps[at % len(steps)]
            at += 1
            u, v, w = x + dx, y + dy, z + dz
            if u * u + v * v + w * w <= radius2:
                break
        else:
            u, v, w = 0.9 * x, 0.9 * y, 0.9 * z
        x, y, z = u, v, w
        pts.append((x, y, z))
    return np.array(pts) + rng.normal(scale=0.05, size=(n, 3))


def _molecules(rng, n_rec, n_lig):
    rec, lig = _globule(n_rec, rng), _globule(n_lig, rng)
    rec -= 0.5 * (rec.min(axis=0) + rec.max(axis=0))
    lig -= 0.5 * (lig.min(axis=0) + lig.max(axis=0))
    return rec, lig, rng.integers(0, N_TYPES, n_rec).astype(np.int32), rng.integers(0, N_TYPES, n_lig).astype(np.int32)


def _rotations(rng, n):
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    w, x, y, z = q.T
    r = np.empty((n, 3, 3))
    r[:, 0, 0], r[:, 0, 1], r[:, 0, 2] = 1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)
    r[:, 1, 0], r[:, 1, 1], r[:, 1, 2] = 2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)
    r[:, 2, 0], r[:, 2, 1], r[:, 2, 2] = 2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)
    return r


def _ace(rng):
    m = rng.uniform(-1.0, 1.0, size=(N_TYPES, N_TYPES))
    return np.triu(m) + np.triu(m, 1).T


def _lj(rng, n):
    return rng.uniform(3.0, 3.9, n), rng.uniform(0.05, 0.6, n), np.full(n, 0.4)


def _scan_inputs(case, seed):
    rng = np.random.default_rng([seed, 1])
    rec, lig, rt, lt = _molecules(rng, case["n_rec"], case["n_lig"])
    return {"rec": rec, "lig": lig, "rt": rt, "lt": lt, "ace": _ace(rng), "rot": _rotations(rng, case["n_rot"]),
            "lj_rec": _lj(rng, len(rec)), "lj_lig": _lj(rng, len(lig))}


def _pair_list(case, seed):
    """Receptors 800-6000 and ligands 300-2000 atoms, log-uniform; the grid
    edge covers both molecules and a margin."""
    rng = np.random.default_rng([seed, 2])
    ace, out = _ace(rng), []
    for _ in range(case["n_pairs"]):
        nr = int(math.exp(rng.uniform(math.log(800), math.log(6000))))
        nl = int(math.exp(rng.uniform(math.log(300), math.log(2000))))
        rec, lig, rt, lt = _molecules(rng, nr, nl)
        need = math.ceil((2 * np.linalg.norm(rec, axis=1).max() + 2 * np.linalg.norm(lig, axis=1).max() + 12) / STEP)
        out.append({"rec": rec, "lig": lig, "rt": rt, "lt": lt, "rot": _rotations(rng, case["n_rot"]),
                    "n": min(n for n in _CUBIC if n >= need or n == _CUBIC[-1])})
    return ace, out


_LAYERS = ((16, 1), (32, 16), (64, 32))


def _network(seed):
    """He-normal weights in the library's parameter order: conv1-3 (weights,
    biases), fc1 [640][256] and bias, fc2 and bias."""
    rng = np.random.default_rng([seed, 3])
    parts = []
    for co, ci in _LAYERS:
        parts += [rng.normal(scale=math.sqrt(2.0 / (27 * ci)), size=co * ci * 27), rng.normal(scale=0.02, size=co)]
    parts += [rng.normal(scale=math.sqrt(2.0 / 640), size=640 * 256), rng.normal(scale=0.02, size=256)]
    parts += [rng.normal(scale=math.sqrt(2.0 / 256), size=256), rng.normal(scale=0.02, size=1)]
    return np.concatenate(parts).astype(np.float32)


def _learned_inputs(case, seed):
    rng = np.random.default_rng([seed, 4])
    n_pairs = case.get("n_pairs", 1)
    ligs, descs = [], []
    for _ in range(n_pairs):
        x = _globule(case["n_lig"], rng)
        ligs.append(x - 0.5 * (x.min(axis=0) + x.max(axis=0)))
        descs.append((rng.random(DESC) / DESC).astype(np.float32))
    n = case.get("n_rot", case.get("n_samples"))
    rots = [_rotations(rng, n) for _ in range(n_pairs)]
    targets = [rng.normal(size=n).astype(np.float32) for _ in range(n_pairs)]
    return ligs, descs, rots, targets


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _context(case, ace):
    cubic = case["nx"] == case["ny"] == case["nz"]
    return FFTScan(ScanConfig(grid_n=case["nx"], grid_dims=None if cubic else (case["nx"], case["ny"], case["nz"]),
                              grid_step=STEP, term_set=case["terms"], peaks_per_rot=case["peaks"], n_types=N_TYPES,
                              ace_matrix=ace, lj_cut=LJ_CUT))


def _set_pair(scan, terms, i):
    if terms in ("lj_comp", "lj_avg"):
        scan.set_pair_lj(i["rec"], *i["lj_rec"], i["lig"], *i["lj_lig"][:2])
    else:
        scan.set_receptor(i["rec"], i["rt"])
        scan.set_ligand(i["lig"], i["lt"])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("scan", "pair"):
        i = _scan_inputs(case, seed)
        s = _context(case, i["ace"])
        if kind == "scan":
            _set_pair(s, case["terms"], i)
        return {"kind": kind, "scan": s, "terms": case["terms"], "inputs": i}
    if kind == "pairs":
        ace, pairs = _pair_list(case, seed)
        cfg = ScanConfig(grid_step=STEP, term_set="shape_ace", peaks_per_rot=case["peaks"], n_types=N_TYPES,
                         ace_matrix=ace)
        inputs = [PairInput(p["rec"], p["lig"], p["rot"], p["rt"], p["lt"], grid_n=p["n"]) for p in pairs]
        return {"kind": kind, "config": cfg, "pairs": inputs}
    ligs, descs, rots, targets = _learned_inputs(case, seed)
    p = Proposal(seed=seed)
    p.params = _network(seed)
    ids = [p.add_pair(x, desc=d) for x, d in zip(ligs, descs)]
    if kind == "predict":
        return {"kind": kind, "net": p, "id": ids[0], "rot": rots[0]}
    for k, r, t in zip(ids, rots, targets):
        p.add_samples(k, r, t)
    return {"kind": kind, "net": p, "steps": case["steps"], "batch": case["batch"], "seed": seed}


def _peaks(r):
    p = r.peaks
    return {"rot_id": p["rot_id"], "cell": p["cell"], "t": p["t"], "score": p["score"], "n": r.n_peaks}


def run(state):
    kind = state["kind"]
    if kind == "scan":
        return _peaks(state["scan"].scan(state["inputs"]["rot"]))
    if kind == "pair":
        _set_pair(state["scan"], state["terms"], state["inputs"])
        return _peaks(state["scan"].scan(state["inputs"]["rot"]))
    if kind == "pairs":
        results, _ = scan_pairs(state["config"], state["pairs"], tune=False, plan=PAIR_PLAN)
        return [_peaks(r) for r in results]
    if kind == "predict":
        return state["net"].predict(state["id"], state["rot"])
    loss = state["net"].train(state["steps"], state["batch"], lr=1e-3, seed=state["seed"])
    return {"loss": loss, "params": state["net"].params}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _scan_work(dims, k, n_rec, n_lig, n_rot, peaks):
    """One forward transform of the ligand per term and one inverse of the
    summed spectrum per rotation; spectra, atoms and rotations read once,
    peaks written once."""
    v = dims[0] * dims[1] * dims[2]
    half = dims[0] * dims[1] * (dims[2] // 2 + 1)
    flops = n_rot * ((k + 1) * 2.5 * v * math.log2(v) + 8.0 * k * half)
    return {"bytes": k * half * 8 + n_rec * 28 + n_lig * 28 + n_rot * (72 + 48 * peaks + 4), "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("scan", "pair"):
        dims = (case["nx"], case["ny"], case["nz"])
        k = {"shape_ace": N_TYPES, "shape": 1, "lj_comp": 2, "lj_avg": 1}[case["terms"]]
        w = _scan_work(dims, k, case["n_rec"], case["n_lig"], case["n_rot"], case["peaks"])
        if kind == "pair":
            v = dims[0] * dims[1] * dims[2]
            w["flops"] += k * 2.5 * v * math.log2(v)
        return w
    if kind == "pairs":
        w = _scan_work((80, 80, 80), N_TYPES, 2600, 900, case["n_rot"], case["peaks"])
        return {m: case["n_pairs"] * x for m, x in w.items()}
    macs = 512 * 27 * 16 + 64 * 432 * 32 + 8 * 864 * 64 + 640 * 256 + 256
    params = 27 * 16 + 16 + 432 * 32 + 32 + 864 * 64 + 64 + 640 * 256 + 256 + 257
    if kind == "predict":
        return {"bytes": case["n_rot"] * 76 + 4 * params, "flops": 2.0 * macs * case["n_rot"]}
    n = case["steps"] * case["batch"]
    return {"bytes": n * 80 + case["steps"] * params * 28, "flops": 6.0 * macs * n}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Grid:
    """Centred grid: zero = -(h + h (n - 1)) / 2 per axis, cell = trunc((x -
    (zero - h)) / h) - 1, centre of cell i = zero + h / 2 + h i."""

    def __init__(self, dims):
        self.dims = torch.tensor(dims, device=_device())
        self.zero = [-(STEP + STEP * (n - 1)) / 2.0 for n in dims]
        self.shape = tuple(dims)

    def cell(self, x):
        z = torch.tensor([v - STEP for v in self.zero], dtype=torch.float64, device=x.device)
        return torch.trunc((x - z) / STEP).to(torch.int64) - 1

    def near(self, xyz, cut):
        """(atom, flat cell, r^2) of the cells in each atom's cropped box."""
        lo = self.cell(xyz - cut).clamp(min=0)
        hi = torch.minimum(self.cell(xyz + cut), self.dims - 1)
        m = int(2 * cut / STEP) + 3
        o = torch.arange(m, device=xyz.device)
        g = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(1, -1, 3)
        c = lo[:, None, :] + g
        ok = (c <= hi[:, None, :]).all(-1)
        base = torch.tensor([z + STEP / 2.0 for z in self.zero], dtype=torch.float64, device=xyz.device)
        d = base + STEP * c.to(torch.float64) - xyz[:, None, :]
        r2 = d[..., 0] ** 2 + d[..., 1] ** 2 + d[..., 2] ** 2
        flat = (c[..., 0] * self.shape[1] + c[..., 1]) * self.shape[2] + c[..., 2]
        atom = torch.arange(len(xyz), device=xyz.device)[:, None].expand_as(flat)
        return atom[ok], flat[ok], r2[ok]


def _receptor_terms(grid, terms, i):
    dev = _device()
    v = grid.shape[0] * grid.shape[1] * grid.shape[2]
    xyz = torch.tensor(i["rec"], dtype=torch.float64, device=dev)
    floor2 = (STEP / 4.0) ** 2
    if terms in ("lj_comp", "lj_avg"):
        sig, eps, alpha = (torch.tensor(a, dtype=torch.float64, device=dev) for a in i["lj_rec"])
        sig_l, eps_l = float(np.mean(i["lj_lig"][0])), float(np.mean(i["lj_lig"][1]))
        out = torch.zeros(2 if terms == "lj_comp" else 1, v, dtype=torch.float64, device=dev)
        for a0 in range(0, len(xyz), 512):
            a, cell, r2 = grid.near(xyz[a0:a0 + 512], LJ_CUT)
            keep = r2 <= LJ_CUT * LJ_CUT
            a, cell, r2 = a[keep] + a0, cell[keep], r2[keep].clamp(min=floor2)
            if terms == "lj_comp":
                e6 = 4 * eps[a].sqrt() * sig[a] ** 3
                big = r2 ** 3 + alpha[a] * (sig[a] * sig_l) ** 3
                out[0].index_add_(0, cell, e6 * sig[a] ** 3 / big / big)
                out[1].index_add_(0, cell, -e6 / big)
            else:
                s6 = (sig[a] * sig_l) ** 3
                e6 = 4 * (eps[a] * eps_l).sqrt() * s6
                e12, as6 = e6 * s6, alpha[a] * s6

                def f(r):
                    big = r ** 6 + as6
                    return (e12 / big - e6) / big
                c = torch.full_like(as6, LJ_CUT)
                big = c ** 6 + as6
                # force and energy zero at the cutoff: f(r) - f(c) - f'(c)(r - c)
                slope = 6 * c ** 5 * (e6 / big ** 2 - 2 * e12 / big ** 3)
                out[0].index_add_(0, cell, f(r2.sqrt()) - f(c) - slope * (r2.sqrt() - c))
        return out.reshape(-1, *grid.shape)
    flag = torch.zeros(v, dtype=torch.int64, device=dev)
    dens = torch.zeros(N_TYPES, v, dtype=torch.float64, device=dev) if terms == "shape_ace" else None
    rt = torch.tensor(i["rt"], device=dev).to(torch.int64)
    for a0 in range(0, len(xyz), 1024):
        _, cell, r2 = grid.near(xyz[a0:a0 + 1024], 2.2 + 1.8)
        near = r2 <= (2.2 + 1.8) * (2.2 + 1.8)
        flag.index_reduce_(0, cell[near], 1 + (r2[near] <= 2.2 * 2.2).to(torch.int64), "amax")
        if dens is not None:
            a, cell, r2 = grid.near(xyz[a0:a0 + 1024], 6.0)
            keep = r2 <= 36.0
            r = r2[keep].clamp(min=floor2).sqrt()
            dens.reshape(-1).index_add_(0, rt[a[keep] + a0] * v + cell[keep],
                                        1.0 / (1.0 + torch.exp(7.0 * (0.15 * r - 0.6))))
    shape = torch.where(flag == 2, -15.0, torch.where(flag == 1, 1.0, 0.0)).to(torch.float64)
    if dens is None:
        return (-shape).reshape(1, *grid.shape)
    e = torch.tensor(i["ace"], dtype=torch.float64, device=dev)
    return (e.T @ dens - shape).reshape(-1, *grid.shape)


def _exact_scan(dims, terms, i, peaks):
    """The lowest correlation cells of every rotation through 3-D FFTs."""
    dev, grid = _device(), _Grid(dims)
    spec = torch.fft.rfftn(_receptor_terms(grid, terms, i), dim=(1, 2, 3)).conj()
    k, v = spec.shape[0], dims[0] * dims[1] * dims[2]
    lig = torch.tensor(i["lig"], dtype=torch.float64, device=dev)
    rot = torch.tensor(i["rot"], dtype=torch.float64, device=dev)
    if terms == "shape_ace":
        term, w = [torch.tensor(i["lt"], device=dev).to(torch.int64)], [torch.ones(len(lig), device=dev)]
    elif terms == "lj_comp":
        sig, eps = (torch.tensor(a, dtype=torch.float64, device=dev) for a in i["lj_lig"][:2])
        term = [torch.full((len(lig),), t, device=dev) for t in (0, 1)]
        w = [eps.sqrt() * sig ** 6, eps.sqrt() * sig ** 3]
    else:
        term, w = [torch.zeros(len(lig), dtype=torch.int64, device=dev)], [torch.ones(len(lig), device=dev)]
    scores, moves = [], []
    n = torch.tensor(dims, device=dev)
    for r in rot:
        p = r[:, 0] * lig[:, :1] + r[:, 1] * lig[:, 1:2] + r[:, 2] * lig[:, 2:]
        c = grid.cell(p)
        flat = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
        g = torch.zeros(k * v, dtype=torch.float64, device=dev)
        for t, x in zip(term, w):
            g.index_add_(0, t * v + flat, x.to(torch.float64))
        f = torch.fft.rfftn(g.reshape(k, *dims), dim=(1, 2, 3))
        corr = torch.fft.irfftn((f * spec).sum(0), s=dims, dim=(0, 1, 2)).reshape(-1)
        s, at = torch.topk(corr, peaks, largest=False, sorted=True)
        cell = torch.stack([at // (dims[1] * dims[2]), (at // dims[2]) % dims[1], at % dims[2]], -1)
        y = -cell
        y = torch.where(y < -(n // 2), y + n, y)
        scores.append(s)
        moves.append(STEP * y.to(torch.float64))
    # equal scores (whole numbers with the shape term alone) leave the choice
    # of the translation open
    t = torch.stack(moves).cpu().numpy() if terms != "shape" else None
    return {"rot_id": None, "cell": None, "t": t, "score": torch.stack(scores).cpu().numpy(), "n": None}


def _exact_predict(case, seed):
    dev = _device()
    ligs, descs, rots, _ = _learned_inputs(case, seed)
    w = torch.tensor(_network(seed), dtype=torch.float64, device=dev)
    xyz, half = ligs[0], np.sqrt((ligs[0] ** 2).sum(1)).max()
    at, layers = 0, []
    for co, ci in _LAYERS:
        layers.append((w[at:at + co * ci * 27].reshape(co, ci, 3, 3, 3), w[at + co * ci * 27:at + co * (ci * 27 + 1)]))
        at += co * (ci * 27 + 1)
    fc1, b1 = w[at:at + 640 * 256].reshape(640, 256), w[at + 640 * 256:at + 641 * 256]
    at += 641 * 256
    fc2, b2 = w[at:at + 256], w[at + 256]
    lig = torch.tensor(xyz, dtype=torch.float64, device=dev)
    desc = torch.tensor(descs[0], dtype=torch.float64, device=dev)
    out = []
    for r in torch.tensor(rots[0], dtype=torch.float64, device=dev).split(500):
        p = r[:, None, :, 0] * lig[:, :1] + r[:, None, :, 1] * lig[:, 1:2] + r[:, None, :, 2] * lig[:, 2:]
        c = torch.floor((p + half) / (2.0 * half / 16)).to(torch.int64).clamp(0, 15)
        flat = (c[..., 0] * 16 + c[..., 1]) * 16 + c[..., 2]
        x = torch.zeros(len(r), 4096, dtype=torch.float64, device=dev)
        x.scatter_add_(1, flat, torch.full_like(flat, 0.25, dtype=torch.float64))
        x = x.reshape(-1, 1, 16, 16, 16)
        for wt, b in layers:
            x = torch.nn.functional.conv3d(x, wt, b, stride=2, padding=1).relu()
        u = torch.cat([x.reshape(len(r), 512), desc.expand(len(r), DESC)], 1)
        out.append((u @ fc1 + b1).relu() @ fc2 + b2)
    return torch.cat(out).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("scan", "pair"):
        dims = (case["nx"], case["ny"], case["nz"])
        k = {"shape_ace": N_TYPES, "shape": 1, "lj_comp": 2, "lj_avg": 1}[case["terms"]]
        if case["n_rot"] * (k + 1) * dims[0] * dims[1] * dims[2] > 4e10:
            return None
        return _exact_scan(dims, case["terms"], _scan_inputs(case, seed), case["peaks"])
    if kind == "pairs":
        ace, pairs = _pair_list(case, seed)
        if case["n_rot"] * (N_TYPES + 1) * sum(p["n"] ** 3 for p in pairs) > 4e10:
            return None
        return [_exact_scan((p["n"],) * 3, "shape_ace", dict(p, ace=ace), case["peaks"]) for p in pairs]
    if kind == "predict":
        return _exact_predict(case, seed)
    return None
