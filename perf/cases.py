"""Performance cases of the D3 dispersion framework: the calls its users make.

The ranges follow the framework's benchmark workloads and tests: single
molecules from a few atoms to a few hundred, clusters of thousands of atoms,
periodic crystals and slabs, ragged batches of thousands of molecules and
batches of periodic frames.  Every case goes through a public entry point:

* ``model``     ``DispersionModel.update`` + ``get_dispersion`` on host arrays,
                the drop-in interface of a quantum chemistry or MD host
* ``batched``   ``BatchedDispersion``: many molecules per call, host arrays
* ``torch``     ``D3Batch``: the autograd wrapper in a float32 training step,
                mixed precision; float32 positions are widened for the call
                and the model's float32 gradients come back
* ``pairwise``  ``DispersionModel.get_pairwise_dispersion``
* ``hessian``   ``DispersionModel.get_hessian``

Geometries are jittered grids (minimum distances of 1.8 to 2 Bohr, the
densities of the benchmark workloads) with element frequencies of organic
molecules or mixed solids; all lengths are in Bohr.
"""
import math
import re
import sys
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "simple-dftd3_b200"))

from dftd3.interface import (  # noqa: E402
    BatchedDispersion, DispersionModel, ModifiedZeroDampingParam, OptimizedPowerDampingParam,
    RationalDampingParam, ZeroDampingParam)
from dftd3.torch_api import D3Batch  # noqa: E402

DISP2, DISP3, CN_CUT = 60.0, 40.0, 40.0      # the default real-space cutoffs
MIN_DISTANCE = 1.8

ORGANIC = ([1, 6, 7, 8, 9, 16, 17], [0.45, 0.28, 0.10, 0.10, 0.03, 0.02, 0.02])
SOLID = ([1, 6, 7, 8, 14, 13], [0.30, 0.25, 0.10, 0.15, 0.10, 0.10])

# PBE parameters of the rational and zero forms; the other families as in the tests
DAMPING = {
    "rational": dict(s6=1.0, s8=0.7875, a1=0.4289, a2=4.4407),
    "zero": dict(s6=1.0, s8=0.722, rs6=1.217, rs8=1.0),
    "mzero": dict(s6=1.0, s8=1.532981, rs6=1.338153, rs8=1.0, bet=0.013988),
    "optimizedpower": dict(s6=1.0, s8=0.43185, a1=0.575, a2=3.0, bet=8.0),
}
CLASSES = {"rational": RationalDampingParam, "zero": ZeroDampingParam, "mzero": ModifiedZeroDampingParam,
           "optimizedpower": OptimizedPowerDampingParam}


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # single point of a solvent-sized molecule inside an SCF host: the smallest call
        dict(name="molecule 12", kind="model", shape="molecule", n=12, damping="rational", atm=False, grad=True,
             graph=False),
        # geometry optimisation step of a drug-sized molecule with D3(BJ)-ATM
        dict(name="molecule 100 atm", kind="model", shape="molecule", n=100, damping="rational", atm=True,
             grad=True, graph=False),
        # MD steps of one mid-sized molecule, zero damping, captured sequence
        dict(name="molecule 251 graph", kind="model", shape="molecule", n=251, damping="zero", atm=False, grad=True,
             graph=True),
        # single-point energy of a two-dimensional periodic slab, another damping family, three-body term
        dict(name="slab 141 energy", kind="model", shape="slab", n=141, damping="optimizedpower", atm=True,
             grad=False, graph=False),
        # cell relaxation of a dense solid: the benchmark's headline system in the default precision
        dict(name="cell 2000", kind="model", shape="cell", n=2000, damping="rational", atm=False, grad=True,
             graph=False),
        # large aggregate with the three-body term, default precision
        dict(name="cluster 5000 atm", kind="model", shape="ball", n=5000, damping="rational", atm=True, grad=True,
             graph=False),
        # screening of a molecule library on host arrays
        dict(name="library 512 atm", kind="batched", nsys=512, nmin=8, nmax=256, damping="rational", atm=True,
             grad=True),
        # the headline system in the mixed form: energy and forces for a float32 model
        dict(name="cell 2000 mixed", kind="torch", shape="cell", nsys=1, nmin=2000, nmax=2000, atm=False,
             cell_grad=False),
        # training batch of molecules: energies and forces
        dict(name="batch 4096 mixed", kind="torch", shape="molecule", nsys=4096, nmin=8, nmax=256, atm=True,
             cell_grad=False),
        # training batch of periodic frames: forces, stress and damping parameters
        dict(name="frames 8 mixed", kind="torch", shape="frame", nsys=8, nmin=512, nmax=512, atm=True,
             cell_grad=True),
        # decomposition analysis of a molecule
        dict(name="pairwise 150", kind="pairwise", n=150, damping="rational", atm=True),
        # harmonic frequencies of a molecule
        dict(name="hessian 73", kind="hessian", n=73, damping="rational", atm=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "model", "model", "batched", "torch", "torch", "pairwise", "hessian"])
    if kind == "model":
        shape = rng.choice(["molecule", "slab", "cell", "ball"])
        atm = rng.random() < 0.5
        lo, hi = {"molecule": (5, 256), "slab": (40, 160 if atm else 600), "cell": (200, 400 if atm else 2000),
                  "ball": (257, 5000)}[shape]
        return dict(kind=kind, shape=shape, n=_log_int(rng, lo, hi), damping=rng.choice(sorted(DAMPING)), atm=atm,
                    grad=rng.random() < 0.75, graph=rng.random() < 0.3)
    if kind == "batched":
        return dict(kind=kind, nsys=_log_int(rng, 16, 1024), nmin=8, nmax=rng.randint(40, 256),
                    damping=rng.choice(["rational", "zero"]), atm=rng.random() < 0.7, grad=rng.random() < 0.75)
    if kind == "torch":
        shape = rng.choice(["molecule", "cell", "frame"])
        if shape == "molecule":
            return dict(kind=kind, shape=shape, nsys=_log_int(rng, 16, 4096), nmin=8, nmax=rng.randint(40, 256),
                        atm=rng.random() < 0.7, cell_grad=False)
        if shape == "cell":
            n = _log_int(rng, 300, 2000)
            return dict(kind=kind, shape=shape, nsys=1, nmin=n, nmax=n, atm=False, cell_grad=rng.random() < 0.5)
        n = rng.randint(300, 512)
        return dict(kind=kind, shape=shape, nsys=rng.randint(1, 8), nmin=n, nmax=n, atm=True,
                    cell_grad=rng.random() < 0.5)
    if kind == "pairwise":
        return dict(kind=kind, n=_log_int(rng, 12, 200), damping=rng.choice(sorted(DAMPING)), atm=rng.random() < 0.7)
    return dict(kind=kind, n=_log_int(rng, 8, 90), damping=rng.choice(["rational", "zero"]), atm=rng.random() < 0.7)


# ------------------------------------------------------------- geometries --

def _elements(rng, n, table):
    return rng.choice(np.asarray(table[0]), size=n, p=np.asarray(table[1]) / np.sum(table[1])).astype(np.int32)


def _grid(rng, n, edges, ball=False):
    """n points (fractions of the edges) of a jittered grid with at least n cells, at random cells or (ball) the
    ones nearest to the centre."""
    spacing = (np.prod(edges) / n) ** (1.0 / 3.0)
    m = np.maximum(1, np.round(np.asarray(edges) / spacing).astype(int))
    while np.prod(m) < n:
        m[np.argmax(np.asarray(edges) / m)] += 1
    cells = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)
    if ball:
        order = np.argsort(np.sum(((cells + 0.5) / m - 0.5) ** 2 * np.asarray(edges) ** 2, axis=1), kind="stable")
        pick = rng.permutation(order[:n])
    else:
        pick = rng.permutation(len(cells))[:n]
    step = np.asarray(edges) / m
    free = np.maximum(step - MIN_DISTANCE, 0.2) / np.asarray(edges)
    return (cells[pick] + 0.5) / m + rng.uniform(-0.5, 0.5, size=(n, 3)) * free


def _system(rng, shape, n):
    """(numbers, positions, lattice, periodic) of one system."""
    if shape == "molecule":
        side = (n / 0.010) ** (1.0 / 3.0)
        return _elements(rng, n, ORGANIC), _grid(rng, n, [side] * 3) * side, None, None
    if shape == "ball":
        side = (n / 0.012) ** (1.0 / 3.0) * (6.0 / math.pi) ** (1.0 / 3.0)
        grid = _grid(rng, int(math.ceil(n * 6.0 / math.pi)), [side] * 3, ball=True)
        near = np.argsort(np.sum((grid - 0.5) ** 2, axis=1), kind="stable")[:n]
        return _elements(rng, n, ORGANIC), rng.permutation(grid[near]) * side, None, None
    if shape == "slab":
        edge = (n / (0.02 * 12.0)) ** 0.5
        edges = [edge * rng.uniform(0.95, 1.05), edge * rng.uniform(0.95, 1.05), 12.0]
        pos = _grid(rng, n, edges) * np.asarray(edges)
        return _elements(rng, n, SOLID), pos, np.diag(edges[:2] + [30.0]), np.array([True, True, False])
    if shape == "frame":
        box = (n / 512.0) ** (1.0 / 3.0) * rng.uniform(28.0, 32.0)
        return _elements(rng, n, ORGANIC), _grid(rng, n, [box] * 3) * box, np.eye(3) * box, np.ones(3, dtype=bool)
    a, b, c = (n / 2000.0) ** (1.0 / 3.0) * rng.uniform(40.0, 45.0, size=3)
    al, be, ga = np.radians(rng.uniform(85.0, 95.0, size=3))
    cx, cy = c * np.cos(be), c * (np.cos(al) - np.cos(be) * np.cos(ga)) / np.sin(ga)
    lat = np.array([[a, 0.0, 0.0], [b * np.cos(ga), b * np.sin(ga), 0.0], [cx, cy, np.sqrt(c * c - cx * cx - cy * cy)]])
    return _elements(rng, n, SOLID), _grid(rng, n, [a, b, c]) @ lat, lat, np.ones(3, dtype=bool)


def _systems(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] in ("model", "pairwise", "hessian"):
        return [_system(rng, case.get("shape", "molecule"), case["n"])]
    if case["nmin"] == case["nmax"]:
        sizes = [case["nmin"]] * case["nsys"]
    else:
        # log-uniform over the range: the same sizes for every seed, in another order
        at = (np.arange(case["nsys"]) + 0.5) / case["nsys"]
        sizes = rng.permutation((case["nmin"] * ((case["nmax"] + 1) / case["nmin"]) ** at).astype(int))
    return [_system(rng, case.get("shape", "molecule"), int(n)) for n in sizes]


# ---------------------------------------------------------------- passes --

def prepare(case, seed):
    systems = _systems(case, seed)
    num, pos, lat, per = systems[0]
    kind = case["kind"]
    if kind == "torch":
        lats = None if lat is None else np.array([s[2] for s in systems])
        pers = None if lat is None else np.array([s[3] for s in systems])
        model = D3Batch([s[0] for s in systems], lattices=lats, periodic=pers, precision="mixed")
        p = DAMPING["rational"]
        x = torch.tensor(np.concatenate([s[1] for s in systems]), dtype=torch.float32, device="cuda",
                         requires_grad=True)
        values = [p["s6"], p["s8"], p["a1"], p["a2"], 1.0 if case["atm"] else 0.0]
        params = torch.tensor(values, dtype=torch.float64, device="cuda", requires_grad=case["cell_grad"])
        strain = torch.zeros((len(systems), 3, 3), dtype=torch.float32, device="cuda",
                             requires_grad=case["cell_grad"])
        return dict(kind=kind, model=model, x=x, params=params, strain=strain)
    param = CLASSES[case["damping"]](**DAMPING[case["damping"]], s9=1.0 if case["atm"] else 0.0)
    if kind == "batched":
        positions = [s[1] for s in systems]
        return dict(kind=kind, model=BatchedDispersion([s[0] for s in systems], positions), positions=positions,
                    param=param, grad=case["grad"])
    model = DispersionModel(num, pos, lat, per)
    if kind == "model":
        model.set_graph(case["graph"])
    return dict(kind=kind, model=model, positions=pos, param=param, grad=case.get("grad", False))


def run(state):
    kind, model = state["kind"], state["model"]
    if kind == "torch":
        x, strain = state["x"], state["strain"]
        wants = [x, strain, state["params"]] if strain.requires_grad else [x]
        energies = model(x.double(), state["params"], strain.double() if strain.requires_grad else None).float()
        grads = torch.autograd.grad(energies.sum(), wants)
        out = dict(energy=energies.detach(), gradient=grads[0])
        if strain.requires_grad:
            out.update(virial=grads[1], params=grads[2].float())
        return out
    if kind == "pairwise":
        return model.get_pairwise_dispersion(state["param"])
    if kind == "hessian":
        return model.get_hessian(state["param"])
    model.update(state["positions"])
    out = model.get_dispersion(state["param"], grad=state["grad"])
    if kind == "batched" and state["grad"]:
        out["gradient"] = np.concatenate(out["gradient"])
    return out


# ------------------------------------------------------------------- work --

# operations of one accepted term with all the derivatives a gradient call returns, and of the energy alone
PAIR_FLOPS, PAIR_ENERGY_FLOPS, CN_FLOPS = 65, 25, 40
TRIPLE_FLOPS, TRIPLE_ENERGY_FLOPS, TRIPLE_HESSIAN_FLOPS = 100, 40, 700


def _translations(lat, per, cutoff):
    if lat is None or not np.any(per):
        return np.zeros((1, 3))
    full = np.array(lat, dtype=float)
    vol = abs(np.linalg.det(full))
    rep = []
    for k in range(3):
        height = vol / np.linalg.norm(np.cross(full[(k + 1) % 3], full[(k + 2) % 3]))
        rep.append(int(math.ceil(cutoff / height)) if per[k] else 0)
    g = np.stack(np.meshgrid(*[np.arange(-r, r + 1) for r in rep], indexing="ij"), -1).reshape(-1, 3)
    return g @ full


def _terms(system, atm):
    """Estimated pair, CN and triple terms of one system (each counted once) from a sample of its atoms."""
    num, pos, lat, per = system
    n = len(num)
    if lat is None and n <= 256:
        return n * (n - 1) / 2, n * (n - 1) / 2, n * (n - 1) * (n - 2) / 6 if atm else 0.0
    rng = np.random.default_rng(0)
    sample = rng.permutation(n)[:8]
    trans = _translations(lat, per, DISP2)
    pairs = cns = triples = 0.0
    for i in sample:
        v = ((pos - pos[i])[:, None] + trans[None]).reshape(-1, 3)
        r2 = np.sum(v * v, axis=1)
        pairs += 0.5 * np.count_nonzero((r2 < DISP2 ** 2) & (r2 > 1e-9))
        near = v[(r2 < DISP3 ** 2) & (r2 > 1e-9)]
        cns += 0.5 * len(near)
        if atm:
            some = near[rng.permutation(len(near))[:400]]
            d2 = np.sum((some[:, None] - some[None]) ** 2, axis=-1)
            share = np.count_nonzero((d2 < DISP3 ** 2) & (d2 > 1e-9)) / max(d2.size, 1)
            triples += share * len(near) ** 2 / 6.0
    return tuple(t * n / len(sample) for t in (pairs, cns, triples))


def work(case):
    systems = _systems(case, 0)
    n = sum(len(s[0]) for s in systems)
    alike = case["kind"] == "torch" and case["nmin"] == case["nmax"]
    terms = [_terms(s, case["atm"]) for s in (systems[:1] if alike else systems)]
    pairs, cns, triples = (sum(t[k] for t in terms) * (len(systems) if alike else 1) for k in range(3))
    deriv = case["kind"] in ("torch", "hessian") or case.get("grad", False)
    flops = cns * (CN_FLOPS if deriv else 16) + pairs * (PAIR_FLOPS if deriv else PAIR_ENERGY_FLOPS)
    per_triple = TRIPLE_HESSIAN_FLOPS if case["kind"] == "hessian" else TRIPLE_FLOPS if deriv else TRIPLE_ENERGY_FLOPS
    flops += triples * per_triple
    word = 4 if case["kind"] == "torch" else 8
    size = 3 * word * n + 4 * n + word * len(systems)
    if case["kind"] == "pairwise":
        size += 2 * 8 * n * n
    elif case["kind"] == "hessian":
        size += 8 * 9 * n * n
        flops += 4 * 9 * n ** 3
    elif deriv:
        size += 3 * word * n + 9 * word * len(systems)
    return dict(bytes=size, flops=flops)


# ------------------------------------------------------------------ exact --
# The published D3 expressions in torch float64 with autograd derivatives.
# The element data (reference C6, radii) are read as text.

KCN, WF, ALP, REFS = 16.0, 4.0, 14.0, 7
EXACT_TRIPLES = 1.2e10     # largest three-body sum evaluated here
BOHR = 1.0 / 0.52917721090380


@lru_cache(maxsize=None)
def _data(name):
    text = (ROOT / "simple-dftd3_b200" / "csrc" / "d3_tables.c").read_text()
    body = re.search(r"\b%s\[\d+\]\s*=\s*\{(.*?)\};" % name, text, re.S).group(1)
    return np.array(body.replace("\n", " ").rstrip(" ,").split(","), dtype=float)


class _Elements:
    """Model data of the elements of a set of systems, on the device."""

    def __init__(self, numbers, device):
        self.zs = sorted(set(int(z) for z in numbers))
        z = np.array(self.zs)
        tri = np.array([[max(a, b) * (max(a, b) - 1) // 2 + min(a, b) - 1 for b in z] for a in z])
        put = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=device)  # noqa: E731
        nref = _data("d3_nref")[z - 1]
        self.valid = torch.tensor(np.arange(REFS)[None] < nref[:, None], device=device)
        self.refcn = put(_data("d3_refcn").reshape(-1, REFS)[z - 1])
        self.rcov = put(4.0 / 3.0 * BOHR * _data("d3_rcov_aa")[z - 1])
        r4r2 = np.sqrt(0.5 * _data("d3_r4_over_r2")[z - 1] * np.sqrt(z))
        self.rrij = put(3.0 * r4r2[:, None] * r4r2[None])
        self.rvdw = put(BOHR * _data("d3_vdwrad_aa")[tri])
        grid = _data("d3_c6ab").reshape(-1, REFS, REFS)
        c6 = np.zeros((len(z), REFS, len(z), REFS))
        for a in range(len(z)):
            for b in range(len(z)):
                m = grid[tri[a, b]]
                c6[a, :, b] = m.T if z[a] > z[b] else m
        ok = self.valid.cpu().numpy()
        c6 *= ok[:, :, None, None] * ok[None, None]
        self.c6 = put(c6.reshape(len(z) * REFS, -1))
        self.max_ref = torch.where(self.valid, self.refcn, torch.full_like(self.refcn, -9.0))

    def index(self, numbers):
        return np.searchsorted(self.zs, numbers)

    def c6_pairs(self, sp, cn, mask):
        """C6 matrices [..., n, n] from species indices and coordination numbers."""
        w = torch.exp(-WF * (cn[..., None] - self.refcn[sp]) ** 2) * self.valid[sp]
        norm = w.sum(-1, keepdim=True)
        best = self.max_ref[sp]
        last = (best == best.max(-1, keepdim=True).values).to(w.dtype)
        low = norm < 1e-300
        w = torch.where(low, last, w / torch.where(low, torch.ones_like(norm), norm)) * mask[..., None]
        hot = torch.nn.functional.one_hot(sp, len(self.zs)).to(w.dtype)
        g = (hot[..., None] * w[..., None, :]).flatten(-2)
        return g @ self.c6 @ g.transpose(-1, -2)


def _cn_term(r2, rc):
    return 1.0 / (1.0 + torch.exp(-KCN * (rc / torch.sqrt(r2) - 1.0)))


def _pair_term(kind, p, r2, rrij, rvdw):
    """-E/C6 of one pair distance for the damping families."""
    if kind == "rational":
        r0 = p["a1"] * torch.sqrt(rrij) + p["a2"]
        return p["s6"] / (r2 ** 3 + r0 ** 6) + p["s8"] * rrij / (r2 ** 4 + r0 ** 8)
    if kind == "optimizedpower":
        r0, r1 = p["a1"] * torch.sqrt(rrij) + p["a2"], torch.sqrt(r2)
        ab, rb = r0 ** p["bet"], r1 ** p["bet"]
        return p["s6"] * rb / (rb * r2 ** 3 + ab * r0 ** 6) + p["s8"] * rrij * rb / (rb * r2 ** 4 + ab * r0 ** 8)
    r1 = torch.sqrt(r2)
    if kind == "zero":
        t6, t8 = (r1 / (p["rs6"] * rvdw)) ** -ALP, (r1 / (p["rs8"] * rvdw)) ** -(ALP + 2.0)
    else:
        t6 = (r1 / (p["rs6"] * rvdw) + p["bet"] * rvdw) ** -ALP
        t8 = (r1 / (p["rs8"] * rvdw) + p["bet"] * rvdw) ** -(ALP + 2.0)
    return p["s6"] / (1.0 + 6.0 * t6) / r2 ** 3 + p["s8"] * rrij / (1.0 + 6.0 * t8) / r2 ** 4


def _triple_term(a, b, c, r0, c6):
    """Three-body energy of squared distances a, b, c, the product of the damping radii and of the C6."""
    w = a * b * c
    w15 = w * torch.sqrt(w)
    ang = 0.375 * (a + b - c) * (a - b + c) * (b + c - a) / (w15 * w) + 1.0 / w15
    return torch.sqrt(c6) * ang / (1.0 + 6.0 * (r0 / torch.sqrt(w)) ** ((ALP + 2.0) / 3.0))


def _molecules(el, sp, x, mask, kind, p, matrices=False):
    """Energies [B] of padded molecules [B, n] as a differentiable function of x [B, n, 3]; with matrices the pair
    and triple energies [B, n, n] of the decomposition instead."""
    n = sp.shape[1]
    both = (mask[:, :, None] & mask[:, None]) & ~torch.eye(n, dtype=torch.bool, device=x.device)
    v = x[:, None] - x[:, :, None]
    r2 = torch.where(both, (v * v).sum(-1), torch.ones((), dtype=x.dtype, device=x.device))
    pair = lambda t: t[sp[:, :, None], sp[:, None]]  # noqa: E731
    rc = el.rcov[sp][:, :, None] + el.rcov[sp][:, None]
    cn = (_cn_term(r2, rc) * (both & (r2 <= CN_CUT ** 2))).sum(-1)
    c6 = torch.where(both, el.c6_pairs(sp, cn, mask), torch.ones_like(r2))
    e2 = -0.5 * c6 * _pair_term(kind, p, r2, pair(el.rrij), pair(el.rvdw)) * (both & (r2 <= DISP2 ** 2))
    s9 = p["s9"]
    e3 = None
    if s9 != 0.0:
        near = both & (r2 <= DISP3 ** 2)
        r0 = 4.0 / 3.0 * pair(el.rvdw)
        ok = near[:, :, :, None] & near[:, :, None, :] & near[:, None]
        t = _triple_term(r2[:, :, :, None], r2[:, :, None, :], r2[:, None],
                         r0[:, :, :, None] * r0[:, :, None, :] * r0[:, None],
                         c6[:, :, :, None] * c6[:, :, None, :] * c6[:, None]) * ok
        e3 = s9 * t
    if matrices:
        # a sixth of every triple to each of its six ordered pairs
        return e2, torch.zeros_like(e2) if e3 is None else e3.sum(3) / 6.0
    return e2.sum((1, 2)) + (0.0 if e3 is None else e3.sum((1, 2, 3)) / 6.0)


def _extended(system, kind, p, device):
    """Energy of one large or periodic system and its derivatives with respect to positions, strain and p: the
    coordination numbers and C6 are separate variables whose derivatives are chained at the end."""
    num, pos, lat, per = system
    n = len(num)
    el = _Elements(num, device)
    sp = torch.tensor(el.index(num), device=device)
    x = torch.tensor(pos, dtype=torch.float64, device=device, requires_grad=True)
    eps = torch.zeros((3, 3), dtype=torch.float64, device=device, requires_grad=True)
    total = 0.0

    def vectors(rows, cols, trans):
        v = (x[cols][None, :, None] - x[rows][:, None, None]) + trans[None, None]
        v = v + v @ eps.T
        return v, (v * v).sum(-1)

    def images(cutoff):
        return torch.tensor(_translations(lat, per, cutoff), dtype=torch.float64, device=device)

    def chunks(trans):
        step = max(1, int(6e7 // (n * len(trans))))
        return [torch.arange(a, min(n, a + step), device=device) for a in range(0, n, step)]

    every = torch.arange(n, device=device)
    one = torch.ones((), dtype=torch.float64, device=device)
    t_cn, t_2 = images(CN_CUT), images(DISP2)

    def cn_rows(rows):
        _, r2 = vectors(rows, every, t_cn)
        ok = (r2 <= CN_CUT ** 2) & (r2 > 1e-12)
        rc = el.rcov[sp[rows]][:, None, None] + el.rcov[sp][None, :, None]
        return (_cn_term(torch.where(ok, r2, one), rc) * ok).sum((1, 2))

    with torch.no_grad():
        cn = torch.cat([cn_rows(r) for r in chunks(t_cn)])
    cn.requires_grad_(True)
    c6_graph = el.c6_pairs(sp, cn, torch.ones(n, dtype=torch.bool, device=device))
    c6 = c6_graph.detach().requires_grad_(True)
    for rows in chunks(t_2):
        _, r2 = vectors(rows, every, t_2)
        ok = (r2 <= DISP2 ** 2) & (r2 > 1e-12)
        term = _pair_term(kind, p, torch.where(ok, r2, one), el.rrij[sp[rows]][:, sp][..., None],
                          el.rvdw[sp[rows]][:, sp][..., None]) * ok
        e = (-0.5 * c6[rows] * term.sum(-1)).sum()
        e.backward()
        total += e.item()
    if bool(p["s9"] != 0.0):
        t_3 = images(DISP3)
        for i in range(n):
            # entries (j <= i, T) of the root, in the order of j; pairs with k <= j
            v, r2 = vectors(every[i:i + 1], every[:i + 1], t_3)
            v, r2 = v.reshape(-1, 3), r2.reshape(-1)
            pick = torch.nonzero((r2 <= DISP3 ** 2) & (r2 > 1e-12))[:, 0]
            if len(pick) < 2:
                continue
            v, r2, at = v[pick], r2[pick], pick // len(t_3)
            sq = ((v[:, None] - v[None]) ** 2).sum(-1)
            ok = (at[None] <= at[:, None]) & (sq <= DISP3 ** 2) & (sq > 1e-12)
            same = (at[:, None] == at[None]).double() + (at == i).double()[:, None] + (at == i).double()[None]
            scale = torch.where(same >= 3, one / 6.0, torch.where(same >= 1, one / 2.0, one)) * ok
            hot = torch.nn.functional.one_hot(at, i + 1).double()
            root = (hot @ c6[i, :i + 1])
            r0 = 4.0 / 3.0 * el.rvdw[sp[at], sp[i]]
            t = _triple_term(r2[:, None], r2[None], torch.where(ok, sq, one),
                             r0[:, None] * r0[None] * (4.0 / 3.0 * el.rvdw[sp[at]][:, sp[at]]),
                             root[:, None] * root[None] * (hot @ c6[:i + 1, :i + 1] @ hot.T))
            e = p["s9"] * (t * scale).sum()
            e.backward()
            total += e.item()
    c6_graph.backward(c6.grad)
    slope = cn.grad.detach()
    for rows in chunks(t_cn):
        (cn_rows(rows) * slope[rows]).sum().backward()
    return total, x.grad, eps.grad


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    systems = _systems(case, seed)
    kind = case.get("damping", "rational")
    if case["kind"] == "torch":     # the positions the float32 model holds
        systems = [(s[0], s[1].astype(np.float32).astype(float), s[2], s[3]) for s in systems]
    p = dict(DAMPING[kind], s9=1.0 if case["atm"] else 0.0)
    leaves = [torch.tensor(p[k], dtype=torch.float64, device=device, requires_grad=True)
              for k in ("s6", "s8", "a1", "a2", "s9")] if case.get("cell_grad") else None
    if leaves:
        p = dict(zip(("s6", "s8", "a1", "a2", "s9"), leaves))
    grad = case["kind"] == "torch" or case.get("grad", False)
    big = [s for s in systems if s[2] is not None or len(s[0]) > 256]
    if big and case["atm"] and _terms(big[0], True)[2] * len(big) > EXACT_TRIPLES:
        return None
    if big:
        got = [_extended(s, kind, p, device) for s in systems]
        energy = np.array([g[0] for g in got])
        gradient = torch.cat([g[1] for g in got]).cpu().numpy()
        virial = torch.stack([g[2] for g in got]).cpu().numpy()
    else:
        el = _Elements(np.concatenate([s[0] for s in systems]), device)
        order = sorted(range(len(systems)), key=lambda k: len(systems[k][0]))
        energy, gradient, virial = np.zeros(len(systems)), [None] * len(systems), np.zeros((len(systems), 3, 3))
        while order:
            n = len(systems[order[-1]][0])
            room = max(1, int(1.5e8 // n ** (3 if case["atm"] else 2)))
            group = [k for k in order[-room:] if len(systems[k][0]) >= n - 16]
            order = order[:-len(group)]
            sp = np.zeros((len(group), n), dtype=np.int64)
            pos, mask = np.zeros((len(group), n, 3)), np.zeros((len(group), n), dtype=bool)
            for b, k in enumerate(group):
                m = len(systems[k][0])
                sp[b, :m], pos[b, :m], mask[b, :m] = el.index(systems[k][0]), systems[k][1], True
            sp, mask = torch.tensor(sp, device=device), torch.tensor(mask, device=device)
            x = torch.tensor(pos, device=device, requires_grad=True)
            if case["kind"] == "pairwise":
                e2, e3 = _molecules(el, sp, x.detach(), mask, kind, p, matrices=True)
                return {"additive pairwise energy": e2[0].cpu().numpy(),
                        "non-additive pairwise energy": e3[0].cpu().numpy()}
            if case["kind"] == "hessian":
                f = lambda y: _molecules(el, sp, y.reshape(1, n, 3), mask, kind, p)[0]  # noqa: E731
                h = torch.autograd.functional.hessian(f, x.detach().reshape(-1))
                return {"energy": np.float64(f(x.detach()).item()), "hessian": h.cpu().numpy()}
            e = _molecules(el, sp, x, mask, kind, p)
            g, = torch.autograd.grad(e.sum(), [x])
            for b, k in enumerate(group):
                m = len(systems[k][0])
                energy[k], gradient[k] = e[b].item(), g[b, :m].cpu().numpy()
                virial[k] = (g[b, :m].T @ x[b, :m].detach()).cpu().numpy()
        gradient = np.concatenate(gradient)
    if case["kind"] == "torch":
        out = dict(energy=energy, gradient=gradient)
        if case["cell_grad"]:
            d = np.array([0.0 if t.grad is None else t.grad.item() for t in leaves])
            # without the three-body term its derivative with respect to s9 is not formed here
            out.update(virial=virial, params=d if case["atm"] else None)
        return out
    out = dict(energy=energy if case["kind"] == "batched" else energy[0])
    if grad:
        out.update(gradient=gradient, virial=virial if case["kind"] == "batched" else virial[0])
    return out
