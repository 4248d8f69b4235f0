"""Performance cases of the SOAP-GAP path: the calls a program makes, over the range of sizes, shapes and precisions
it makes them with.

A case is a dict of plain values:

  do        what is called: predict, md, autograd, features or training
  system    clusters (non-periodic random-walk molecules of 3..29 atoms), cells (sheared periodic cells of 32..512
            atoms), boxes (periodic cubes of `atoms` atoms) or bulk (one cube of `atoms` atoms at a lower density)
  count     structures in the batch
  precision fp32 (adjoint path) or fp64 (reference arithmetic)
  n, l      max_radial and max_angular; `rc`, `sigma` the cutoff and the Gaussian width
  species   atomic numbers, as text; `sparse` sparse points in all, `zeta` the kernel's power
  stress, forces   whether they are asked for

Every structure is new on each pass: positions, species and cells go in from host arrays (`StructureSet.set`, or the
positions alone in an MD step) and energies, forces and matrices come back to the host, except for `autograd`, which
keeps tensors on the device. The sparse points are environments of further structures of the same kind, as a fit
picks them. The weights have a mean as well as a spread: fitted energies are bound, all of one sign.
"""
import math

import numpy as np
import torch

import librascal_b200 as rb

ORGANIC = "1 6 7 8 9"


def listed():
    return [
        # one step of a small periodic MD run: latency and launches
        dict(name="md_box150", do="md", system="boxes", count=1, atoms=150, precision="fp32", n=8, l=6, rc=5.0,
             sigma=0.4, species="1 8", sparse=400, zeta=2, stress=True, forces=True),
        # one step of an ordinary MD run of an oxide
        dict(name="md_box2000", do="md", system="boxes", count=1, atoms=2000, precision="fp32", n=8, l=6, rc=5.0,
             sigma=0.4, species="8 14", sparse=2000, zeta=2, stress=True, forces=True),
        # a request of a hundred molecules
        dict(name="clusters100", do="predict", system="clusters", count=100, atoms=0, precision="fp32", n=8, l=6,
             rc=5.0, sigma=0.4, species=ORGANIC, sparse=1000, zeta=2, stress=False, forces=True),
        # the batch of the repository's benchmark
        dict(name="clusters10000", do="predict", system="clusters", count=10000, atoms=0, precision="fp32", n=8, l=6,
             rc=5.0, sigma=0.4, species=ORGANIC, sparse=4000, zeta=2, stress=False, forces=True),
        # one large box at a large basis
        dict(name="bulk100000", do="predict", system="bulk", count=1, atoms=100000, precision="fp32", n=12, l=9,
             rc=6.0, sigma=0.5, species="8 14", sparse=4000, zeta=2, stress=False, forces=True),
        # uneven periodic cells with their stress; an odd basis and the cubic kernel
        dict(name="cells97_n7_zeta3", do="predict", system="cells", count=97, atoms=0, precision="fp32", n=7, l=5,
             rc=5.0, sigma=0.4, species="1 6 7 8", sparse=1500, zeta=3, stress=True, forces=True),
        # screening: energies alone
        dict(name="energies3000", do="predict", system="clusters", count=3000, atoms=0, precision="fp32", n=6, l=5,
             rc=4.5, sigma=0.4, species="1 6 8", sparse=1111, zeta=2, stress=False, forces=False),
        # the energy inside a differentiable program: forward and backward on device tensors
        dict(name="autograd1000", do="autograd", system="clusters", count=1000, atoms=0, precision="fp32", n=8, l=6,
             rc=5.0, sigma=0.4, species=ORGANIC, sparse=2000, zeta=2, stress=False, forces=True),
        # the model class's default precision: one periodic box with stress
        dict(name="fp64_box64", do="predict", system="boxes", count=1, atoms=64, precision="fp64", n=6, l=4, rc=4.0,
             sigma=0.3, species="1 8", sparse=200, zeta=2, stress=True, forces=True),
        # the same precision on a batch of molecules
        dict(name="fp64_clusters300", do="predict", system="clusters", count=300, atoms=0, precision="fp64", n=8, l=6,
             rc=5.0, sigma=0.4, species=ORGANIC, sparse=1000, zeta=2, stress=False, forces=True),
        # descriptors alone, reference arithmetic, as input to other regressors
        dict(name="features_boxes16", do="features", system="boxes", count=16, atoms=64, precision="fp64", n=6, l=4,
             rc=4.0, sigma=0.3, species="1 8", sparse=0, zeta=2, stress=False, forces=False),
        # the kernel matrices of a fit: energy rows and gradient rows
        dict(name="training_clusters100", do="training", system="clusters", count=100, atoms=0, precision="fp64", n=8,
             l=6, rc=5.0, sigma=0.4, species=ORGANIC, sparse=500, zeta=2, stress=False, forces=True),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    case = dict(do=rng.choice(["md", "predict", "predict", "predict", "autograd", "features", "training"]),
                precision="fp32", stress=False, forces=True, count=1, atoms=0, zeta=rng.choice([1, 2, 2, 3]),
                rc=rng.choice([4.0, 5.0]), sigma=rng.choice([0.3, 0.4, 0.5]), n=rng.choice([5, 6, 7, 8]),
                l=rng.choice([3, 4, 5, 6]), species=rng.choice(["8 14", "1 8", "1 6 7 8", "1 6 8", ORGANIC]))
    if case["do"] in ("features", "training"):
        case["precision"] = "fp64"
    elif case["do"] == "predict":
        case["precision"] = rng.choice(["fp32", "fp32", "fp64"])
    slow = case["precision"] == "fp64"
    case["sparse"] = 0 if case["do"] == "features" else spread(100, 1000 if slow else 4000)
    if case["do"] == "md":
        case.update(system="boxes", atoms=spread(150, 2000), stress=rng.random() < 0.5)
        return case
    case["system"] = rng.choice(["clusters", "clusters", "cells"] if slow else ["clusters", "clusters", "cells", "bulk"])
    if case["system"] == "clusters":
        case["count"] = spread(11, 150) if case["do"] == "training" else spread(11, 300 if slow else 7000)
    elif case["system"] == "cells":
        case["count"] = spread(1, 3) if case["do"] == "training" else spread(1, 5 if slow else 150)
    else:
        case.update(atoms=spread(3000, 60000), rc=rng.choice([5.0, 6.0]), n=rng.choice([8, 9, 12]), l=rng.choice([6, 8, 9]),
                    species="8 14")
    if case["do"] == "predict":
        case["stress"] = case["system"] != "clusters" and rng.random() < 0.5
        case["forces"] = case["stress"] or rng.random() < 0.8
    return case


# ------------------------------------------------------------------ structures

def _species(case):
    return [int(z) for z in case["species"].split()]


def _fractions(case):
    """Share of each species: half hydrogen in molecules, two oxygen per silicon, else even."""
    sp = _species(case)
    if case["system"] == "clusters" and 1 in sp:
        return [0.5 if z == 1 else 0.5 / (len(sp) - 1) for z in sp]
    if sp == [8, 14]:
        return [2.0 / 3.0, 1.0 / 3.0]
    return [1.0 / len(sp)] * len(sp)


def _numbers(rng, atoms, species, share):
    """Species in their shares, dealt at random: every seed has the same number of each."""
    upto = np.round(np.cumsum(share) * atoms).astype(int)
    return rng.permutation(np.repeat(species, np.diff(np.concatenate([[0], upto])))).astype(np.int32)


def _clusters(rng, size, species, share):
    """Random-walk chains with bonds of 1.0..1.6 A and no two atoms nearer than 0.9 A, all chains grown together."""
    count = len(size)
    pos = np.zeros((count, 29, 3))
    for k in range(1, 29):
        todo, tries = np.flatnonzero(size > k), 0
        while len(todo):
            anchor = np.full(len(todo), k - 1) if tries < 20 else rng.integers(0, k, len(todo))
            v = rng.normal(size=(len(todo), 3))
            v *= (rng.uniform(1.0, 1.6, len(todo)) / np.linalg.norm(v, axis=1))[:, None]
            p = pos[todo, anchor] + v
            fits = ((pos[todo, :k] - p[:, None]) ** 2).sum(-1).min(1) >= 0.81
            pos[todo[fits], k] = p[fits]
            todo, tries = todo[~fits], tries + 1
    inside = np.arange(29)[None, :] < size[:, None]
    low = np.where(inside[..., None], pos, np.inf).min(1)
    high = np.where(inside[..., None], pos, -np.inf).max(1)
    side = np.maximum((high - low) * 1.05, 1.0)
    pos = pos + (0.5 * side - 0.5 * (high + low))[:, None]
    return dict(atom_offsets=np.concatenate([[0], np.cumsum(size)]).astype(np.int64), positions=pos[inside],
                numbers=_numbers(rng, int(size.sum()), species, share), cells=side[:, :, None] * np.eye(3),
                pbc=np.zeros((count, 3), np.int32))


def _periodic(rng, sizes, density, near, shear, species, share):
    """Atoms on random sites of a grid, moved by as much as keeps them about `near` apart."""
    pos, cells = [], []
    for m in sizes:
        a = np.eye(3) + (1 - np.eye(3)) * rng.uniform(-shear, shear, (3, 3))
        cell = a * (m / density / abs(np.linalg.det(a))) ** (1 / 3)
        g = math.ceil(round(m ** (1 / 3), 9))
        site = rng.permutation(g ** 3)[:m]
        frac = np.stack([site // (g * g), site // g % g, site % g], 1) + 0.5
        step = (m / density) ** (1 / 3) / g
        frac = (frac + rng.uniform(-0.5, 0.5, (m, 3)) * max(0.1, 1 - near / step)) / g
        pos.append(frac @ cell)
        cells.append(cell)
    return dict(atom_offsets=np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64), positions=np.concatenate(pos),
                numbers=_numbers(rng, int(np.sum(sizes)), species, share), cells=np.array(cells),
                pbc=np.ones((len(sizes), 3), np.int32))


def _batch(case, rng, atoms=None):
    """The structures of a case, or (with `atoms`) about that many atoms of the same kind. How many atoms each has
    goes by the case alone."""
    sp, share, kind = _species(case), _fractions(case), case["system"]
    if kind == "clusters":
        count = case["count"] if atoms is None else -(-atoms // 15)
        return _clusters(rng, np.random.default_rng(count).integers(3, 30, count), sp, share)
    if kind == "cells":
        count = case["count"] if atoms is None else max(4, -(-atoms // 250))
        return _periodic(rng, np.random.default_rng(count).integers(32, 513, count), 0.1, 0.9, 0.1, sp, share)
    sizes = [case["atoms"]] * case["count"] if atoms is None else [max(atoms, 600)]
    return _periodic(rng, sizes, 0.05 if kind == "bulk" else 0.064, 1.2 if kind == "bulk" else 0.9, 0.0, sp, share)


def _selection(case, seed):
    """The structures the sparse points come from, the chosen atoms (in batch order) and the weights (in the
    columns' order: species ascending)."""
    rng = np.random.default_rng([seed, 2])
    batch = _batch(case, rng, int(1.6 * case["sparse"]) + 200)
    chosen = []
    for z, f in zip(_species(case), _fractions(case)):
        ids = np.flatnonzero(batch["numbers"] == z)
        chosen.append(rng.permutation(ids)[:max(1, int(round(case["sparse"] * f)))])
    chosen = np.sort(np.concatenate(chosen))
    weights = rng.normal(size=len(chosen)) - 1.0
    return batch, chosen, weights


# ------------------------------------------------------------------ the calls

def prepare(case, seed):
    batch = _batch(case, np.random.default_rng([seed, 1]))
    hypers = dict(interaction_cutoff=case["rc"], cutoff_smooth_width=0.5, max_radial=case["n"], max_angular=case["l"],
                  gaussian_sigma_type="Constant", gaussian_sigma_constant=case["sigma"], normalize=True)
    state = dict(case=case, soap=rb.SphericalInvariants(**hypers), batch=batch, structures=rb.StructureSet(batch))
    if case["sparse"]:
        from_, chosen, weights = _selection(case, seed)
        off = from_["atom_offsets"]
        managers = state["soap"].transform(rb.AtomsList(rb.StructureSet(from_)))
        points = rb.SparsePoints(state["soap"])
        points.extend(managers, [chosen[(chosen >= a) & (chosen < b)] - a for a, b in zip(off[:-1], off[1:])])
        state["points"] = points
        if case["do"] == "training":
            state["kernel"] = rb.Kernel(state["soap"], zeta=case["zeta"])
            state["kernel"]._model(points)
        else:
            state["model"] = rb.GAPModel(state["soap"], points, weights, case["zeta"])
    if case["do"] == "autograd":
        rng = np.random.default_rng([seed, 3])
        state["positions"] = torch.tensor(batch["positions"], dtype=torch.float32, device="cuda", requires_grad=True)
        state["upstream"] = torch.tensor(rng.uniform(0.5, 1.5, case["count"]), dtype=torch.float32, device="cuda")
    return state


def _as_computed(case, values):
    """The FP32 path hands its 32-bit results over in FP64 arrays: a program keeps what they hold."""
    return [v.astype(np.float32) for v in values if v is not None] if case["precision"] == "fp32" else \
        [v for v in values if v is not None]


def run(state):
    case, structures = state["case"], state["structures"]
    if case["do"] == "md":
        return _as_computed(case, state["model"].md_step(structures, state["batch"]["positions"], stress=case["stress"]))
    if case["do"] == "autograd":
        energies = rb.gap_energy(state["positions"], state["model"], structures)
        gradient, = torch.autograd.grad(energies, state["positions"], state["upstream"])
        return [energies.detach(), gradient]
    structures.set(state["batch"])
    if case["do"] == "predict":
        if case["stress"]:
            return _as_computed(case, state["model"].predict_stress(structures, case["precision"]))
        return _as_computed(case, state["model"].predict(structures, case["precision"], forces=case["forces"]))
    managers = state["soap"].transform(rb.AtomsList(structures))
    if case["do"] == "features":
        return [managers.get_features(state["soap"])]
    return [state["kernel"](managers, state["points"]), state["kernel"](managers, state["points"], grad=(True, False))]


def work(case):
    """Inputs and outputs once; the multiplications of the expansion, of the power spectrum and of the kernel (and, for
    forces, of their adjoints), with every distinct feature counted once."""
    atoms = 16 * case["count"] if case["system"] == "clusters" else 272 * case["count"] if case["system"] == "cells" \
        else case["atoms"] * case["count"]
    density = 0.05 if case["system"] == "bulk" else 0.1 if case["system"] == "cells" else 0.064
    pairs = 14 * atoms if case["system"] == "clusters" else atoms * density * 4 / 3 * math.pi * case["rc"] ** 3
    sn, lm = len(_species(case)) * case["n"], (case["l"] + 1) ** 2
    features = sn * (sn + 1) // 2 * (case["l"] + 1)
    same = sum(f * f for f in _fractions(case))
    expand, square = 2 * pairs * case["n"] * lm, atoms * sn * (sn + 1) * lm
    kernel = 2 * atoms * same * case["sparse"] * features
    real = 4 if case["precision"] == "fp32" else 8
    data = atoms * (24 + 4) + case["sparse"] * features * real
    if case["do"] == "features":
        return dict(bytes=data + atoms * 8 * _columns(case), flops=expand + square)
    if case["do"] == "training":
        return dict(bytes=data + 8 * case["sparse"] * (case["count"] + 3 * atoms),
                    flops=expand + square + kernel + 3 * 2 * pairs * same * case["sparse"] * case["n"] * lm)
    if case["forces"]:
        return dict(bytes=data + 24 * atoms, flops=4 * expand + 3 * square + 2 * kernel)
    return dict(bytes=data, flops=expand + square + kernel)


def _columns(case):
    s = len(_species(case))
    return s * (s + 1) // 2 * case["n"] ** 2 * (case["l"] + 1)


# ------------------------------------------------------------------ the same in 64 bits, plain numpy and torch

def _radial_fit(case):
    """Chebyshev coefficients over r in [0, rc] of the orthonormalised GTO radial integrals, [terms][n][l+1], and the
    centre's own integral [n]."""
    n, l1, rc, terms = case["n"], case["l"] + 1, case["rc"], 96
    c = 0.5 / case["sigma"] ** 2
    i = np.arange(n)
    width = np.maximum(np.sqrt(i), 1.0) * rc / n
    d = 0.5 / width ** 2
    gamma = np.vectorize(math.gamma)
    norm = 0.25 * np.sqrt(2.0 / (gamma(1.5 + i) * width ** (3 + 2 * i)))
    a, b = i[:, None], i[None, :]
    overlap = (d[:, None] + d[None, :]) ** (-0.5 * (3 + a + b)) / (width[:, None] ** a * width[None, :] ** b) \
        * gamma(0.5 * (3 + a + b)) / ((width[:, None] * width[None, :]) ** 1.5 * np.sqrt(gamma(1.5 + a) * gamma(1.5 + b)))
    value, vector = np.linalg.eigh(overlap)
    ortho = norm[:, None] * ((vector / np.sqrt(value)) @ vector.T)
    theta = math.pi * (np.arange(terms) + 0.5) / terms
    r = 0.5 * rc * (1 + np.cos(theta))[:, None, None]
    nn, ll = i[None, :, None], np.arange(l1)[None, None, :]
    p, q = 0.5 * (nn + ll + 3), ll + 1.5
    z = c * c * r * r / (c + d[None, :, None])
    term = np.ones_like(z * p * q)
    total = term.copy()
    for k in range(600):
        term = term * (p + k) / (q + k) * z / (k + 1)
        total += term
    raw = (c + d[None, :, None]) ** (-p) * (c * r) ** ll * gamma(p) / gamma(q) * total * np.exp(-c * r * r)
    values = np.einsum("ki,rkl->ril", ortho, raw)
    fit = np.einsum("tr,ril->til", np.cos(np.arange(terms)[:, None] * theta[None, :]), values) * 2 / terms
    fit[0] *= 0.5
    own = ortho.T @ (gamma(0.5 * (3 + i)) / math.gamma(1.5) * (c + d) ** (-0.5 * (3 + i)))
    return fit, own / math.sqrt(4 * math.pi)


def _spline(case):
    """The natural cubic spline through those integrals that the representation is defined by, as fine as its accuracy
    of 1e-8 asks: grid, values and second derivatives times h^2/6 [points][n (l+1)], and the centre's integral."""
    fit, own = _radial_fit(case)
    fit = fit.reshape(len(fit), -1)

    def integrals(r):
        return np.cos(np.arange(len(fit))[None, :] * np.arccos(np.clip(2 * r / case["rc"] - 1, -1, 1))[:, None]) @ fit

    points, low, high = 64, 1e-5, case["rc"]
    while True:
        grid = np.linspace(low, high, points)
        y, h = integrals(grid), grid[1] - grid[0]
        bend, sweep = np.zeros(points), np.zeros_like(y)
        for k in range(1, points - 1):
            p = 0.5 * bend[k - 1] + 2
            bend[k] = -0.5 / p
            sweep[k] = (3 * (y[k + 1] - 2 * y[k] + y[k - 1]) / h ** 2 - 0.5 * sweep[k - 1]) / p
        second = np.zeros_like(y)
        for k in range(points - 2, 0, -1):
            second[k] = bend[k] * second[k + 1] + sweep[k]
        second *= h * h / 6
        half = (high - low) / (2 * (points - 1))
        middle = np.linspace(low + half, high - half, points - 1)
        k, a = _interval(torch.tensor(middle), torch.tensor(grid))
        k, a = k.numpy(), a.numpy()[:, None]
        b = 1 - a
        value = a * (y[k] + (a * a - 1) * second[k]) + b * (y[k + 1] + (b * b - 1) * second[k + 1])
        if np.abs(value - integrals(middle)).mean() < 1e-8 or points >= 100000:
            return grid, y, second, own
        points *= 2


def _interval(r, grid):
    """The spline's interval of each r, by the grid search it is defined with, and the weight of its left end."""
    k = ((r - grid[0]) * (len(grid) / (grid[-1] - grid[0]))).long() - 1
    k = k.clamp(0, len(grid) - 2)
    return k, (grid[k + 1] - r) / (grid[1] - grid[0])


def _pairs(batch, rc, device):
    """(i, j, shift vector) of all pairs up to rc, the self pairs left out, sorted by i."""
    off, found = batch["atom_offsets"], []
    pos = torch.tensor(batch["positions"], device=device)
    if not batch["pbc"].any():
        index = torch.full((len(off) - 1, 29), -1, dtype=torch.int64, device=device)
        where = np.concatenate([np.arange(k) for k in np.diff(off)])
        owner = np.repeat(np.arange(len(off) - 1), np.diff(off))
        index[torch.tensor(owner, device=device), torch.tensor(where, device=device)] = torch.arange(len(pos), device=device)
        s, a, b = torch.nonzero((index[:, :, None] >= 0) & (index[:, None, :] >= 0), as_tuple=True)
        i, j = index[s, a], index[s, b]
        near = (i != j) & ((pos[i] - pos[j]).square().sum(1) <= rc * rc)
        return i[near], j[near], torch.zeros((int(near.sum()), 3), dtype=torch.float64, device=device)
    for s in range(len(off) - 1):
        cell = torch.tensor(batch["cells"][s], device=device)
        p = pos[off[s]:off[s + 1]]
        height = 1 / torch.linalg.inv(cell).norm(dim=0)
        image = bool((height > 2 * rc).all())  # then one image of each pair at most is near
        reach = [0 if image else int(math.ceil(rc / h)) for h in height.tolist()]
        shifts = torch.cartesian_prod(*[torch.arange(-k, k + 1, device=device, dtype=torch.float64) for k in reach]).reshape(-1, 3)
        rows = max(1, 40_000_000 // len(p))
        for a in range(0, len(p), rows):
            for shift in shifts:
                diff = p[None] - p[a:a + rows, None]
                if image:
                    turn = -torch.round(diff @ torch.linalg.inv(cell))
                    diff = diff + turn @ cell
                else:
                    diff = diff + shift @ cell
                d2 = diff.square().sum(2)
                i, j = torch.nonzero((d2 <= rc * rc) & (d2 > 1e-12), as_tuple=True)
                vector = turn[i, j] @ cell if image else (shift @ cell).expand(len(i), 3)
                found.append((i + a + int(off[s]), j + int(off[s]), vector))
    i, j, v = (torch.cat(x) for x in zip(*found))
    order = torch.argsort(i, stable=True)
    return i[order], j[order], v[order]


def _harmonics(u, l_max):
    """Orthonormal real spherical harmonics of unit vectors, [pairs][(l+1)^2], as polynomials of x, y and z."""
    x, y, z = u.unbind(1)
    out = [None] * (l_max + 1) ** 2
    cos, sin = torch.ones_like(x), torch.zeros_like(x)
    for m in range(l_max + 1):
        last, leg = torch.zeros_like(z), torch.full_like(z, float(np.prod(np.arange(1, 2 * m, 2, dtype=float))))
        for l in range(m, l_max + 1):
            if l > m:
                last, leg = leg, ((2 * l - 1) * z * leg - (l + m - 1) * last) / (l - m)
            f = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m) * (2 if m else 1))
            out[l * l + l + m] = f * leg * cos
            if m:
                out[l * l + l - m] = f * leg * sin
        cos, sin = x * cos - y * sin, x * sin + y * cos
    return torch.stack(out, 1)


class _Soap:
    """Normalised power spectra in the reference's dense order, differentiable in the positions."""

    def __init__(self, case, batch, device):
        self.case, self.device = case, device
        self.grid, self.y, self.second, self.own = (torch.tensor(v, device=device) for v in _spline(case))
        sp, n = _species(case), case["n"]
        self.sort = torch.tensor(np.searchsorted(sp, batch["numbers"]), device=device)
        self.i, self.j, self.shift = _pairs(batch, case["rc"], device)
        self.first = torch.searchsorted(self.i, torch.arange(len(batch["numbers"]) + 1, device=device)).tolist()
        s = len(sp)
        columns, scale = [], []
        for a in range(s):
            for b in range(a, s):
                k = (np.arange(a * n, a * n + n)[:, None] * (s * n) + np.arange(b * n, b * n + n)[None]).reshape(-1)
                columns.append(k)
                scale.append(np.full(len(k), 1.0 if a == b else math.sqrt(2)))
        self.columns = torch.tensor(np.concatenate(columns), device=device)
        self.scale = torch.tensor(np.concatenate(scale), device=device)

    def rows(self, pos, c0, c1):
        """Features of the centres c0..c1 and their pairs' vectors."""
        case, p = self.case, slice(self.first[c0], self.first[c1])
        n, l1, s = case["n"], case["l"] + 1, len(_species(case))
        i, j = self.i[p], self.j[p]
        vector = pos[j] - pos[i] + self.shift[p]
        r = vector.norm(dim=1)
        k, a = _interval(r, self.grid)
        a = a[:, None]
        b = 1 - a
        radial = a * (self.y[k] + (a * a - 1) * self.second[k]) + b * (self.y[k + 1] + (b * b - 1) * self.second[k + 1])
        fc = torch.where(r <= case["rc"] - 0.5, 1.0, 0.5 * (1 + torch.cos(math.pi * (r - case["rc"] + 0.5) / 0.5)))
        radial = radial.reshape(-1, n, l1) * fc[:, None, None]
        angular = _harmonics(vector / r[:, None], l1 - 1)
        degree = torch.tensor([l for l in range(l1) for _ in range(2 * l + 1)], device=self.device)
        density = radial[:, :, degree] * angular[:, None, :]
        c = torch.zeros(((c1 - c0) * s, n, l1 * l1), dtype=torch.float64, device=self.device)
        c = c.index_add(0, (i - c0) * s + self.sort[j], density)
        centre = torch.zeros_like(c)
        centre[torch.arange(c1 - c0, device=self.device) * s + self.sort[c0:c1], :, 0] = self.own
        c = (c + centre).reshape(c1 - c0, s * n, l1 * l1)
        gram = [torch.einsum("cam,cbm->cab", b, b) / math.sqrt(2 * l + 1)
                for l, b in ((l, c[:, :, l * l:(l + 1) ** 2]) for l in range(l1))]
        f = torch.stack(gram, 3).reshape(c1 - c0, (s * n) ** 2, l1)[:, self.columns] * self.scale[None, :, None]
        f = f.reshape(c1 - c0, -1)
        return f / f.norm(dim=1, keepdim=True), vector

    def chunks(self, most=400_000_000):
        """Ranges of centres whose pair densities, and whose Gram matrices, stay below `most` values."""
        per = self.case["n"] * (self.case["l"] + 1) ** 2
        full = (len(_species(self.case)) * self.case["n"]) ** 2 * (self.case["l"] + 1)
        c0, total = 0, len(self.first) - 1
        while c0 < total:
            c1 = c0 + 1
            while c1 < total and (self.first[c1 + 1] - self.first[c0]) * per + (c1 + 1 - c0) * full < most:
                c1 += 1
            yield c0, c1
            c0 = c1


def exact(case, seed):
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    batch = _batch(case, np.random.default_rng([seed, 1]))
    if case["do"] == "autograd":
        batch["positions"] = batch["positions"].astype(np.float32).astype(float)
    soap = _Soap(case, batch, device)
    pos = torch.tensor(batch["positions"], device=device, requires_grad=True)
    if case["do"] == "features":
        with torch.no_grad():
            return [torch.cat([soap.rows(pos, *c)[0] for c in soap.chunks()])]
    from_, chosen, weights = _selection(case, seed)
    order = chosen[np.argsort(from_["numbers"][chosen], kind="stable")]
    species = np.searchsorted(_species(case), from_["numbers"][order])
    with torch.no_grad():
        other, at = _Soap(case, from_, device), torch.tensor(from_["positions"], device=device)
        points = torch.cat([other.rows(at, *c)[0] for c in other.chunks()])[torch.tensor(order, device=device)]
    weights = torch.tensor(weights, device=device)
    owner = torch.tensor(np.repeat(np.arange(len(batch["cells"])), np.diff(batch["atom_offsets"])), device=device)
    upstream = torch.ones(len(batch["cells"]), dtype=torch.float64, device=device)
    if case["do"] == "autograd":
        upstream = torch.tensor(np.random.default_rng([seed, 3]).uniform(0.5, 1.5, case["count"]).astype(np.float32).astype(float),
                                device=device)

    def kernels(x, c0, c1):
        for s in range(len(_species(case))):
            rows = torch.nonzero(soap.sort[c0:c1] == s)[:, 0]
            cols = torch.tensor(np.flatnonzero(species == s), device=device)
            if len(rows) and len(cols):
                yield rows, cols, (x[rows] @ points[cols].T) ** case["zeta"]

    if case["do"] == "training":
        energy = torch.zeros((len(batch["cells"]), len(points)), dtype=torch.float64, device=device)
        gradient = torch.zeros((pos.numel(), len(points)), dtype=torch.float64, device=device)
        for c0, c1 in soap.chunks(100_000_000):
            x, _ = soap.rows(pos, c0, c1)
            for rows, cols, k in kernels(x, c0, c1):
                with torch.no_grad():
                    part = torch.zeros((len(batch["cells"]), len(cols)), dtype=torch.float64, device=device)
                    energy[:, cols] += part.index_add(0, owner[c0 + rows], k)
                total = k.sum(0)
                for m, col in enumerate(cols.tolist()):
                    gradient[:, col] += torch.autograd.grad(total[m], pos, retain_graph=True)[0].reshape(-1)
        return [energy, gradient]
    energy = torch.zeros(len(batch["cells"]), dtype=torch.float64, device=device)
    gradient = torch.zeros_like(pos)
    virial = torch.zeros((len(batch["cells"]), 6), dtype=torch.float64, device=device)
    for c0, c1 in soap.chunks():
        x, vector = soap.rows(pos, c0, c1)
        e = torch.zeros(c1 - c0, dtype=torch.float64, device=device)
        for rows, cols, k in kernels(x, c0, c1):
            e = e.index_add(0, rows, k @ weights[cols])
        energy.index_add_(0, owner[c0:c1], e.detach())
        if case["forces"]:
            g, pull = torch.autograd.grad((e * upstream[owner[c0:c1]]).sum(), (pos, vector))
            gradient += g
            r, t = -vector.detach(), pull
            terms = torch.stack([r[:, 0] * t[:, 0], r[:, 1] * t[:, 1], r[:, 2] * t[:, 2], r[:, 1] * t[:, 2], r[:, 2] * t[:, 0],
                                 r[:, 0] * t[:, 1]], 1)
            virial.index_add_(0, owner[soap.i[soap.first[c0]:soap.first[c1]]], terms)
    if case["do"] == "autograd":
        return [energy, gradient]
    volume = torch.tensor(np.abs(np.linalg.det(batch["cells"])), device=device)
    return [energy] + [-gradient] * case["forces"] + [virial / volume[:, None]] * case["stress"]
