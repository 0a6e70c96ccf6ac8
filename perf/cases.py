"""Cases by which the speed of the 2-body + 3-body path is measured.

Every case is work that a program using this library gives it through its
public entry points: force calls of periodic boxes and clusters (FP64 and
mixed precision, host and device arrays, energies alone or with gradients and
virial), batches of path-integral beads and clusters, and fits of the linear
coefficients through torch autograd.  Sizes are those of the benchmark and the
tests of this repository, or lie between and beyond them.

``exact`` evaluates the same model in plain torch, in 64 bits, from the model
constants alone (sites, variables, switch radii, term tables, coefficients):
n-mers by comparing all first-atom distances, polynomials as one matrix
product over half-monomials, gradients by torch autograd.
"""
import gzip
import os

import numpy as np
import torch

import mbx_b200
from mbx_b200 import batch, capi, specs, system, torch_ops, workloads

CUT2, CUT3 = 9.0, 7.0
DENSITY = 2048 / 39.44 ** 3          # molecules / A^3 of the water boxes
DATA = os.path.join(os.path.dirname(os.path.abspath(mbx_b200.__file__)), "data")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a small gas-phase cluster in a geometry optimisation: host arrays,
        # both terms in one call; latency and launches count
        dict(name="cluster_8", kind="system", what="cluster", n=8, mixed=False, grads=True, api="host"),
        # Monte Carlo moves of a small periodic box: energies alone
        dict(name="water_256_energy", kind="system", what="water", n=256, mixed=False, grads=False, api="device"),
        # molecular dynamics of the small box of the tests, arrays on the device
        dict(name="water_256", kind="system", what="water", n=256, mixed=False, grads=True, api="device"),
        # the benchmark's box, both precisions
        dict(name="water_2048", kind="system", what="water", n=2048, mixed=False, grads=True, api="device"),
        dict(name="water_2048_mixed", kind="system", what="water", n=2048, mixed=True, grads=True, api="device"),
        # a large box through the drop-in interface: the two terms called one
        # after the other with host arrays, as the reference's callers do
        dict(name="water_6859_host", kind="system", what="water", n=6859, mixed=False, grads=True, api="terms"),
        # path-integral beads and clusters in one call, mixed precision
        dict(name="beads_batch_mixed", kind="batch", beads=8, n=2048, clusters=16, nmax=256, mixed=True),
        # the benchmark's 1 M salt solution
        dict(name="nacl_2048", kind="system", what="na+,cl-", n=2048, ions=64, mixed=False, grads=True, api="device"),
        # the methane-water box of the tests
        dict(name="methane_water_570", kind="system", what="methane", n=570, mixed=False, grads=True, api="device"),
        # carbon dioxide in water, for a caller that keeps its own atom order
        # on the device (i-PI, LAMMPS)
        dict(name="co2_water_700_real", kind="system", what="co2", n=700, ions=100, mixed=False, grads=True,
             api="real"),
        # one step of a fit of the linear coefficients: energies of gas-phase
        # n-mers, gradients of the loss by coefficients and coordinates
        dict(name="refit_dimers_20000", kind="refit", evaluator="mbpol2b", n=20000, mixed=False),
        dict(name="refit_trimers_20000", kind="refit", evaluator="mbpol3b", n=20000, mixed=False),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["cluster", "water", "water", "salt", "methane", "co2", "batch", "refit", "refit"])
    if kind == "cluster":
        return dict(kind="system", what="cluster", n=_log(rng, 4, 400), mixed=rng.random() < 0.3,
                    grads=rng.random() < 0.8, api=rng.choice(["host", "terms", "device"]))
    if kind == "water":
        return dict(kind="system", what="water", n=_log(rng, 220, 6000), mixed=rng.random() < 0.4,
                    grads=rng.random() < 0.8, api=rng.choice(["host", "terms", "device", "real"]))
    if kind == "salt":
        n = _log(rng, 700, 2000)
        pair = rng.choice(["li+,cl-", "na+,cl-", "k+,cl-", "rb+,br-", "cs+,i-", "na+,f-", "k+,br-"])
        return dict(kind="system", what=pair, n=n, ions=2 * rng.randint(2, n // 64), mixed=rng.random() < 0.3,
                    grads=rng.random() < 0.8, api=rng.choice(["host", "device"]))
    if kind == "methane":
        return dict(kind="system", what="methane", n=rng.randint(545, 600), mixed=rng.random() < 0.3,
                    grads=rng.random() < 0.8, api=rng.choice(["host", "terms", "device", "real"]))
    if kind == "co2":
        n = _log(rng, 400, 1200)
        return dict(kind="system", what="co2", n=n, ions=rng.randint(1, n // 7), mixed=False,
                    grads=rng.random() < 0.8, api=rng.choice(["host", "device", "real"]))
    if kind == "batch":
        return dict(kind="batch", beads=rng.randint(2, 8), n=_log(rng, 256, 2048), clusters=rng.randint(0, 12),
                    nmax=_log(rng, 12, 256), mixed=rng.random() < 0.7)
    return dict(kind="refit", evaluator=rng.choice(["mbpol2b", "mbpol3b", "ch4h2o2b", "ch4h2o3b"]),
                n=_log(rng, 50, 16000), mixed=False)


# ------------------------------------------------------------------ inputs
def _lattice(n):
    """Lattice of the repository's water boxes for n molecules: (sites per edge, box edge)."""
    side = int(np.ceil((n * 2744 / 2048) ** (1.0 / 3.0) - 1e-9))
    return side, float((n / DENSITY) ** (1.0 / 3.0))


def _molecules(case, seed):
    """(ids, input-order coordinates, box or None).  The types come in
    ascending number, so that the library's internal order is the input's."""
    n, what = case["n"], case["what"]
    if what == "cluster":
        ids, xyz = workloads.water_cluster(n, seed=seed)
        return ids, xyz, None
    if what == "methane":
        k = n // 10
        edge = (n / 570) ** (1.0 / 3.0)
        return workloads.methane_water_box(k, n - k, (24.6 * edge, 24.6 * edge, 31.0 * edge), seed=seed)
    side, edge = _lattice(n)
    if what == "water":
        return workloads.water_box(side, n, edge, seed=seed)
    if what == "co2":
        ids = ["co2"] * case["ions"] + ["h2o"] * (n - case["ions"])
    else:
        a, b = what.split(",")
        h = case["ions"] // 2
        ids = [a] * h + [b] * h + ["h2o"] * (n - 2 * h)
    return workloads.molecule_box(ids, side, edge, seed=seed)


def _configurations(case, seed):
    side, edge = _lattice(case["n"])
    ids, xyz, box = workloads.water_box(side, case["n"], edge, seed=seed)
    out = [(ids, b, box) for b in workloads.beads(xyz, case["beads"], 0.05, seed + 1)]
    # clusters of sizes spread over 8 .. nmax, the same ones for every seed
    for k, m in enumerate(np.linspace(8, case["nmax"], case["clusters"])):
        cid, cxyz = workloads.water_cluster(int(m), seed=seed + 1000 + k)
        out.append((cid, cxyz, None))
    return out


def _nmers(case, seed):
    """[n, 3 * atoms] coordinates of gas-phase n-mers in evaluator order."""
    name, n = case["evaluator"], case["n"]
    if name == "mbpol2b":
        return workloads.gas_dimers(n, 2.2, 7.5, seed=seed)
    if name == "mbpol3b":
        return workloads.gas_trimers(n, 2.4, 6.5, seed=seed)
    rng = np.random.default_rng(seed)
    parts = []
    for k, m in enumerate(specs.SPECS[name].monomers):
        v = rng.normal(size=(n, 3))
        r = rng.uniform(3.0, 8.0, size=n) * (k > 0)
        centres = v / np.linalg.norm(v, axis=1, keepdims=True) * r[:, None]
        parts.append(workloads.place(rng, workloads.BODIES[m](), centres))
    return np.concatenate(parts, 1).reshape(n, -1)


def _fit_targets(case, seed):
    return np.random.default_rng(seed + 7).normal(0.0, 1.0, size=case["n"])


def prepare(case, seed):
    stream = torch.cuda.current_stream().cuda_stream or 1     # 1: the legacy default stream
    if case["kind"] == "refit":
        return dict(case=case, coef=torch.tensor(_fit(case["evaluator"]), device="cuda", requires_grad=True),
                    xyz=torch.tensor(_nmers(case, seed), device="cuda", requires_grad=True),
                    target=torch.tensor(_fit_targets(case, seed), device="cuda"))
    if case["kind"] == "batch":
        # on a stream of its own: the batch replays a captured graph
        return dict(case=case, batch=batch.Batch(_configurations(case, seed), CUT2, CUT3))
    ids, xyz, box = _molecules(case, seed)
    ctx = capi.Context(0, stream)
    s = system.from_arrays(ids, xyz, box, CUT2, CUT3, precision="mixed" if case["mixed"] else "fp64", context=ctx)
    st = dict(case=case, system=s, ctx=ctx, xyz=xyz)
    if case["api"] == "device":
        st["sites"] = torch.tensor(s.sites, device="cuda")
        st["grad"] = torch.zeros_like(st["sites"])
    elif case["api"] == "real":
        st["xyz"] = torch.tensor(xyz, device="cuda")
        st["grad"] = torch.zeros_like(st["xyz"])
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "refit":
        e = torch_ops.nmer_energies(case["evaluator"], state["xyz"], state["coef"], mixed=case["mixed"])
        loss = ((e - state["target"]) ** 2).mean()
        dxyz, dcoef = torch.autograd.grad(loss, (state["xyz"], state["coef"]))
        return dict(e=e.detach(), dxyz=dxyz, dcoef=dcoef)
    if case["kind"] == "batch":
        b = state["batch"]
        b.grad.zero_()
        e2, e3, vir = b.energy_2b3b(mixed=case["mixed"], virials=True)
        return dict(e2=e2, e3=e3, grad=b.grad, virial=vir)
    s, grads, api = state["system"], case["grads"], case["api"]
    if api == "device":
        if not grads:
            e2, e3 = state["ctx"].energy_2b3b(state["sites"], None, None, mixed=case["mixed"], grads=False)
            return dict(e2=e2, e3=e3)
        vir = np.zeros(9)
        state["grad"].zero_()
        e2, e3 = state["ctx"].energy_2b3b(state["sites"], state["grad"], vir, mixed=case["mixed"])
        return dict(e2=e2, e3=e3, grad=state["grad"], virial=vir)
    if api == "real":
        state["grad"].zero_()
        e2, v2 = s.EnergyFromRealXyz(2, state["xyz"], state["grad"], grads)
        e3, v3 = s.EnergyFromRealXyz(3, state["xyz"], state["grad"], grads)
        return dict(e2=e2, e3=e3, grad=state["grad"], virial=v2 + v3) if grads else dict(e2=e2, e3=e3)
    s.SetRealXyz(state["xyz"])
    if api == "host":
        e2, e3 = s.TwoAndThreeBodyEnergy(grads)
        return dict(e2=e2, e3=e3, grad=s.GetRealGrads(), virial=s.GetVirial()) if grads else dict(e2=e2, e3=e3)
    out = dict(e2=s.TwoBodyEnergy(grads))
    if grads:
        out.update(grad2=s.GetRealGrads(), virial2=s.GetVirial())
    out["e3"] = s.ThreeBodyEnergy(grads)
    if grads:
        out.update(grad3=s.GetRealGrads(), virial3=s.GetVirial())
    return out


# ------------------------------------------------------------------ the work
def _terms(name):
    """(coefficient index, multiplicity, variables) of every term of a polynomial."""
    with gzip.open(os.path.join(DATA, specs.SPECS[name].pip_table + ".pip.gz"), "rt") as f:
        rows = [line.split() for line in f.read().splitlines()[2:]]
    return [(int(r[0]), float(r[1]), tuple(int(v) for v in r[3:3 + int(r[2])])) for r in rows]


def _fit(name):
    path = os.path.join(DATA, name + ".fit")
    if not os.path.exists(path):
        path = os.path.join(DATA, specs.KERNEL_ALIASES[name] + ".fit")
    with open(path) as f:
        return np.array([float(v) for v in f.read().split()])


_term_counts = {}


def _flops(name, grads):
    """Operations of one n-mer's polynomial as nested products of its terms:
    about one per term for the value, 2.4 with the gradient (what the
    generated programs of the water polynomials come to)."""
    if name not in _term_counts:
        with gzip.open(os.path.join(DATA, specs.SPECS[name].pip_table + ".pip.gz"), "rt") as f:
            f.readline()
            _term_counts[name] = int(f.readline().split()[3])
    return _term_counts[name] * (2.4 if grads else 1.0)


def work(case):
    if case["kind"] == "refit":
        spec = specs.SPECS[case["evaluator"]]
        # coordinates and targets in, energies, their gradient and the
        # coefficients' gradient out; value, gradient and adjoint
        return {"bytes": 8 * (case["n"] * (6 * spec.nreal + 2) + 2 * spec.ncoef),
                "flops": case["n"] * (2 * _flops(case["evaluator"], False) + _flops(case["evaluator"], True))}
    if case["kind"] == "batch":
        systems, grads = _configurations(case, 1), True
    else:
        systems, grads = [_molecules(case, 1)], case["grads"]
    flops = atoms = 0
    for ids, xyz, box in systems:
        flops += sum(len(index) * _flops(name, grads) for name, index in _System(ids, xyz, box).nmers())
        atoms += len(xyz)
    return {"bytes": 8 * atoms * (2 if grads else 1), "flops": flops}


def tolerance(case):
    if case["mixed"]:
        # FP16-split operands and FP32 accumulation of the 3-body polynomial
        return {"rel": 4e-5, "max": 4e-3}
    return {"rel": 2e-11, "max": 1e-9}


# ------------------------------------------------------------------ 64 bits, plain torch
class _Poly:
    """A polynomial as sum_ij left_i C_ij right_j over half-monomials."""

    def __init__(self, name, dev):
        terms = _terms(name)
        nv = specs.SPECS[name].nvars
        wide = max((len(v) + 1) // 2 for _, _, v in terms)
        left, right, li, ri = {}, {}, [], []
        for _, _, v in terms:
            v = tuple(sorted(v))
            h = len(v) // 2
            li.append(left.setdefault(v[:h], len(left)))
            ri.append(right.setdefault(v[h:], len(right)))

        def columns(d):
            t = np.full((len(d), wide), nv)
            for m, i in d.items():
                t[i, :len(m)] = m
            return torch.tensor(t, device=dev)

        self.left, self.right = columns(left), columns(right)
        self.shape = (len(left), len(right))
        self.at = torch.tensor(np.array(li) * len(right) + np.array(ri), device=dev)
        self.k = torch.tensor([t[0] for t in terms], device=dev)
        self.mult = torch.tensor([t[1] for t in terms], dtype=torch.float64, device=dev)

    def matrix(self, a):
        c = torch.zeros(self.shape[0] * self.shape[1], dtype=torch.float64, device=a.device)
        return c.index_add(0, self.at, a[self.k] * self.mult).reshape(self.shape)

    def value(self, x, c):
        x = torch.cat([x, torch.ones_like(x[:, :1])], 1)

        def half(cols):
            m = x[:, cols[:, 0]]
            for q in range(1, cols.shape[1]):
                m = m * x[:, cols[:, q]]
            return m

        return ((half(self.left) @ c) * half(self.right)).sum(1)


_polys = {}


def _poly(name, dev):
    if (name, dev) not in _polys:
        _polys[(name, dev)] = _Poly(name, dev)
    return _polys[(name, dev)]


def _switched(name, poly, c, r):
    """Switched energy of n-mers r [n, atoms, 3] in evaluator order, imaged."""
    spec = specs.SPECS[name]
    sites = [r[:, i] for i in range(spec.nreal)]
    for _, o, _, _ in spec.lp:
        a, b = sites[o + 1] - sites[o], sites[o + 2] - sites[o]
        mid = sites[o] + 0.5 * specs.LP_GAMMA_IN * (a + b)
        out = specs.LP_GAMMA_OUT * torch.linalg.cross(a, b)
        sites += [mid + out, mid - out]
    x = []
    for kind, i, j, k, d0 in spec.variables:
        d = ((sites[i] - sites[j]) ** 2).sum(1).sqrt()
        v = torch.exp(k * (d0 - d))
        x.append(v / d if kind == "coul" else v)
    e = poly.value(torch.stack(x, 1), c)
    first = np.cumsum([0] + list(spec.nat))[:-1]

    def sw(i, j):
        d = ((r[:, first[i]] - r[:, first[j]]) ** 2).sum(1).sqrt()
        s = 0.5 * (1 + torch.cos(np.pi * (d - spec.ri) / (spec.rf - spec.ri)))
        return torch.where(d <= spec.ri, torch.ones_like(d), torch.where(d > spec.rf, torch.zeros_like(d), s))

    if spec.switch == "pair":
        return sw(0, 1) * e
    s01, s02, s12 = sw(0, 1), sw(0, 2), sw(1, 2)
    s = s01 * s02 + s01 * s12 + s02 * s12
    if spec.switch == "triple2":
        s = s - 2 * s01 * s02 * s12
    return s * e


class _System:
    """Molecules of one configuration, n-mers from all first-atom distances
    (orthogonal boxes, the images of an n-mer those next to its first
    monomer)."""

    def __init__(self, ids, xyz, box):
        self.dev = "cuda"
        self.ids = ids
        self.box = None if box is None else torch.tensor(np.asarray(box).reshape(3, 3).diagonal().copy(),
                                                         device=self.dev)
        self.nat = np.array([specs.MONOMER_ATOMS[m] for m in ids])
        self.start = np.cumsum(np.concatenate([[0], self.nat]))[:-1]
        nsite = np.array([specs.MONOMER_SITES[m] for m in ids])
        self.site = np.cumsum(np.concatenate([[0], nsite]))[:-1]
        self.numsites = int(nsite.sum())
        self.xyz = torch.tensor(np.asarray(xyz).reshape(-1, 3), device=self.dev)
        self.types = sorted(set(ids))
        code = {t: i for i, t in enumerate(self.types)}
        self.type = torch.tensor([code[m] for m in ids], device=self.dev)
        self.first = self.xyz[torch.tensor(self.start, device=self.dev)]

    def shift(self, d):
        return torch.zeros_like(d) if self.box is None else self.box * torch.round(d / self.box)

    def pairs(self, rc):
        """All ordered pairs (i, j) of monomers closer than rc, sorted by i."""
        n, out = len(self.ids), []
        for b in range(0, n, 1024):
            d = self.first[None, :, :] - self.first[b:b + 1024, None, :]
            d = d - self.shift(d)
            i, j = ((d ** 2).sum(2) <= rc * rc).nonzero(as_tuple=True)
            out.append(torch.stack([i + b, j], 1)[i + b != j])
        return torch.cat(out)

    def nmers(self):
        """(evaluator, [n, nbody] monomers in evaluator order) of everything that evaluates."""
        n = len(self.ids)
        for name, spec in specs.SPECS.items():
            if not set(spec.monomers) <= set(self.types):
                continue
            p = self.pairs(spec.rf)
            if spec.nbody == 2:
                t = p[p[:, 0] < p[:, 1]]
            else:
                # two of the three distances within the switch: a centre and two neighbours
                deg = torch.bincount(p[:, 0], minlength=n)
                off = torch.cumsum(deg, 0) - deg
                rep = deg[p[:, 0]]
                a = torch.repeat_interleave(torch.arange(len(p), device=self.dev), rep)
                k = torch.arange(len(a), device=self.dev) - torch.repeat_interleave(torch.cumsum(rep, 0) - rep, rep)
                b = off[p[a, 0]] + k
                keep = p[a, 1] < p[b, 1]
                t = torch.stack([p[a, 0], p[a, 1], p[b, 1]], 1)[keep].sort(dim=1).values
            want = torch.tensor(sorted(self.types.index(m) for m in spec.monomers), device=self.dev)
            t = t[(self.type[t].sort(dim=1).values == want).all(1)]
            if not len(t):
                continue
            t = torch.unique(t, dim=0) if spec.nbody == 3 else t
            # evaluator order: by the place of the type among its monomers
            place = torch.tensor([spec.monomers.index(ty) if ty in spec.monomers else 9 for ty in self.types],
                                 device=self.dev)
            order = torch.sort(place[self.type[t]], dim=1, stable=True).indices
            yield name, torch.gather(t, 1, order)

    def evaluate(self, grads):
        """{2: [energy, gradient of the atoms, virial], 3: ...}"""
        out = {nb: [0.0, torch.zeros(len(self.xyz), 3, dtype=torch.float64, device=self.dev),
                    torch.zeros(3, 3, dtype=torch.float64, device=self.dev)] for nb in (2, 3)}
        start = torch.tensor(self.start, device=self.dev)
        for name, index in self.nmers():
            spec = specs.SPECS[name]
            poly = _poly(name, self.dev)
            c = poly.matrix(torch.tensor(_fit(name), device=self.dev))
            for part in index.split(8192):
                atoms, r = [], []
                for s in range(spec.nbody):
                    a = start[part[:, s], None] + torch.arange(spec.nat[s], device=self.dev)
                    d = self.first[part[:, s]] - self.first[part[:, 0]]
                    atoms.append(a)
                    r.append(self.xyz[a] - self.shift(d)[:, None, :])
                atoms, r = torch.cat(atoms, 1), torch.cat(r, 1).requires_grad_(grads)
                e = _switched(name, poly, c, r).sum()
                out[spec.nbody][0] += float(e.detach())
                if grads:
                    g, = torch.autograd.grad(e, r)
                    out[spec.nbody][1].index_add_(0, atoms.reshape(-1), g.reshape(-1, 3))
                    out[spec.nbody][2] -= torch.einsum("nai,naj->ij", r.detach(), g)
        return out

    def sites(self, g):
        """Gradient of the atoms as the library's site array."""
        at = np.concatenate([s + np.arange(n) for s, n in zip(self.site, self.nat)])
        full = np.zeros((self.numsites, 3))
        full[at] = g.cpu().numpy()
        return full.reshape(-1)


def exact(case, seed):
    if case["kind"] == "refit":
        name = case["evaluator"]
        a = torch.tensor(_fit(name), device="cuda", requires_grad=True)
        x = torch.tensor(_nmers(case, seed), device="cuda")
        y = torch.tensor(_fit_targets(case, seed), device="cuda")
        poly = _poly(name, "cuda")
        es, gs, da = [], [], torch.zeros_like(a)
        for b in range(0, case["n"], 8192):
            r = x[b:b + 8192].reshape(-1, specs.SPECS[name].nreal, 3).requires_grad_(True)
            e = _switched(name, poly, poly.matrix(a), r)
            loss = ((e - y[b:b + 8192]) ** 2).sum() / case["n"]
            g, ga = torch.autograd.grad(loss, (r, a))
            es.append(e.detach())
            gs.append(g.reshape(len(g), -1))
            da = da + ga
        return dict(e=torch.cat(es), dxyz=torch.cat(gs), dcoef=da.detach())
    if case["kind"] == "batch":
        out = dict(e2=[], e3=[], grad=[], virial=[])
        for ids, xyz, box in _configurations(case, seed):
            s = _System(ids, xyz, box)
            r = s.evaluate(True)
            out["e2"].append(r[2][0])
            out["e3"].append(r[3][0])
            out["grad"].append(s.sites(r[2][1] + r[3][1]))
            out["virial"].append((r[2][2] + r[3][2]).cpu().numpy().reshape(-1))
        return dict(e2=np.array(out["e2"]), e3=np.array(out["e3"]),
                    grad=torch.tensor(np.concatenate(out["grad"])), virial=np.array(out["virial"]))
    ids, xyz, box = _molecules(case, seed)
    s = _System(ids, xyz, box)
    r = s.evaluate(case["grads"])
    out = dict(e2=r[2][0], e3=r[3][0])
    if not case["grads"]:
        return out
    if case["api"] == "terms":
        for nb in (2, 3):
            out["grad%d" % nb] = r[nb][1].reshape(-1).cpu().numpy()
            out["virial%d" % nb] = r[nb][2].cpu().numpy().reshape(-1)
        return out
    g = r[2][1] + r[3][1]
    out["virial"] = (r[2][2] + r[3][2]).cpu().numpy().reshape(-1)
    if case["api"] == "device":
        out["grad"] = torch.tensor(s.sites(g))
    else:
        out["grad"] = g.reshape(-1) if case["api"] == "real" else g.reshape(-1).cpu().numpy()
    return out
