"""Symmetry-adapted variables of the permutationally invariant polynomials.

Every polynomial is invariant under the exchange of like atoms.  Take K, a set
of disjoint exchanges of two like sites (H1 <-> H2 of a water, the two lone
pairs, two pairs of methane's hydrogens, ...), each of which maps the variables
x onto one another.  They commute, so sums and differences of the variables of
an orbit of K,

    w_i = sum_v W_iv x_v,   W_iv in {-1, 0, 1},

change at most their sign under any element of K, and a monomial of the w can
only occur in the polynomial when the signs of its factors cancel for every
element.  Most monomials drop out: MB-pol 3b has 33525 terms in x and 6773 in
w, MB-pol 2b 12725 and 2226, CH4-H2O-H2O 29887 and 5522, CH4-CH4 201250 and
25995.  The kernels therefore transform x to w (additions only), evaluate
the polynomial and its gradient in w, and transform the gradient back,
dP/dx_v = sum_i W_iv dP/dw_i: exact algebra, the rounding of the few additions
aside.

The remaining symmetry (exchanges of monomers, of pairs of atoms) permutes the
w up to signs; it groups the monomials into orbits with one coefficient each,
up to sign.  The coefficient of an orbit is linear in the fitted ones,
c = F a, so the number of coefficients a kernel reads stays that of the model
or a small multiple of it.

Reference points.  Some polynomials are badly conditioned in exponentials that
hardly vary over the range of the evaluator: their terms are 10^3 - 10^5 times
their sum, and rounding the coefficients c to FP64 then shifts every n-mer's
energy the same way (MB-pol 3b: 7e-11 of the mean).  SHIFTED lists them; their
w are taken relative to a point in the middle of that range, w = W x - w0, and
the terms no longer cancel (error of a trimer 1e-14 kcal/mol instead of
1e-11).  w0 has 8 significant bits, so that the factors of F are exact, and
c = F a is summed in twice the precision (two_sum / two_prod in the library).

Symmetries are not taken from a list: every exchange of two sites or two like
monomers is tried, and kept when it maps the variables (with their constants)
and the term table onto themselves.
"""
import collections
import concurrent.futures
import functools
import itertools
import os
import pickle
import subprocess
import sys
from fractions import Fraction

import numpy as np

from mbx_b200.specs import LP_GAMMA_IN, LP_GAMMA_OUT, ONEBODY_SPECS, SPECS
from mbx_b200.tables import load_pip

# relative error of the mean energy of random n-mers from rounding c, without
# a reference point: MB-pol 3b 7e-11, the alkali ions' 3b 1e-10, CO2-CO2 1e-11;
# all others are below 1e-12
SHIFTED = ("mbpol3b", "mbpbe3b", "h2oli3b", "h2ona3b", "h2ok3b", "h2orb3b", "h2ocs3b", "co2co22b", "co2a2b",
           "cm595co22b", "cm590co22b", "cm585co22b", "cm5875co22b", "cm580co22b")
W0_BITS = 8


def reference_variables(spec, group, n=400):
    """Variables in the middle of what the evaluator sees: medians over random
    rigid n-mers with first-atom distances from 2.6 A to the switch radius,
    the same for variables that a symmetry exchanges."""
    from mbx_b200 import workloads
    rng = np.random.default_rng(0)
    parts = []
    for m, name in enumerate(spec.monomers):
        v = rng.normal(size=(n, 3))
        r = rng.uniform(2.6, min(spec.rf, 6.0), size=n) * (m > 0)
        body = workloads.BODIES[name]() if name in workloads.BODIES else np.zeros((1, 3))
        parts.append(workloads.place(rng, body, v / np.linalg.norm(v, axis=1, keepdims=True) * r[:, None]))
    sites = list(np.concatenate(parts, 1).transpose(1, 0, 2))
    for _, o, _, _ in spec.lp:
        a, b = sites[o + 1] - sites[o], sites[o + 2] - sites[o]
        mid, out = sites[o] + 0.5 * LP_GAMMA_IN * (a + b), LP_GAMMA_OUT * np.cross(a, b)
        sites += [mid + out, mid - out]
    med = np.empty(spec.nvars)
    for v, (kind, i, j, k, d0) in enumerate(spec.variables):
        d = np.linalg.norm(sites[i] - sites[j], axis=1)
        x = np.exp(k * (d0 - d))
        med[v] = np.median(x / d if kind == "coul" else x)
    return np.array([np.mean([med[p[v]] for p in group]) for v in range(spec.nvars)])


def _variable_permutation(spec, site_map):
    """Where each variable goes when site i becomes site site_map[i]; None
    when the variables are not mapped onto themselves."""
    index = {}
    for v, (kind, a, b, k, d0) in enumerate(spec.variables):
        index[(kind, min(a, b), max(a, b), k, d0)] = v
    out = []
    for kind, a, b, k, d0 in spec.variables:
        a, b = site_map[a], site_map[b]
        v = index.get((kind, min(a, b), max(a, b), k, d0))
        if v is None:
            return None
        out.append(v)
    return tuple(out) if sorted(out) == list(range(len(out))) else None


def _leaves_invariant(table, perm):
    """Does the table map onto itself, coefficient by coefficient?"""
    p = np.array(list(perm) + [-1])
    v0 = np.sort(table.var, axis=1)
    v1 = np.sort(p[table.var], axis=1)
    o0, o1 = np.lexsort(v0.T), np.lexsort(v1.T)
    return (np.array_equal(v0[o0], v1[o1]) and np.array_equal(table.k[o0], table.k[o1])
            and np.array_equal(table.coef[o0], table.coef[o1]))


def symmetries(spec, table):
    """(exchanges, generators): [(site a, site b, variable permutation)] of
    single exchanges, and variable permutations generating the whole group."""
    ns = len(spec.sites)
    identity = tuple(range(spec.nvars))
    exchanges = []
    for a, b in itertools.combinations(range(ns), 2):
        m = list(range(ns))
        m[a], m[b] = b, a
        p = _variable_permutation(spec, m)
        if p and p != identity and _leaves_invariant(table, p):
            exchanges.append((a, b, p))
    gens = [p for _, _, p in exchanges]
    first = np.cumsum([0] + list(spec.nat))
    virtual = list(range(spec.nreal, ns))
    for m1, m2 in itertools.combinations(range(spec.nbody), 2):
        if spec.monomers[m1] != spec.monomers[m2]:
            continue
        for image in itertools.permutations(virtual):
            m = list(range(ns))
            for i in range(spec.nat[m1]):
                m[first[m1] + i], m[first[m2] + i] = first[m2] + i, first[m1] + i
            for a, b in zip(virtual, image):
                m[a] = b
            p = _variable_permutation(spec, m)
            if p and _leaves_invariant(table, p):
                if p != identity:
                    gens.append(p)
                break
    return exchanges, gens


def _closure(gens, identity, mul):
    group, frontier = {identity}, [identity]
    while frontier:
        new = []
        for g in frontier:
            for h in gens:
                x = mul(h, g)
                if x not in group:
                    group.add(x)
                    new.append(x)
        frontier = new
    return group


class WTable:
    """Term table in the w variables: P = sum_t sign_t c[k_t] prod w, with
    c = F a (rows of F: {fitted index: factor}), and the transform
    w = W x - w0.

    The fields nvars, ncoef, k, coef, deg and var are those of a PipTable
    (coef: the signs)."""

    def __init__(self, name, shifted):
        spec = SPECS[name] if name in SPECS else ONEBODY_SPECS[name]
        table = load_pip(name)
        nv = spec.nvars
        self.name, self.nvars, self.degree, self.nfit = name, nv, table.degree, table.ncoef
        exchanges, gens = symmetries(spec, table)
        used, K = set(), []
        for a, b, p in exchanges:
            if not used & {a, b}:
                used |= {a, b}
                K.append(p)
        kgroup = [tuple(range(nv))]
        for p in K:
            kgroup += [tuple(p[j] for j in q) for q in kgroup]
        # W: for every orbit of K on the variables, the sign patterns that the
        # orbit carries; chi: the exchanges that change the sign of a w
        rows, chi, seen = [], [], set()
        for v in range(nv):
            if v in seen:
                continue
            seen |= {p[v] for p in kgroup}
            for c in range(1 << len(K)):
                row = np.zeros(nv)
                for e, p in enumerate(kgroup):
                    row[p[v]] += -1.0 if bin(e & c).count("1") & 1 else 1.0
                if np.abs(row).max() > 0:
                    rows.append(row / np.abs(row).max())
                    chi.append(c)
        self.W = np.array(rows)
        assert self.W.shape == (nv, nv)
        inverse = np.linalg.inv(self.W)
        x_of_w = [[(i, inverse[v, i]) for i in range(nv) if abs(inverse[v, i]) > 1e-12] for v in range(nv)]
        # the polynomial in w: one representative of every orbit of K on the
        # terms, expanded; the average over K keeps the monomials whose signs cancel
        mono, seen = collections.defaultdict(lambda: collections.defaultdict(float)), set()
        for t in range(table.nterms):
            m = tuple(sorted(table.var[t, :table.deg[t]].tolist()))
            if m in seen:
                continue
            orbit = {tuple(sorted(p[v] for v in m)) for p in kgroup}
            seen |= orbit
            for factors in itertools.product(*[x_of_w[v] for v in m]):
                c, f = 0, float(len(orbit)) * table.coef[t]
                for i, y in factors:
                    c ^= chi[i]
                    f *= y
                if c == 0:
                    mono[tuple(sorted(i for i, _ in factors))][int(table.k[t])] += f
        group = _closure(gens, tuple(range(nv)), lambda h, g: tuple(h[i] for i in g))
        self.w0 = np.zeros(nv)
        if shifted:
            # relative to w0 (only the w that no exchange changes have one)
            w0 = self.W @ reference_variables(spec, group)
            for i in range(nv):
                if chi[i] == 0:
                    unit = 2.0 ** (np.floor(np.log2(abs(w0[i]))) + 1 - W0_BITS)
                    self.w0[i] = round(w0[i] / unit) * unit
            moved = collections.defaultdict(lambda: collections.defaultdict(Fraction))
            for m, d in mono.items():
                for keep in itertools.product((False, True), repeat=len(m)):
                    f = Fraction(1)
                    for i, kept in zip(m, keep):
                        if not kept:
                            f *= Fraction(float(self.w0[i]))
                    if f:
                        q = moved[tuple(i for i, kept in zip(m, keep) if kept)]
                        for k, y in d.items():
                            q[k] += f * Fraction(y)
            mono = {m: {k: float(f) for k, f in d.items()} for m, d in moved.items()}
            assert all(Fraction(f) == moved[m][k] for m, d in mono.items() for k, f in d.items())
        mono = {m: {k: f for k, f in d.items() if f != 0.0} for m, d in mono.items()}
        mono = {m: d for m, d in mono.items() if d}
        # the rest of the group as signed permutations of the w
        signed = set()
        for p in group:
            P = np.zeros((nv, nv))
            P[list(p), range(nv)] = 1.0
            M = self.W @ P @ inverse
            A = np.abs(M)
            if np.allclose(A.sum(1), 1.0, atol=1e-9) and np.allclose(A.max(1), 1.0, atol=1e-9):
                j = A.argmax(1)
                signed.add((tuple(int(i) for i in j), tuple(int(round(M[i, j[i]])) for i in range(nv))))
        signed = self._signed = sorted(signed)
        # orbits of the monomials: one coefficient, up to sign
        self.F, k, sign, var = [], [], [], []
        done = set()
        for m in sorted(mono, key=lambda m: (len(m), m)):
            if m in done:
                continue
            o = len(self.F)
            self.F.append(dict(sorted(mono[m].items())))
            for j, s in signed:
                q = tuple(sorted(j[i] for i in m))
                if q in done:
                    continue
                f = 1
                for i in m:
                    f *= s[i]
                d = mono[q]
                assert set(d) == set(mono[m]) and all(abs(d[n] - f * y) <= 1e-12 * abs(y) for n, y in mono[m].items())
                done.add(q)
                k.append(o)
                sign.append(float(f))
                var.append(q)
        assert len(done) == len(mono)
        order = sorted(range(len(k)), key=lambda t: (k[t], var[t]))
        self.k = np.array([k[t] for t in order], np.int32)
        self.coef = np.array([sign[t] for t in order])
        self.deg = np.array([len(var[t]) for t in order], np.int32)
        self.var = np.full((len(order), max(4, self.degree)), -1, np.int32)
        for n, t in enumerate(order):
            self.var[n, :len(var[t])] = var[t]
        self.ncoef = len(self.F)

    @property
    def nterms(self):
        return len(self.k)

    @functools.cached_property
    def halves(self):
        """(basis, pairs): monomials of at most half the degree (rounded up)
        and, for every term, the two of them whose product it is.  For sums
        over n-mers of all terms (the coefficient adjoint): one product per
        term instead of one per factor.  A greedy cover over the orbits of the
        terms, pruned; not the smallest possible."""
        signed = sorted({j for j, _ in self._signed})
        orbit = {}

        def rep(m):
            if m not in orbit:
                members = {tuple(sorted(j[i] for i in m)) for j in signed}
                r = min(members)
                for x in members:
                    orbit[x] = (r, len(members))
            return orbit[m]

        def splits(m):
            """All (a, b) with a b = m, a of half the degree (rounded down)."""
            power = sorted(collections.Counter(m).items())
            out = []
            for take in itertools.product(*[range(e + 1) for _, e in power]):
                if sum(take) == len(m) // 2:
                    a = [v for (v, _), n in zip(power, take) for _ in range(n)]
                    b = [v for (v, e), n in zip(power, take) for _ in range(e - n)]
                    out.append((tuple(a), tuple(b)))
            return out

        terms = [tuple(int(v) for v in self.var[t, :self.deg[t]]) for t in range(self.nterms)]
        wanted = {}
        for m in terms:
            r, _ = rep(m)
            if r not in wanted:
                wanted[r] = {(rep(a)[0], rep(b)[0]) for a, b in splits(r)}

        def covered(pairs, have):
            return any(a in have and b in have for a, b in pairs)

        have = {()}
        todo = {r: p for r, p in wanted.items() if not covered(p, have)}
        while todo:
            score = collections.Counter()
            for r, pairs in todo.items():
                best = {}
                for a, b in pairs:
                    need = {x for x in (a, b) if x not in have}
                    gain = rep(r)[1] / (sum(rep(x)[1] for x in need) * len(need))
                    for x in need:
                        best[x] = max(best.get(x, 0.0), gain)
                score.update(best)
            have.add(max(sorted(score), key=lambda x: score[x]))
            todo = {r: p for r, p in todo.items() if not covered(p, have)}
        for x in sorted(have - {()}, key=lambda x: (-rep(x)[1], x)):
            rest = have - {x}
            if all(covered(p, rest) for p in wanted.values()):
                have = rest
        basis = sorted({tuple(sorted(j[i] for i in r)) for r in have for j in signed}, key=lambda m: (len(m), m))
        index = {m: n for n, m in enumerate(basis)}
        pairs = []
        for m in terms:
            pairs.append(next((index[a], index[b]) for a, b in splits(m) if a in index and b in index))
        return basis, pairs

    def coefficients(self, a):
        """c = F a, rounded once (the library sums in twice the precision)."""
        return np.array([float(sum(Fraction(f) * Fraction(float(a[k])) for k, f in row.items())) for row in self.F])


def table_key(name):
    """The key of an evaluator's WTable.  Evaluators that share a term table
    share its symmetry (their variables connect the same sites), so they share
    this too, unless they have a reference point of their own."""
    spec = SPECS[name] if name in SPECS else ONEBODY_SPECS[name]
    return name if name in SHIFTED else spec.pip_table


_tables = {}


def by_key(key):
    """WTable of a key: an evaluator of SHIFTED, or a term table (without a
    reference point, for caller-supplied variables)."""
    if key not in _tables:
        name = key
        if key not in SHIFTED:
            name = next(n for n, spec in list(SPECS.items()) + list(ONEBODY_SPECS.items()) if spec.pip_table == key)
        _tables[key] = WTable(name, key in SHIFTED)
    return _tables[key]


_ONE_TABLE = """
import pickle, sys
sys.path.insert(0, sys.argv[1])
from mbx_b200.codegen.wbasis import by_key
w = by_key(sys.argv[2])
w.halves
sys.stdout.buffer.write(pickle.dumps(w))
"""


def prepare(keys):
    """Makes the WTables of the keys, half-monomials included, in processes of
    their own side by side (all of them: 80 s in one process)."""
    root = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

    def one(key):
        r = subprocess.run([sys.executable, "-c", _ONE_TABLE, root, key], capture_output=True)
        if r.returncode != 0:
            raise RuntimeError("table %s:\n%s" % (key, r.stderr.decode()[-2000:]))
        return key, pickle.loads(r.stdout)

    todo = [k for k in keys if k not in _tables]
    with concurrent.futures.ThreadPoolExecutor(os.cpu_count() or 4) as ex:
        _tables.update(ex.map(one, todo))


def wtable(name):
    """WTable of an evaluator."""
    return by_key(table_key(name))


def emit(w, name, out, back):
    """CUDA code of the transform NAME_to_w (x -> w = W x - w0 in place) and,
    with back, of NAME_from_w (dP/dw -> dP/dx in place)."""
    nv = w.nvars

    def rows(M, w0):
        text = []
        for i in range(nv):
            parts = [("+" if M[i, v] > 0 else "-", "t[%d]" % v) for v in range(nv) if M[i, v] != 0.0]
            if w0[i] != 0.0:
                parts.append(("-", repr(float(w0[i]))))
            if parts == [("+", "t[%d]" % i)]:
                continue
            text.append("    x[%d] = %s;" % (i, " ".join("%s %s" % p for p in parts).lstrip("+ ")))
        return text

    for fn, M, w0 in (("to_w", w.W, w.w0), ("from_w", w.W.T, np.zeros(nv)))[:2 if back else 1]:
        out.append("__device__ __forceinline__ void %s_%s(double (&x)[%d]) {" % (name, fn, nv))
        text = rows(M, w0)
        if text:
            out.append("    double t[%d];" % nv)
            out.append("#pragma unroll")
            out.append("    for (int i = 0; i < %d; ++i) t[i] = x[i];" % nv)
            out.extend(text)
        out.append("}")


def emit_chain(w, spec, out):
    """NAME_chain_w: the chain rule from shared-memory columns of the w
    (xm[i * S]) and of dP/dw (gm[i * S]), orbit by orbit of the variables: an
    orbit's variables and their gradients from its few w, then each variable's
    share of the site gradients.  The variables are not evaluated again (no
    exponential, square root or division), and no array of all of them is
    held in registers."""
    nv, name, ns = w.nvars, spec.name, len(spec.sites)
    a = out.append
    a("template <int S>")
    a("__device__ __forceinline__ void %s_chain_w(const double (&s)[%d][3], const double* __restrict__ xm, "
      "const double* __restrict__ gm, double (&sg)[%d][3]) {" % (name, ns, ns))
    a("#pragma unroll")
    a("    for (int i = 0; i < %d; ++i) { sg[i][0] = 0.0; sg[i][1] = 0.0; sg[i][2] = 0.0; }" % ns)
    inverse = np.linalg.inv(w.W)
    done = set()
    for v in range(nv):
        if v in done:
            continue
        rows = [i for i in range(nv) if w.W[i, v] != 0.0]
        orbit = sorted({u for i in rows for u in range(nv) if w.W[i, u] != 0.0})
        assert sorted({i for u in orbit for i in range(nv) if w.W[i, u] != 0.0}) == rows
        done |= set(orbit)
        a("    {")
        for i in rows:
            base = "" if w.w0[i] == 0.0 else " + %r" % float(w.w0[i])
            a("        const double w%d = xm[%d * S]%s, g%d = gm[%d * S];" % (i, i, base, i, i))
        for u in orbit:
            kind, p, q, k, _ = spec.variables[u]
            scale = abs(inverse[u, rows[0]])
            assert all(abs(inverse[u, i]) == scale for i in rows)
            x = " ".join("%s w%d" % ("+" if inverse[u, i] > 0 else "-", i) for i in rows).lstrip("+ ")
            g = " ".join("%s g%d" % ("+" if w.W[i, u] > 0 else "-", i) for i in rows).lstrip("+ ")
            x = x if scale == 1.0 else "%r * (%s)" % (float(scale), x)
            fn = "dvar_exp_v" if kind == "exp" else "dvar_coul_v"
            a("        %s(s[%d], s[%d], %r, %s, %s, sg[%d], sg[%d]);" % (fn, p, q, float(k), x, g, p, q))
        a("    }")
    for (m, o, xp, xm) in spec.lp:
        a("    lp_grads(s[%d], s[%d], s[%d], sg[%d], sg[%d], sg[%d], sg[%d], sg[%d]);" %
          (o, o + 1, o + 2, xp, xm, o, o + 1, o + 2))
    a("}")
