#!/usr/bin/env python3
"""Generate the per-evaluator CUDA device code from the declarative specs.

For each evaluator in ``mbx_b200.specs.SPECS`` this writes
``mbx_b200/csrc/gen/<name>.cuh`` holding:

* ``<name>_vars``: the polynomial variables (straight-line FP64: differences,
  sqrt, exp) and the factor that turns dP/dv into a Cartesian gradient;
* ``<name>_pip``: the polynomial and its reverse-mode gradient, as a
  multivariate Horner trie over the expanded term table;
* ``<name>_pip_e``: the energy-only Horner evaluation;
* ``<name>_qf`` (types in QF_TYPES): the quadratic form of the type's FP32
  basis (codegen/shift.py, codegen/qf.py), the mixed-precision polynomial.

The tries are those of the polynomial in the symmetry-adapted variables w
(codegen/wbasis.py), which has 3 to 8 times fewer terms than in the variables
of the model.  Every evaluator also gets a table unit ``<name>_t.cu`` (the
coefficient adjoint) over the term tables that ``write_term_tables`` packs
into one binary embedded in the library.

The trie.  Every term is a monomial x_v1 x_v2 ... (variables sorted in a fixed
order); the monomials form a prefix tree.  With P(n) the product along the path
to node n and V(n) = c_n + sum_children x_var(child) V(child), the polynomial
is V(root) and reverse mode gives dP/dx_var(n) += P(parent(n)) V(n) for every
node.  A depth-first walk keeps only one (P, V) pair per depth live, so the
whole evaluation runs out of registers: nvars values, nvars gradient
accumulators and eight temporaries.  Each leaf costs two FMAs (one into V,
one into its gradient), each inner node one multiply and two FMAs.

Coefficients come from ``coef[k]``, ``coef`` being a template parameter of
the generated functions (a view of a ``__constant__`` array or of a global
pointer).
"""
import argparse
import collections
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
sys.path.insert(0, os.path.dirname(PKG))

from mbx_b200.specs import SPECS, ONEBODY_SPECS, LP_GAMMA_IN, LP_GAMMA_OUT  # noqa: E402
from mbx_b200.tables import load_pip  # noqa: E402
from mbx_b200.codegen.wbasis import (by_key as wtable_by_key, emit as emit_transforms, emit_chain,  # noqa: E402
                                      prepare as prepare_tables, table_key, wtable)

OUT = os.path.join(PKG, "csrc", "gen")



def lit(v):
    r = repr(float(v))
    if "e" not in r and "." not in r and "inf" not in r and "nan" not in r:
        r += ".0"
    return r


class Trie:
    """The monomials as a tree.  At every node the variable that occurs in
    the most of the remaining monomials is split off first (a multivariate
    Horner scheme): fewer inner nodes than one variable order for the whole
    tree (MB-pol 3b: 1390, 17.5k FP64 operations a trimer; with the variables
    in the order of the model 2611 and 20.5k, the rarest first 2137 and
    18.4k)."""

    def __init__(self, table):
        self.root = self._node([(table.var[t, :table.deg[t]].tolist(), (int(table.k[t]), float(table.coef[t])))
                                for t in range(table.nterms)])

    def _node(self, terms):
        node = {"coef": [c for m, c in terms if not m], "kids": collections.OrderedDict()}
        terms = [(m, c) for m, c in terms if m]
        while terms:
            freq = collections.Counter(v for m, _ in terms for v in set(m))
            best = max(freq, key=lambda v: (freq[v], -v))
            mine = []
            for m, c in terms:
                if best in m:
                    i = m.index(best)
                    mine.append((m[:i] + m[i + 1:], c))
            terms = [(m, c) for m, c in terms if best not in m]
            node["kids"][best] = self._node(mine)
        return node

    def counts(self):
        leaves = inner = 0
        stack = [self.root]
        while stack:
            n = stack.pop()
            for ch in n["kids"].values():
                if ch["kids"]:
                    inner += 1
                    stack.append(ch)
                else:
                    leaves += 1
        return leaves, inner


# Mixed precision (the "s" kernels).  "median": the
# polynomial is re-expanded around a symmetric reference point in the middle
# of liquid data (codegen/shift.py); "identity": the original basis in FP32.
# Types not listed run FP64 in the mixed mode.  MB-pol 2b is not listed: in
# FP32 (identity basis, FP32 coefficients and leaf sums) its energy over the
# 2048-water box is off by 1.1e-5 even with the dimers below 4.5 A in FP64
# (the shifted basis does not condition it either).
SHIFT_TYPES = {"mbpol3b": "median"}
# Types of SHIFT_TYPES whose mixed kernel is the quadratic form on the tensor
# cores (codegen/qf.py, csrc/qf_kernel.cuh):
# MB-pol 3b, 442 products of degree 2 in the basis (data/mbpol3b.qf.json).
QF_TYPES = {"mbpol3b"}
# Optional: n-mers whose first-atom distance is below this radius (A) run the
# FP64 kernel in the mixed mode (a type of SHIFT_TYPES whose short-range
# n-mers cancel too strongly for FP32); the builder puts them in a bucket of
# their own.
MIXED_FP64_RADIUS = {}


# Terms up to which a trie reads its coefficients in the order of its leaves
# (one constant per leaf, sign included: consecutive constants, fetched in
# pairs) instead of one per orbit; a unit's constant memory holds 8192 doubles.
LEAF_ORDER_TERMS = 8000


class Coefficients:
    """Names of the coefficients in a trie's code: coef[orbit], or coef[i] in
    the order of emission (leaves lists the (orbit, sign) of every i)."""

    def __init__(self, by_leaf):
        self.by_leaf = by_leaf
        self.leaves = []

    def __call__(self, coefs):
        """Sum of the coefficients of the terms ending at a node, None without one."""
        parts = []
        for k, c in coefs:
            assert c in (1.0, -1.0)
            if self.by_leaf:
                parts.append("coef[%d]" % len(self.leaves))
                self.leaves.append((k, c))
            else:
                parts.append("coef[%d]" % k if c > 0 else "(-coef[%d])" % k)
        return " + ".join(parts) if parts else None


def split_terms(trie, nparts):
    """The trie cut into nparts sub-tries of contiguous terms in depth-first
    order, each carrying the path nodes its terms hang from.  A path node's
    own coefficient goes with the range that holds it, so every term is in
    exactly one sub-trie; each sub-trie evaluates to its share of the
    polynomial (the trie value is linear in the terms)."""
    terms = []

    def walk(node, path):
        if node is not trie.root and node["coef"]:
            terms.append((path, node["coef"]))
        for v, ch in node["kids"].items():
            walk(ch, path + (v,))
    walk(trie.root, ())
    per = -(-len(terms) // max(1, nparts))
    roots = []
    for lo in range(0, len(terms), per):
        root = {"coef": [], "kids": collections.OrderedDict()}
        for path, coefs in terms[lo:lo + per]:
            node = root
            for v in path:
                node = node["kids"].setdefault(v, {"coef": [], "kids": collections.OrderedDict()})
            node["coef"].extend(coefs)
        roots.append(root)
    return [list(r["kids"].items()) for r in roots]


def lock_threads(nvars):
    """Threads of a lockstep evaluation block.  The kernels wait for
    instructions more than for anything else, and a block's warps share every
    fetch, so as many warps as the columns of x and g leave room for in 227 KB
    of shared memory: 384 threads (168 registers) up to 36 variables, else 256
    (255 registers), 128 above 56 variables, where the columns of 256 do not
    fit.  MB-pol 3b gradients of 132k trimers: 410 us with 384 threads, 475
    with 320, 550 with 256; MB-pol 2b, 39k dimers: 81 us with 384, 109 with 256.
    The energy kernels, which have the columns of x alone, take the same number;
    more threads have not been measured there."""
    if nvars > 56:
        return 128
    return 384 if nvars <= 36 else 256


def parts_for(nterms, nvars=36):
    """Number of separately compiled pieces of a trie.  A single straight-line
    function of 10^4 FMAs leaves the register allocator live ranges it cannot
    fit, and the code of a piece should stay small enough for the instruction
    cache that the warps of a lockstep block share.  Measured on 132k MB-pol 3b
    trimers (256 threads): 570, 550 and 564 us at 300, 600 and 900 terms a
    piece; on 76k N2O5-H2O-H2O trimers, 78 variables (128 threads): 641, 574 and
    562 us at 200, 600 and 1000.  Small batches are cut by pieces over the SMs
    (LockPlan), which asks for no larger ones: MB-pol 2b, with 250, 400 and 600
    terms a piece, takes 130, 125 and 120 us for 76k dimers, and a call on 8
    waters 130, 131 and 136."""
    per = 400 if nvars <= 32 else 600
    return max(1, (nterms + per - 1) // per)


def emit_split(trie, nvars, name, out, nparts, arrays, body, coef_expr, ret="double"):
    """Emits name_partK as __noinline__ functions over strided pointers to the
    caller's arrays, and the dispatcher name_piece.

    arrays: [(name, ctype, role)] with role "in" (read: copied into a local
    register array on entry) or "acc" (accumulated: zeroed locally, added to
    the caller's array on exit).  A piece reads element v of an array at
    pointer[v * S], S a template parameter: S = 1 for a thread's own local
    array, S = block size for a shared-memory array laid out [v][thread] (the
    lockstep kernels keep x and g there: shared memory instead of the
    thread's stack for the values every piece loads and stores).  body(w,
    subtrees) writes the evaluation of the subtrees into the local arrays and
    into E."""
    import re
    w = out.append
    zero = {"double": "0.0"}
    e0 = "0.0"
    pieces = split_terms(trie, nparts)
    params = ", ".join("%s%s* __restrict__ %sm" % ("const " if role == "in" else "", ct, a) for a, ct, role in arrays)
    constant = coef_expr(trie.root["coef"])
    for i, sub in enumerate(pieces):
        text = []
        body(text.append, sub)
        if i == 0 and constant:
            text.append("    E += %s;" % constant)
        code = "\n".join(text)
        w("template <class Coef, int S>")
        w("__device__ __noinline__ %s %s_part%d(const Coef& coef, %s) {" % (ret, name, i, params))
        w("    %s E = %s;" % (ret, e0))
        for a, ct, role in arrays:
            used = sorted({int(v) for v in re.findall(r"\b%s\[(\d+)\]" % a, code)})
            w("    %s %s[%d];" % (ct, a, nvars))
            for v in used:
                w("    %s[%d] = %s;" % (a, v, ("%sm[%d * S]" % (a, v)) if role == "in" else zero[ct]))
        w(code)
        for a, ct, role in arrays:
            if role == "acc":
                used = sorted({int(v) for v in re.findall(r"\b%s\[(\d+)\]" % a, code)})
                for v in used:
                    w("    %sm[%d * S] += %s[%d];" % (a, v, a, v))
        w("    return E;")
        w("}")

    # name_piece<S>(k, coef, xm, gm): piece k over shared arrays [v][S]
    # (pointers at the thread's column).  The lockstep kernels run the pieces
    # of a chunk in turn with a block barrier after each, so that all warps of
    # a block share the instruction fetches of a piece; their prefetch launch
    # runs one piece per block
    w("template <int S, class Coef>")
    w("__device__ __forceinline__ %s %s_piece(int k, const Coef& coef, %s) {" % (ret, name, params))
    w("    switch (k) {")
    args = ", ".join("%sm" % a for a, _, _ in arrays)
    for i in range(len(pieces)):
        w("    case %d: return %s_part%d<Coef, S>(coef, %s);" % (i, name, i, args))
    w("    default: return %s;" % e0)
    w("    }")
    w("}")


def emit_pip(trie, nvars, name, out, coef_expr, nparts=1):
    """FP64 value + gradient (multivariate Horner trie, reverse mode)."""
    out.append("// %s: polynomial and reverse-mode gradient (multivariate Horner trie)" % name)

    def body(w, subtrees):
        def node(n, var, depth, pexpr):
            # pexpr: expression for P(parent), None at the root's children (P = 1)
            P = "P%d" % depth
            V = "V%d" % depth
            if pexpr is None:
                w("    { const double %s = x[%d];" % (P, var))
            else:
                w("    { const double %s = %s * x[%d];" % (P, pexpr, var))
            ce = coef_expr(n["coef"])
            w("      double %s = %s;" % (V, ce if ce else "0.0"))
            for cv, ch in n["kids"].items():
                if ch["kids"]:
                    node(ch, cv, depth + 1, P)
                else:
                    c = coef_expr(ch["coef"])
                    w("      %s = fma(%s, x[%d], %s); g[%d] = fma(%s, %s, g[%d]);" % (V, c, cv, V, cv, c, P, cv))
            if pexpr is None:
                w("      g[%d] += %s; E = fma(x[%d], %s, E); }" % (var, V, var, V))
            else:
                w("      g[%d] = fma(%s, %s, g[%d]); V%d = fma(x[%d], %s, V%d); }" %
                  (var, pexpr, V, var, depth - 1, var, V, depth - 1))

        for var, ch in subtrees:
            if ch["kids"]:
                node(ch, var, 1, None)
            else:
                c = coef_expr(ch["coef"])
                w("    E = fma(%s, x[%d], E); g[%d] += %s;" % (c, var, var, c))

    emit_split(trie, nvars, name, out, nparts, [("x", "double", "in"), ("g", "double", "acc")], body, coef_expr)


def shifted_pip(name):
    """codegen.shift.ShiftedPip of a type in SHIFT_TYPES (cached)."""
    from mbx_b200.codegen import shift
    if name in _SHIFTED:
        return _SHIFTED[name]
    spec, table = SPECS[name], load_pip(name)
    if SHIFT_TYPES[name] == "median":
        sp = shift.shifted(spec, table)
    else:
        monos = [tuple(sorted(table.var[t, :table.deg[t]].tolist())) for t in range(table.nterms)]
        sp = shift.ShiftedPip(spec.nvars, spec.ncoef, np.zeros(spec.nvars), monos,
                              [int(k) for k in table.k], {}, [{k: 1.0} for k in range(spec.ncoef)], [])
        # the identity basis keeps the term multiplicities of the table
        assert all(c == 1.0 for c in table.coef)
    _SHIFTED[name] = sp
    return sp


_SHIFTED = {}


def emit_pip_energy(trie, nvars, name, out, coef_expr, nparts=1):
    """FP64 value only: plain Horner over the trie."""
    def body(w, subtrees):
        def node(n, var, depth):
            V = "V%d" % depth
            ce = coef_expr(n["coef"])
            w("    { double %s = %s;" % (V, ce if ce else "0.0"))
            for cv, ch in n["kids"].items():
                if ch["kids"]:
                    node(ch, cv, depth + 1)
                else:
                    w("      %s = fma(%s, x[%d], %s);" % (V, coef_expr(ch["coef"]), cv, V))
            tgt = "E" if depth == 1 else "V%d" % (depth - 1)
            w("      %s = fma(x[%d], %s, %s); }" % (tgt, var, V, tgt))

        for var, ch in subtrees:
            if ch["kids"]:
                node(ch, var, 1)
            else:
                w("    E = fma(%s, x[%d], E);" % (coef_expr(ch["coef"]), var))

    emit_split(trie, nvars, name, out, nparts, [("x", "double", "in")], body, coef_expr)


def emit_vars(spec, out):
    """Sites (incl. lone pairs), variables and their Cartesian derivative factors."""
    w = out.append
    ns = len(spec.sites)
    nv = spec.nvars
    w("// sites, variables and dv/d(p1-p2) factors for %s (%s)" % (spec.name, spec.ref))
    w("__device__ __forceinline__ void %s_sites(const double (&r)[%d][3], double (&s)[%d][3]) {" %
      (spec.name, spec.nreal, ns))
    w("#pragma unroll")
    w("    for (int i = 0; i < %d; ++i) { s[i][0] = r[i][0]; s[i][1] = r[i][1]; s[i][2] = r[i][2]; }" % spec.nreal)
    for (m, o, xp, xm) in spec.lp:
        w("    lp_sites(s[%d], s[%d], s[%d], s[%d], s[%d]);" % (o, o + 1, o + 2, xp, xm))
    w("}")
    w("__device__ __forceinline__ void %s_vars(const double (&s)[%d][3], double (&x)[%d]) {" % (spec.name, ns, nv))
    for v, (kind, a, b, k, d0) in enumerate(spec.variables):
        fn = "var_exp" if kind == "exp" else "var_coul"
        w("    x[%d] = %s(s[%d], s[%d], %s, %s);" % (v, fn, a, b, lit(k), lit(d0)))
    w("}")
    # the variables with their radial factors, for a chain rule in another
    # kernel that reads the factors back (NAME_chain_q); q.put(v, factor)
    # stores each as soon as it is known
    w("template <class QW>")
    w("__device__ __forceinline__ void %s_vars_q(const double (&s)[%d][3], double (&x)[%d], QW& q) {" %
      (spec.name, ns, nv))
    for v, (kind, a, b, k, d0) in enumerate(spec.variables):
        fn = "var_exp_q" if kind == "exp" else "var_coul_q"
        w("    { double f; x[%d] = %s(s[%d], s[%d], %s, %s, f); q.put(%d, f); }" % (v, fn, a, b, lit(k), lit(d0), v))
    w("}")
    w("template <class G, class Q>")
    w("__device__ __forceinline__ void %s_chain_q(const double (&s)[%d][3], const G& g, const Q& q, "
      "double (&sg)[%d][3]) {" % (spec.name, ns, ns))
    w("#pragma unroll")
    w("    for (int i = 0; i < %d; ++i) { sg[i][0] = 0.0; sg[i][1] = 0.0; sg[i][2] = 0.0; }" % ns)
    for v, (kind, a, b, k, d0) in enumerate(spec.variables):
        w("    dvar_q(s[%d], s[%d], g[%d], q[%d], sg[%d], sg[%d]);" % (a, b, v, v, a, b))
    for (m, o, xp, xm) in spec.lp:
        w("    lp_grads(s[%d], s[%d], s[%d], sg[%d], sg[%d], sg[%d], sg[%d], sg[%d]);" %
          (o, o + 1, o + 2, xp, xm, o, o + 1, o + 2))
    w("}")
    if spec.name not in ONEBODY_SPECS:
        return   # the n-mer kernels' chain rules are chain_w (wbasis.py) and chain_q
    # chain rule of the 1-body kernel: site gradients from dP/dv
    w("template <class G>")
    w("__device__ __forceinline__ void %s_chain(const double (&s)[%d][3], const G& g, "
      "double (&sg)[%d][3]) {" % (spec.name, ns, ns))
    w("#pragma unroll")
    w("    for (int i = 0; i < %d; ++i) { sg[i][0] = 0.0; sg[i][1] = 0.0; sg[i][2] = 0.0; }" % ns)
    for v, (kind, a, b, k, d0) in enumerate(spec.variables):
        fn = "dvar_exp" if kind == "exp" else "dvar_coul"
        w("    %s(s[%d], s[%d], %s, %s, g[%d], sg[%d], sg[%d]);" % (fn, a, b, lit(k), lit(d0), v, a, b))
    for (m, o, xp, xm) in spec.lp:
        w("    lp_grads(s[%d], s[%d], s[%d], sg[%d], sg[%d], sg[%d], sg[%d], sg[%d]);" %
          (o, o + 1, o + 2, xp, xm, o, o + 1, o + 2))
    w("}")


def emit_traits(spec, straight, npieces, out):
    """Compile-time description the kernel templates in holder_kernel.cuh use."""
    w = out.append
    n = spec.name
    nat = list(spec.nat) + [0] * (3 - len(spec.nat))
    first = [0, nat[0], nat[0] + nat[1]]
    ns = len(spec.sites)
    w("struct %s_T {" % n)
    w("    static constexpr int NBODY = %d, NVARS = %d, NREAL = %d, NSITES = %d;" %
      (spec.nbody, spec.nvars, spec.nreal, ns))
    w("    static constexpr int NAT0 = %d, NAT1 = %d, NAT2 = %d;" % tuple(nat))
    w("    static constexpr int FIRST0 = %d, FIRST1 = %d, FIRST2 = %d;" % tuple(first))
    w("    static constexpr int SWITCH_TRIPLE = %d, SKIP = %d;" %
      ({"pair": 0, "triple": 1, "triple2": 2, "cos2": 3, "none": 0}[spec.switch],
       {"pair_gt": 0, "two_of_three_gt": 1, "all_three_gt": 2, "none": 0}[spec.skip]))
    w("    static constexpr int TPAIRS = %d;  // (variable, exponent) pairs of a term, at most" %
      term_pairs_max(table_key(n)))
    w("    static constexpr double RI = %s, RF = %s;" % (lit(spec.ri), lit(spec.rf)))
    w("    static constexpr int VIRIAL_RAW = %d;  // virial of the unswitched polynomial gradient" %
      (1 if spec.virial == "raw" else 0))
    w("    static constexpr int LOCK_THREADS = %d;  // threads of a lockstep evaluation block" %
      lock_threads(spec.nvars))
    w("    __device__ __forceinline__ static void to_w(double (&x)[%d]) { %s_to_w(x); }" % (spec.nvars, n))
    if not straight:
        w("    __device__ __forceinline__ static void from_w(double (&g)[%d]) { %s_from_w(g); }" % (spec.nvars, n))
    if straight and n in SHIFT_TYPES:
        w("    __device__ __forceinline__ static void shift(const double (&x)[%d], float (&xf)[%d]) "
          "{ %s_shift(x, xf); }" % (spec.nvars, spec.nvars, n))
    w("    __device__ __forceinline__ static void sites(const double (&r)[%d][3], double (&s)[%d][3]) { %s_sites(r, s); }" %
      (spec.nreal, ns, n))
    w("    __device__ __forceinline__ static void vars(const double (&s)[%d][3], double (&x)[%d]) { %s_vars(s, x); }" %
      (ns, spec.nvars, n))
    if not straight:
        w("    template <class G> __device__ __forceinline__ static void chain(const double (&s)[%d][3], const G& g, "
          "double (&sg)[%d][3]) { %s_chain(s, g, sg); }" % (ns, ns, n))
    w("    template <class QW> __device__ __forceinline__ static void vars_q(const double (&s)[%d][3], "
      "double (&x)[%d], QW& q) { %s_vars_q(s, x, q); }" % (ns, spec.nvars, n))
    w("    template <class G, class Q> __device__ __forceinline__ static void chain_q(const double (&s)[%d][3], "
      "const G& g, const Q& q, double (&sg)[%d][3]) { %s_chain_q(s, g, q, sg); }" % (ns, ns, n))
    if straight:
        w("    template <int S> __device__ __forceinline__ static void chain_w(const double (&s)[%d][3], "
          "const double* __restrict__ x, const double* __restrict__ g, double (&sg)[%d][3]) "
          "{ %s_chain_w<S>(s, x, g, sg); }" % (ns, ns, n))
        w("    static constexpr int NPIECES = %d, NPIECES_E = %d;  // of the two tries" % (npieces, npieces))
        w("    template <int S, class C> __device__ __forceinline__ static double pip_piece(int k, const C& c, "
          "const double* __restrict__ x, double* __restrict__ g) { return %s_pip_piece<S>(k, c, x, g); }" % n)
        w("    template <int S, class C> __device__ __forceinline__ static double pip_e_piece(int k, const C& c, "
          "const double* __restrict__ x) { return %s_pip_e_piece<S>(k, c, x); }" % n)
    w("};")


def write_if_changed(path, text):
    old = open(path).read() if os.path.exists(path) else None
    if old != text:
        with open(path, "w") as f:
            f.write(text)


def generate(name):
    """Writes <name>.cuh (sizes, sites, variables, chain rule, traits) and one
    header per polynomial variant, so that a change to one variant rebuilds
    only the units that include it."""
    spec = SPECS[name] if name in SPECS else ONEBODY_SPECS[name]
    table = load_pip(name)
    straight = name in SPECS
    wt = wtable(name)
    trie = Trie(wt) if straight else None
    leaves, inner = trie.counts() if straight else (table.nterms, 0)
    head = ["// Generated by mbx_b200/codegen/gen_kernels.py from mbx_b200/specs.py and",
            "// mbx_b200/data/%s.pip.gz -- do not edit." % name]
    out = head + ["// %d terms: %d leaves, %d inner nodes" % (table.nterms, leaves, inner),
                  "#pragma once"]
    emit_vars(spec, out)
    nv = spec.nvars
    nparts = parts_for(wt.nterms, nv) if straight else 0
    npieces = len(split_terms(trie, nparts)) if straight else 0
    out.append("// %d terms in the w variables" % wt.nterms)
    emit_transforms(wt, name, out, back=not straight)
    if straight:
        emit_chain(wt, spec, out)
        out += ["template <int S, class Coef> __device__ __forceinline__ double %s_pip_piece(int, const Coef&, "
                "const double* __restrict__, double* __restrict__);" % name,
                "template <int S, class Coef> __device__ __forceinline__ double %s_pip_e_piece(int, const Coef&, "
                "const double* __restrict__);" % name]
        if name in SHIFT_TYPES:
            sp = shifted_pip(name)
            out.append("// dx = x - x0, the reference point of the FP32 basis (%s)" % SHIFT_TYPES[name])
            out.append("__device__ __forceinline__ void %s_shift(const double (&x)[%d], float (&xf)[%d]) {" %
                       (name, nv, nv))
            for v in range(nv):
                if sp.x0[v] == 0.0:
                    out.append("    xf[%d] = (float)x[%d];" % (v, v))
                else:
                    out.append("    xf[%d] = (float)(x[%d] - %s);" % (v, v, lit(float(sp.x0[v]))))
            out.append("}")
    emit_traits(spec, straight, npieces, out)
    os.makedirs(OUT, exist_ok=True)
    write_if_changed(os.path.join(OUT, name + ".cuh"), "\n".join(out) + "\n")
    if straight:
        for suffix, emitter, arg in (("pip", emit_pip, trie), ("pip_e", emit_pip_energy, trie)):
            body = head + ["#pragma once", '#include "%s.cuh"' % name]
            coef = Coefficients(wt.nterms <= LEAF_ORDER_TERMS)
            emitter(arg, nv, "%s_%s" % (name, suffix), body, coef, nparts)
            if coef.by_leaf:
                body.append("// (orbit + 1) of every coefficient, negative for -1")
                body.append("#define %s_%s_LEAVES %s" % (name, suffix, ",".join(
                    str((k + 1) * int(c)) for k, c in coef.leaves)))
            write_if_changed(os.path.join(OUT, "%s_%s.cuh" % (name, suffix)), "\n".join(body) + "\n")
        if name in QF_TYPES:
            from mbx_b200.codegen import qf
            write_if_changed(os.path.join(OUT, "%s_qf.cuh" % name),
                             qf.emit_cuda(qf.QuadForm(name, shifted_pip(name)), name, nv))
    return os.path.join(OUT, name + ".cuh"), leaves, inner


TU_HEAD = """// Generated by mbx_b200/codegen/gen_kernels.py -- do not edit.
// %(what)s for the %(name)s evaluator.
#include <cstring>
#include <vector>
#include "../holder_kernel.cuh"
#include "../launch_cache.cuh"
#include "%(name)s.cuh"
%(include)s
static __constant__ double c_%(name)s[%(nc)d];
struct %(name)s_CC {
    __device__ __forceinline__ double operator[](int k) const { return c_%(name)s[k]; }
};

%(setter)s"""

# coefficients by orbit: the w coefficients as they are
SET_ORBIT = """// the coefficients in the w variables (%(nc)d doubles, on the host or the device)
int mbx_set_coef_%(name)s_%(v)s(const double* c, int from_device, cudaStream_t s) {
    return (int)cudaMemcpyToSymbolAsync(c_%(name)s, c, sizeof(double) * %(nc)d, 0,
                                        from_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s);
}
"""

# coefficients by leaf of the trie
SET_LEAF = """// the coefficients in the w variables (on the host or the device), one per leaf
static const short leaf_h_%(name)s[%(nc)d] = {%(name)s_%(pip)s_LEAVES};
static __device__ const short leaf_d_%(name)s[%(nc)d] = {%(name)s_%(pip)s_LEAVES};
static __device__ double leaf_c_%(name)s[%(nc)d];

static __global__ void k_leaf_%(name)s(const double* __restrict__ c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= %(nc)d) return;
    const int o = leaf_d_%(name)s[i];
    leaf_c_%(name)s[i] = o > 0 ? c[o - 1] : -c[-o - 1];
}

int mbx_set_coef_%(name)s_%(v)s(const double* c, int from_device, cudaStream_t s) {
    if (!from_device) {
        std::vector<double> h(%(nc)d);
        for (int i = 0; i < %(nc)d; ++i) h[i] = leaf_h_%(name)s[i] > 0 ? c[leaf_h_%(name)s[i] - 1] : -c[-leaf_h_%(name)s[i] - 1];
        cudaError_t e = cudaMemcpyToSymbolAsync(c_%(name)s, h.data(), sizeof(double) * %(nc)d, 0, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        return (int)e;
    }
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, leaf_c_%(name)s);
    if (e != cudaSuccess) return (int)e;
    k_leaf_%(name)s<<<(%(nc)d + 127) / 128, 128, 0, s>>>(c);
    e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbolAsync(c_%(name)s, p, sizeof(double) * %(nc)d, 0, cudaMemcpyDeviceToDevice, s);
    return (int)e;
}
"""

LOCK_LAUNCH = """
int mbx_launch_%(name)s_%(v)s(const HolderArgs& A, int grid, int block, cudaStream_t s) {
    // persistent grid of lockstep blocks: every resident block slot once
    // (blocks claim units of LOCK_THREADS n-mers dynamically, LockPlan); the
    // variables%(gtext)s of the block's n-mers in dynamic shared memory
    auto kern = holder_lock_kernel<%(name)s_T, %(name)s_CC, %(mode)s>;
    block = %(name)s_T::LOCK_THREADS;
    const int smem = %(ncol)d * %(name)s_T::NVARS * %(name)s_T::LOCK_THREADS * (int)sizeof(double);
    static LaunchCache lc;
    int sms = 0, bps = 0;
    const int r = launch_facts(lc, kern, block, smem, smem, &sms, &bps);
    if (r) return r;
    const long need = (A.n + block - 1) / block * (A.split ? %(name)s_T::%(npieces)s : 1);
    grid = (int)(need < (long)sms * bps ? need : (long)sms * bps);
    if (grid < 1) grid = 1;
    kern<<<grid, block, smem, s>>>(A);
    return (int)cudaGetLastError();
}

int mbx_prime_%(name)s_%(v)s(cudaStream_t s) {
    // code prefetch of the %(what2)s: a launch of the evaluation kernel itself in its
    // prefetch mode (prime_pieces), one warp per SM, every piece run by at
    // least four of them
    auto kern = holder_lock_kernel<%(name)s_T, %(name)s_CC, %(mode)s>;
    const int smem_full = %(ncol)d * %(name)s_T::NVARS * %(name)s_T::LOCK_THREADS * (int)sizeof(double);
    const int smem = %(name)s_T::NVARS * %(name)s_T::LOCK_THREADS * (int)sizeof(double);
    static LaunchCache lc;
    int sms = 0, bps = 0;
    const int r = launch_facts(lc, kern, 0, smem_full, 0, &sms, &bps);
    if (r) return r;
    HolderArgs A;
    memset(&A, 0, sizeof(A));
    A.prime_npieces = %(name)s_T::%(npieces)s;
    A.prime_passes = (4 * A.prime_npieces + sms - 1) / sms;
    kern<<<sms, 32, smem, s>>>(A);
    return (int)cudaGetLastError();
}
"""

VARIANTS = {
    # variant: (description, body)
    "g": ("FP64 energy + gradient kernel", LOCK_LAUNCH % {
        "name": "%(name)s", "v": "g", "gtext": " and their gradient accumulators", "mode": "HM_GRAD_FP64",
        "ncol": 2, "what2": "FP64 gradient trie", "npieces": "NPIECES"}),
    "e": ("FP64 energy-only kernel", LOCK_LAUNCH % {
        "name": "%(name)s", "v": "e", "gtext": "", "mode": "HM_ENERGY",
        "ncol": 1, "what2": "FP64 energy trie", "npieces": "NPIECES_E"}),
}

# The adjoint unit of every evaluator: the variables of its n-mers for the
# coefficient adjoint (csrc/table_kernels.cu does the rest from the tables).
TABLE_TU = """// Generated by mbx_b200/codegen/gen_kernels.py -- do not edit.
// Variables of the %(name)s evaluator for the coefficient adjoint.
#include "../holder_kernel.cuh"
#include "%(name)s.cuh"

int mbx_launch_%(name)s_c(const HolderArgs& A, const double* w, long first, int count, double* wv, cudaStream_t s) {
    holder_wvars_kernel<%(name)s_T><<<(count + 127) / 128, 128, 0, s>>>(A, w, first, count, wv);
    return (int)cudaGetLastError();
}
"""

# Polynomials of at most this many terms (MBX_SMALL_TERMS) have their whole
# adjoint in one kernel.
SMALL_TERMS = 32
SMALL_TU = """
int mbx_launch_%(name)s_d(const HolderArgs& A, const double* w, const AdjointTable& P, double* part, unsigned* ticket,
                          double* out, int sms, cudaStream_t s) {
    static_assert(%(nterms)d <= MBX_SMALL_TERMS, "terms");
    const long need = (A.n + 127) / 128;
    const int grid = (int)(need < 2L * sms ? (need > 0 ? need : 1) : 2L * sms);
    holder_dcoef_small_kernel<%(name)s_T><<<grid, 128, 0, s>>>(A, w, P, part, ticket, out);
    return (int)cudaGetLastError();
}
"""

ONEBODY_TU = """// Generated by mbx_b200/codegen/gen_kernels.py -- do not edit.
// Table-driven 1-body kernel of the %(name)s evaluator.
#include <cstring>
#include "../holder_kernel.cuh"
#include "../launch_cache.cuh"
#include "%(name)s.cuh"

int mbx_launch_%(name)s_o(const HolderArgs& A, int grid, int block, cudaStream_t s) {
    // a lane per monomer; x and gradient columns of four warps in dynamic shared memory
    auto kern = onebody_table_kernel<%(name)s_T>;
    const int smem = 4 * 2 * %(name)s_T::NVARS * 32 * (int)sizeof(double);
    static LaunchCache lc;
    int sms = 0, bps = 0;
    const int r = launch_facts(lc, kern, 128, smem, smem, &sms, &bps);
    if (r) return r;
    if (A.n <= 0) return 0;
    const long need = (A.n + 127) / 128;
    const int g = (int)(need < (long)sms * bps ? need : (long)sms * bps);
    kern<<<g, 128, smem, s>>>(A);
    return (int)cudaGetLastError();
}
"""


def has_small_adjoint(name):
    return wtable(name).nterms <= SMALL_TERMS


def variants_of(name):
    from mbx_b200.specs import KERNEL_ALIASES
    if name in ONEBODY_SPECS:
        return "o"
    name = KERNEL_ALIASES.get(name, name)
    return "ge" + ("s" if name in SHIFT_TYPES else "") + "t"


QF_TU = """// Generated by mbx_b200/codegen/gen_kernels.py -- do not edit.
// Mixed-precision evaluation of the %(name)s polynomial on the tensor cores
// (quadratic form over the %(basis)s FP32 basis, csrc/qf_kernel.cuh).
#include <cuda_fp16.h>

#include <cmath>
#include <cstring>
#include <vector>
#include "../holder_kernel.cuh"
#include "../launch_cache.cuh"
#include "%(name)s.cuh"
#include "%(name)s_qf.cuh"

// b = F a: the basis coefficients are linear in the fitted ones.  Row j of F
// (entries sF_row[j] .. sF_row[j+1]) lists (k, factor); sF0 is the constant.
static const int sF_row_%(name)s[%(norb1)d] = {%(rows)s};
static const int sF_k_%(name)s[%(nnz)d] = {%(ks)s};
static const double sF_f_%(name)s[%(nnz)d] = {%(fs)s};
static const int sF0_k_%(name)s[%(nnz0)d] = {%(k0)s};
static const double sF0_f_%(name)s[%(nnz0)d] = {%(f0)s};
%(tables)s
// the same for the device
static __device__ const int dF_row_%(name)s[%(norb1)d] = {%(rows)s};
static __device__ const int dF_k_%(name)s[%(nnz)d] = {%(ks)s};
static __device__ const double dF_f_%(name)s[%(nnz)d] = {%(fs)s};
static __device__ const int dF0_k_%(name)s[%(nnz0)d] = {%(k0)s};
static __device__ const double dF0_f_%(name)s[%(nnz0)d] = {%(f0)s};
%(dtables)s
// IEEE binary16 of x, rounded to nearest even (subnormals kept; |x| < 65504 here)
static unsigned short qf_half(double x) {
    const unsigned short sign = std::signbit(x) ? 0x8000 : 0;
    const double a = std::fabs(x);
    if (a == 0.0) return sign;
    int e;
    const double f = std::frexp(a, &e);   // a = f 2^e, f in [0.5, 1)
    if (e >= -13) {                        // normal: a >= 2^-14
        double m = std::nearbyint(std::ldexp(f, 11));
        if (m == 2048.0) {
            m = 1024.0;
            ++e;
        }
        return (unsigned short)(sign | ((e + 14) << 10) | ((int)m - 1024));
    }
    return (unsigned short)(sign | (int)std::nearbyint(std::ldexp(a, 24)));   // subnormal: m 2^-24
}

static double qf_half_value(unsigned short h) {
    const int e = (h >> 10) & 0x1f, m = h & 0x3ff;
    const double v = e ? std::ldexp(1024.0 + m, e - 25) : std::ldexp((double)m, -24);
    return (h & 0x8000) ? -v : v;
}

// The tensor-core operands for fitted coefficients a: the C' image in the
// kernel's layout (%(name)s_Q::IMAGE_BYTES bytes), the column factors
// 2^-(s_j + t_j) (NB floats) and the constant term.  Host only.
int mbx_qf_image_%(name)s(const double* a, unsigned char* img, float* colf, double* b0_out) {
    constexpr int NB = %(name)s_Q::NB;
    std::vector<double> b(%(norb)d);
    for (int j = 0; j < %(norb)d; ++j) {
        double acc = 0.0;
        for (int q = sF_row_%(name)s[j]; q < sF_row_%(name)s[j + 1]; ++q) acc += sF_f_%(name)s[q] * a[sF_k_%(name)s[q]];
        b[j] = acc;
    }
    double b0 = 0.0;
    for (int q = 0; q < %(nnz0)d; ++q) b0 += sF0_f_%(name)s[q] * a[sF0_k_%(name)s[q]];
    *b0_out = b0;
    // C (symmetric), then C' = D C D, D = diag(2^t)
    std::vector<double> C((size_t)NB * NB, 0.0);
    for (int q = 0; q < qf_nmono_%(name)s; ++q) {
        const int i = qf_mi_%(name)s[q], j = qf_mj_%(name)s[q];
        const double c = b[qf_mo_%(name)s[q]];
        if (i == j) {
            C[(size_t)i * NB + i] += c;
        } else {
            C[(size_t)i * NB + j] += 0.5 * c;
            C[(size_t)j * NB + i] += 0.5 * c;
        }
    }
    for (int i = 0; i < NB; ++i)
        for (int j = 0; j < NB; ++j) C[(size_t)i * NB + j] = std::ldexp(C[(size_t)i * NB + j], qf_t_%(name)s[i] + qf_t_%(name)s[j]);
    // column exponents: largest |C'_ij 2^s_j| of a column below 2^14
    std::vector<int> sj(NB, 0);
    for (int j = 0; j < NB; ++j) {
        double m = 0.0;
        for (int i = 0; i < NB; ++i) m = std::fmax(m, std::fabs(C[(size_t)i * NB + j]));
        if (m > 0.0) {
            int e;
            std::frexp(m, &e);        // floor(log2 m) = e - 1
            sj[j] = 14 - e;
        }
        colf[j] = (float)std::ldexp(1.0, -(sj[j] + qf_t_%(name)s[j]));
    }
    // K block s, pass p (columns pass_col(p) .. + pass_n(p)): B[n][k] =
    // C'_kn 2^s_n in hi, mid[, lo] FP16 parts of pass_n(p) rows x 16, core
    // matrix (n' / 8, k / 8) of a part at (n' / 8) 128 + (k / 8) (pass_n / 8) 128
    // (row groups contiguous), row n' %% 8 at 16 (n' %% 8), n' = n - pass_col(p)
    memset(img, 0, (size_t)%(name)s_Q::IMAGE_BYTES);
    for (int s = 0; s < %(name)s_Q::KS; ++s) {
        const int parts = %(name)s_Q::parts(s);
        for (int p = 0; p < %(name)s_Q::NPASS; ++p) {
            const int width = %(name)s_Q::pass_n(p), c0 = %(name)s_Q::pass_col(p);
            unsigned char* st = img + %(name)s_Q::chunk_offset(s, p);
            for (int nn = 0; nn < width; ++nn)
                for (int kk = 0; kk < 16; ++kk) {
                    const int k = 16 * s + kk, n = c0 + nn;
                    double x = std::ldexp(C[(size_t)k * NB + n], sj[n]);
                    const size_t off = (size_t)(nn / 8) * 128 + (size_t)(kk / 8) * (width / 8) * 128 + (nn %% 8) * 16 +
                                       (kk %% 8) * 2;
                    for (int pt = 0; pt < parts; ++pt) {
                        const unsigned short h = qf_half(x);
                        memcpy(st + (size_t)pt * width * 32 + off, &h, 2);
                        x -= qf_half_value(h);
                    }
                }
        }
    }
    return 0;
}

// The same on the device (mbx_set_coefficients): the steps of the host
// builder above, operation for operation (every product and sum rounded on
// its own), so that both write the same bytes.
static __device__ double qfd_a_%(name)s[%(ncoef)d], qfd_b_%(name)s[%(norb)d];
static __device__ double qfd_C_%(name)s[%(name)s_Q::NB * %(name)s_Q::NB];
static __device__ int qfd_sj_%(name)s[%(name)s_Q::NB];
static __device__ float qfd_colf_%(name)s[%(name)s_Q::NB];   // to constant memory by a copy
static __device__ double qfd_b0_%(name)s[1];

// a warp per row; the products of a row are added in order, as on the host
__global__ void __launch_bounds__(128) k_qf_b_%(name)s() {
    __shared__ double stage[4][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, j = blockIdx.x * 4 + w;
    if (j > %(norb)d) return;
    const bool c0 = j == %(norb)d;   // the constant term
    const int b = c0 ? 0 : dF_row_%(name)s[j], e = c0 ? %(nnz0)d : dF_row_%(name)s[j + 1];
    double acc = 0.0;
    for (int q0 = b; q0 < e; q0 += 32) {
        const int q = q0 + lane;
        double p = -0.0;   // (adding it changes nothing)
        if (q < e)
            p = c0 ? __dmul_rn(dF0_f_%(name)s[q], qfd_a_%(name)s[dF0_k_%(name)s[q]])
                   : __dmul_rn(dF_f_%(name)s[q], qfd_a_%(name)s[dF_k_%(name)s[q]]);
        stage[w][lane] = p;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 32; ++i) acc = __dadd_rn(acc, stage[w][i]);
        __syncwarp();
    }
    if (lane == 0) (c0 ? qfd_b0_%(name)s[0] : qfd_b_%(name)s[j]) = acc;
}

// C' = D C D from zeroed C: every monomial has an entry (i, j) of its own
__global__ void k_qf_c_%(name)s() {
    constexpr int NB = %(name)s_Q::NB;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= dqf_nmono_%(name)s) return;
    const int i = dqf_mi_%(name)s[q], j = dqf_mj_%(name)s[q];
    const double c = qfd_b_%(name)s[dqf_mo_%(name)s[q]];
    const int t = dqf_t_%(name)s[i] + dqf_t_%(name)s[j];
    const double v = ldexp(i == j ? c : 0.5 * c, t);
    qfd_C_%(name)s[i * NB + j] = v;
    qfd_C_%(name)s[j * NB + i] = v;
}

// column exponents and factors: a warp per column
__global__ void k_qf_cols_%(name)s() {
    constexpr int NB = %(name)s_Q::NB;
    const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (j >= NB) return;
    double m = 0.0;
    for (int i = lane; i < NB; i += 32) m = fmax(m, fabs(qfd_C_%(name)s[j * NB + i]));   // (C is symmetric)
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane) return;
    int sj = 0;
    if (m > 0.0) {
        int e;
        frexp(m, &e);
        sj = 14 - e;
    }
    qfd_sj_%(name)s[j] = sj;
    qfd_colf_%(name)s[j] = (float)ldexp(1.0, -(sj + dqf_t_%(name)s[j]));
}

// the image: a thread per (K block, column, k)
__global__ void k_qf_image_%(name)s() {
    constexpr int NB = %(name)s_Q::NB;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= %(name)s_Q::KS * NB * 16) return;
    const int kk = idx %% 16, n = idx / 16 %% NB, s = idx / (16 * NB);
    int p = 0;
    while (p + 1 < %(name)s_Q::NPASS && n >= %(name)s_Q::pass_col(p + 1)) ++p;
    const int width = %(name)s_Q::pass_n(p), nn = n - %(name)s_Q::pass_col(p);
    double x = ldexp(qfd_C_%(name)s[(16 * s + kk) * NB + n], qfd_sj_%(name)s[n]);
    unsigned char* st = qf_img_%(name)s + %(name)s_Q::chunk_offset(s, p);
    const size_t off = (size_t)(nn / 8) * 128 + (size_t)(kk / 8) * (width / 8) * 128 + (nn %% 8) * 16 + (kk %% 8) * 2;
    const int parts = %(name)s_Q::parts(s);
    for (int pt = 0; pt < parts; ++pt) {
        const __half h = __double2half(x);
        *reinterpret_cast<__half*>(st + (size_t)pt * width * 32 + off) = h;
        x -= (double)__half2float(h);
    }
}

int mbx_set_coef_%(name)s_s(const double* a, int from_device, cudaStream_t s) {
    cudaError_t e = cudaMemcpyToSymbolAsync(qfd_a_%(name)s, a, sizeof(double) * %(ncoef)d, 0,
                                            from_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s);
    void *C = nullptr, *colf = nullptr, *b0 = nullptr;
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&C, qfd_C_%(name)s);
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&colf, qfd_colf_%(name)s);
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&b0, qfd_b0_%(name)s);
    if (e == cudaSuccess) e = cudaMemsetAsync(C, 0, sizeof(qfd_C_%(name)s), s);
    if (e != cudaSuccess) return (int)e;
    constexpr int NB = %(name)s_Q::NB;
    k_qf_b_%(name)s<<<(%(norb)d + 4) / 4, 128, 0, s>>>();
    k_qf_c_%(name)s<<<(qf_nmono_%(name)s + 127) / 128, 128, 0, s>>>();
    k_qf_cols_%(name)s<<<(NB * 32 + 127) / 128, 128, 0, s>>>();
    k_qf_image_%(name)s<<<(%(name)s_Q::KS * NB * 16 + 127) / 128, 128, 0, s>>>();
    e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbolAsync(qf_colf_%(name)s, colf, sizeof(float) * NB, 0, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(qf_b0_%(name)s, b0, sizeof(double), 0, cudaMemcpyDeviceToDevice, s);
    return (int)e;
}

// The operands as they are on the current device.
int mbx_qf_device_image_%(name)s(unsigned char* img, float* colf, double* b0) {
    cudaError_t e = cudaMemcpyFromSymbol(img, qf_img_%(name)s, (size_t)%(name)s_Q::IMAGE_BYTES);
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(colf, qf_colf_%(name)s, sizeof(float) * %(name)s_Q::NB);
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(b0, qf_b0_%(name)s, sizeof(double));
    return (int)e;
}

int mbx_launch_%(name)s_s(const HolderArgs& A, int grid, int block, cudaStream_t s) {
    // three kernels: the FP64 variables shifted to the FP32 basis at full
    // occupancy (pair_vars_kernel), the quadratic form on the tensor cores
    // (qf_eval_kernel: one CTA per SM, persistent over tiles of 128 n-mers),
    // the FP64 chain rule and sums at full occupancy (pair_finish_kernel);
    // A.ps holds the scratch between them (capacity A.ps.cap >= A.n)
    if (!A.ps.dx || !A.ps.q || A.ps.cap < A.n) return (int)cudaErrorInvalidValue;
    auto kern = qf_eval_kernel<%(name)s_T, %(name)s_Q>;
    static LaunchCache lc;
    int sms = 0, bps = 0;
    const int r = launch_facts(lc, kern, qf::THREADS, qf::Layout<%(name)s_Q>::SMEM, qf::Layout<%(name)s_Q>::SMEM, &sms,
                               &bps);
    if (r) return r;
    const long wide = (long)sms * 16;
    const long gv = (A.n + 255) / 256, gf = (A.n + 127) / 128;
    pair_vars_kernel<%(name)s_T><<<(int)(gv < wide ? (gv > 0 ? gv : 1) : wide), 256, 0, s>>>(A);
    const long tiles = (A.n + 127) / 128;
    grid = (int)(tiles < (long)sms ? (tiles > 0 ? tiles : 1) : sms);
    kern<<<grid, qf::THREADS, qf::Layout<%(name)s_Q>::SMEM, s>>>(A);
    pair_finish_kernel<%(name)s_T><<<(int)(gf < wide ? (gf > 0 ? gf : 1) : wide), 128, 0, s>>>(A);
    return (int)cudaGetLastError();
}

int mbx_prime_%(name)s_s(cudaStream_t) {
    return 0;   // the tensor-core kernel's code is small: nothing to prefetch
}
"""


def write_qf_tu(name, path):
    from mbx_b200.codegen import qf
    sp = shifted_pip(name)
    q = qf.QuadForm(name, sp)
    rows, ks, fs = [0], [], []
    for row in sp.F:
        for k, f in sorted(row.items()):
            ks.append(k)
            fs.append(f)
        rows.append(len(ks))
    k0 = sorted(sp.const_F)
    d = {"name": name, "basis": SHIFT_TYPES[name], "norb": sp.norb, "norb1": sp.norb + 1,
         "ncoef": SPECS[name].ncoef, "nnz": len(ks), "nnz0": max(1, len(k0)),
         "rows": ",".join(map(str, rows)), "ks": ",".join(map(str, ks)),
         "fs": ",".join(repr(float(f)) for f in fs),
         "k0": ",".join(map(str, k0)) if k0 else "0",
         "f0": ",".join(repr(float(sp.const_F[k])) for k in k0) if k0 else "0.0",
         "tables": qf.emit_tables(q, name, "static const", "qf"),
         "dtables": qf.emit_tables(q, name, "static __device__ const", "dqf")}
    write_tu(path, QF_TU % d)


def write_tu(path, text):
    old = open(path).read() if os.path.exists(path) else None
    if old != text:
        with open(path, "w") as f:
            f.write(text)


def write_kernels_cu(name):
    paths = []
    inc = {"g": "pip", "e": "pip_e"}
    if name in ONEBODY_SPECS:
        path = os.path.join(OUT, "%s_t.cu" % name)
        write_tu(path, ONEBODY_TU % {"name": name})
        return [path]
    spec = SPECS[name]
    for v in variants_of(name):
        if v == "s":
            path = os.path.join(OUT, "%s_s.cu" % name)
            write_qf_tu(name, path)
            paths.append(path)
            continue
        path = os.path.join(OUT, "%s_%s.cu" % (name, v))
        if v == "t":
            small = SMALL_TU % {"name": name, "nterms": wtable(name).nterms} if has_small_adjoint(name) else ""
            write_tu(path, TABLE_TU % {"name": name} + small)
        else:
            what, body = VARIANTS[v]
            wt = wtable(name)
            by_leaf = wt.nterms <= LEAF_ORDER_TERMS
            d = {"name": name, "v": v, "what": what, "pip": inc[v], "nc": wt.nterms if by_leaf else wt.ncoef,
                 "include": '#include "%s_%s.cuh"\n' % (name, inc[v])}
            d["setter"] = (SET_LEAF if by_leaf else SET_ORBIT) % d
            write_tu(path, (TU_HEAD + body) % d)
        paths.append(path)
    return paths


def term_runs(vars_):
    """(variable, exponent) runs of a term's variable list, in order."""
    runs = []
    for v in vars_:
        if runs and runs[-1][0] == v:
            runs[-1][1] += 1
        else:
            runs.append([v, 1])
    return runs


@__import__("functools").lru_cache(maxsize=None)
def _table_runs(table_name):
    t = wtable_by_key(table_name)
    return [term_runs(t.var[q, :t.deg[q]].tolist()) for q in range(t.nterms)]


def term_pairs_max(table_name):
    return max(1, max(len(r) for r in _table_runs(table_name)))


def table_names():
    """Keys of the term tables in registry order (evaluators with the same
    key share an entry), the plain tables of the evaluators with a reference
    point (for caller-supplied variables), the 1-body evaluators' last."""
    from mbx_b200.specs import KERNEL_ALIASES
    names = []
    kern = [KERNEL_ALIASES.get(n, n) for n in SPECS]
    for key in [table_key(n) for n in kern] + [SPECS[n].pip_table for n in kern] + \
            [table_key(n) for n in ONEBODY_SPECS]:
        if key not in names:
            names.append(key)
    return names


def write_term_tables():
    """Every polynomial's term table in the w variables (csrc/term_table.cuh
    encoding), its coefficient map c = F a and its transform w = W x, in one
    binary file, embedded in the library by terms_blob.cpp (.incbin), plus
    the index of the tables."""
    blob = bytearray()
    index = []

    def put(array):
        off = len(blob)
        blob.extend(array.tobytes())
        blob.extend(b"\0" * (-len(blob) % 16))
        return off

    def csr(rows):
        """(row starts, columns, factors) of rows {column: factor}"""
        start = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
        return (start, np.array([k for r in rows for k in r], np.int32),
                np.array([f for r in rows for f in r.values()], np.float64))

    for tname in table_names():
        t = wtable_by_key(tname)
        runs = _table_runs(tname)
        words = np.zeros((t.nterms, 4), np.int32)
        words[:, 0] = t.k
        for q, rr in enumerate(runs):
            if len(rr) > 6:
                raise ValueError("%s term %d has more than six distinct variables" % (tname, q))
            packed = [0, 0, 0]
            for i in range(6):
                v, e = (rr[i] if i < len(rr) else (255, 0))
                if not (0 <= v < 255 and 0 < e < 256) and v != 255:
                    raise ValueError("%s term %d: variable %d exponent %d out of range" % (tname, q, v, e))
                packed[i >> 1] |= ((v & 255) | (e << 8)) << (16 * (i & 1))
            for j in range(3):
                words[q, 1 + j] = packed[j] - (1 << 32) if packed[j] >= 1 << 31 else packed[j]
        offs = [put(words), put(np.ascontiguousarray(t.coef, np.float64))]
        fr, fk, ff = csr(t.F)
        offs += [put(fr), put(fk), put(ff)]
        for M in (t.W, t.W.T):
            wr, wk, wf = csr([{v: M[i, v] for v in range(t.nvars) if M[i, v] != 0.0} for i in range(t.nvars)])
            # column v with sign s as s (v + 1)
            offs += [put(wr), put(((wk + 1) * wf).astype(np.int32))]
        offs.append(put(np.ascontiguousarray(t.w0, np.float64)))
        # half-monomials of the coefficient adjoint: up to three (variable,
        # exponent) byte pairs each (255: unused), and per term its two of them
        basis, pairs = t.halves
        half = np.zeros((len(basis), 2), np.int32)
        for i, m in enumerate(basis):
            rr = term_runs(list(m))
            if len(rr) > 3:
                raise ValueError("%s: half-monomial %s has more than three distinct variables" % (tname, m))
            rr = rr + [(255, 0)] * (3 - len(rr))
            half[i] = [sum(v << (8 * n) for n, (v, _) in enumerate(rr)), sum(e << (8 * n) for n, (_, e) in enumerate(rr))]
        # (terms in the order of their first half: a warp's lanes share it)
        by_half = sorted(range(t.nterms), key=lambda q: pairs[q])
        offs += [put(half), put(np.array([pairs[q][0] | (pairs[q][1] << 16) for q in by_half], np.int32)),
                 put(np.array(by_half, np.int32))]
        # first term of every coefficient (the table is sorted by them), and F
        # transposed
        offs.append(put(np.searchsorted(t.k, np.arange(t.ncoef + 1)).astype(np.int32)))
        by_k = [{} for _ in range(t.nfit)]
        for j, row in enumerate(t.F):
            for k, f in row.items():
                by_k[k][j] = f
        offs += [put(a) for a in csr(by_k)]
        index.append((tname, t.nterms, term_pairs_max(tname), t.ncoef, len(basis), offs))
    bin_path = os.path.join(OUT, "terms.bin")
    old = open(bin_path, "rb").read() if os.path.exists(bin_path) else None
    if old != bytes(blob):
        with open(bin_path, "wb") as f:
            f.write(bytes(blob))
    lines = ["// Generated by mbx_b200/codegen/gen_kernels.py -- do not edit.", "#pragma once",
             "// term tables in terms.bin: name, number of terms, (variable, exponent) pairs per",
             "// term at most, coefficients in the w variables; byte offsets of the int4 terms, the",
             "// double signs, the rows of F (starts, columns, factors), of W and of its transpose",
             "// (starts, signed columns), of w0, of the half-monomials, of the terms' pairs of them (by",
             "// the first one) and the terms in that order, of the",
             "// first term of every coefficient and of the rows of F transposed",
             "struct TermTableInfo { const char* name; long nterms; int pairs, ncw, nhalf; long off_terms, off_tcoef, "
             "off_frow, off_fk, off_ff, off_wrow, off_w, off_wtrow, off_wt, off_w0, off_half, off_pair, off_term, "
             "off_first, off_ftrow, off_ftk, off_ftf; };",
             "static const TermTableInfo mbx_term_tables[] = {"]
    for tname, nt, npair, ncw, nhalf, offs in index:
        lines.append('    {"%s", %d, %d, %d, %d, %s},' % (tname, nt, npair, ncw, nhalf, ", ".join(map(str, offs))))
    lines.append("};")
    lines.append("static const int mbx_num_term_tables = %d;" % len(index))
    lines.append("static const long mbx_terms_bytes = %d;" % len(blob))
    write_tu(os.path.join(OUT, "terms_index.inc"), "\n".join(lines) + "\n")
    # the binary is referenced by absolute path (generated per checkout)
    write_tu(os.path.join(OUT, "terms_blob.cpp"),
             "// Generated by mbx_b200/codegen/gen_kernels.py -- do not edit.\n"
             "// The term tables of every evaluator (terms.bin), embedded read-only.\n"
             "__asm__(\".section .rodata\\n\"\n"
             "        \".balign 16\\n\"\n"
             "        \".globl mbx_terms_blob\\n\"\n"
             "        \".type mbx_terms_blob, @object\\n\"\n"
             "        \"mbx_terms_blob:\\n\"\n"
             "        \".incbin \\\"%s\\\"\\n\"\n"
             "        \".size mbx_terms_blob, %d\\n\"\n"
             "        \".previous\\n\");\n" % (bin_path, len(blob)))


def write_ps1b():
    """The Partridge-Schwenke polynomial sums of the water 1-body term
    (mbx_b200/data/ps1b.json, extracted by codegen/onebody_extract.py) as
    straight-line code: for every term j of ps::pot_nasa's loop
    (potential/1b/ps.cpp:455-476) the four sums with the term's indices and
    coefficient as literals, every product and sum rounded on its own in the
    reference's operand order."""
    import json
    d = json.load(open(os.path.join(PKG, "data", "ps1b.json")))
    L = ["// Generated by mbx_b200/codegen/gen_kernels.py from mbx_b200/data/ps1b.json -- do not edit.",
         "#pragma once",
         "#define PS1B_REOH %s" % lit(d["reoh"]), "#define PS1B_B1 %s" % lit(d["b1"]),
         "#define PS1B_ROH %s" % lit(d["roh"]), "#define PS1B_ALPHAOH %s" % lit(d["alphaoh"]),
         "#define PS1B_PHH2 %s" % lit(d["phh2"]), "#define PS1B_DEOH %s" % lit(d["deoh"]),
         "#define PS1B_PHH1 %s" % lit(d["phh1"]), "#define PS1B_COSTHE %s" % lit(d["costhe"]),
         "#define PS1B_OFFSET %s" % lit(d["offset"]), "#define PS1B_CM1_KCALMOL %s" % lit(d["cm1_kcalmol"]),
         "#define PS1B_C0 %s" % lit(d["c5z"][0]),
         "__device__ __forceinline__ void ps1b_sums(const double (&f0)[16], const double (&f1)[16], "
         "const double (&f2)[16], double& s0, double& s1, double& s2, double& s3) {"]
    M, A = "__dmul_rn", "__dadd_rn"
    for j in range(1, len(d["c5z"])):
        I, J, K = d["idx1"][j], d["idx2"][j], d["idx3"][j]
        c = lit(d["c5z"][j])
        sym = "%s(%s(f0[%d], f1[%d]), %s(f0[%d], f1[%d]))" % (A, M, I, J, M, J, I)
        L.append("    { const double sym = %s;" % sym)
        L.append("      s0 = %s(s0, %s(%s(%s, sym), f2[%d]));" % (A, M, M, c, K))
        t1 = "%s(%s(%s(%s, f0[%d]), f1[%d]), %s(%s(%s, f0[%d]), f1[%d]))" % (
            A, M, M, lit(float(I - 1)), I - 1, J, M, M, lit(float(J - 1)), J - 1, I)
        L.append("      s1 = %s(s1, %s(%s(%s, %s), f2[%d]));" % (A, M, M, c, t1, K))
        t2 = "%s(%s(%s(%s, f0[%d]), f1[%d]), %s(%s(%s, f0[%d]), f1[%d]))" % (
            A, M, M, lit(float(J - 1)), I, J - 1, M, M, lit(float(I - 1)), J, I - 1)
        L.append("      s2 = %s(s2, %s(%s(%s, %s), f2[%d]));" % (A, M, M, c, t2, K))
        L.append("      s3 = %s(s3, %s(%s(%s(%s, sym), %s), f2[%d])); }" % (A, M, M, M, c, lit(float(K - 1)), K - 1))
    L.append("}")
    write_tu(os.path.join(OUT, "ps1b.inc"), "\n".join(L) + "\n")


def write_registry():
    """Host tables: evaluator descriptions and default coefficients."""
    from mbx_b200.tables import load_fit
    from mbx_b200.specs import KERNEL_ALIASES
    lines = ["// Generated by mbx_b200/codegen/gen_kernels.py -- do not edit.", "#pragma once",
             '#include "../holder_kernel.cuh"', ""]
    for name in SPECS:
        vs = variants_of(name)
        if name in KERNEL_ALIASES:
            vs = ""   # runs the kernels of KERNEL_ALIASES[name], declared there
        for v in "ges":
            if v in vs:
                lines.append("int mbx_launch_%s_%s(const HolderArgs& A, int grid, int block, cudaStream_t s);" %
                             (name, v))
                lines.append("int mbx_prime_%s_%s(cudaStream_t s);" % (name, v))
                lines.append("int mbx_set_coef_%s_%s(const double* a, int from_device, cudaStream_t s);" % (name, v))
        if "t" in vs:
            lines.append("int mbx_launch_%s_c(const HolderArgs& A, const double* w, long first, int count, double* wv, "
                         "cudaStream_t s);" % name)
            if has_small_adjoint(name):
                lines.append("int mbx_launch_%s_d(const HolderArgs& A, const double* w, const AdjointTable& P, "
                             "double* part, unsigned* ticket, double* out, int sms, cudaStream_t s);" % name)
        fit = load_fit(name)
        lines.append("static const double mbx_fit_%s[%d] = {" % (name, len(fit)))
        for i in range(0, len(fit), 4):
            lines.append("    " + ", ".join(repr(float(x)) for x in fit[i:i + 4]) + ",")
        lines.append("};")
    lines.append("")
    names = list(SPECS)
    tables = table_names()
    lines.append("static const EvaluatorInfo mbx_evaluators[] = {")
    for name, spec in SPECS.items():
        vs = variants_of(name)
        kern = KERNEL_ALIASES.get(name, name)
        ids = list(spec.monomers) + ["", ""][:3 - len(spec.monomers)]
        skip = {"pair_gt": 0, "two_of_three_gt": 1, "all_three_gt": 2}[spec.skip]

        def fn(v, kind):
            # the table unit ("t") holds the coefficient adjoint ("c")
            have = ("t" in vs) if v == "c" else (v in vs)
            return ("mbx_%s_%s_%s" % (kind, kern, v)) if have else "nullptr"
        small = "mbx_launch_%s_d" % kern if has_small_adjoint(kern) else "nullptr"
        lines.append('    {"%s", %d, {"%s", "%s", "%s"}, %s, %d, %d, %d, %d, mbx_fit_%s, %s, %s, %s, %s, %s, %s,' %
                     (name, spec.nbody, ids[0], ids[1], ids[2], lit(spec.rf), skip, spec.ncoef, spec.nreal,
                      spec.nvars, name, fn("g", "launch"), fn("e", "launch"), fn("c", "launch"), small,
                      fn("s", "launch"), lit(MIXED_FP64_RADIUS.get(name, 0.0))))
        lines.append("     %s, %s, %s," % (fn("g", "prime"), fn("e", "prime"), fn("s", "prime")))
        lines.append("     {%s}, %s, %d, %d, %d}," %
                     (", ".join(fn(v, "set_coef") for v in "ge"), fn("s", "set_coef"),
                      tables.index(table_key(kern)), tables.index(SPECS[kern].pip_table), names.index(kern)))
    lines.append("};")
    lines.append("static const int mbx_num_evaluators = %d;" % len(SPECS))
    # host builders of the tensor-core operands of the mixed mode (QF_TYPES)
    from mbx_b200.codegen import qf as qfmod
    lines.append("struct QfInfo { const char* name; long image_bytes; int nb; "
                 "int (*build)(const double*, unsigned char*, float*, double*); "
                 "int (*device)(unsigned char*, float*, double*); };")
    for name in sorted(QF_TYPES):
        lines.append("int mbx_qf_image_%s(const double* a, unsigned char* img, float* colf, double* b0);" % name)
        lines.append("int mbx_qf_device_image_%s(unsigned char* img, float* colf, double* b0);" % name)
    lines.append("static const QfInfo mbx_qf_types[] = {")
    for name in sorted(QF_TYPES):
        q = qfmod.QuadForm(name, shifted_pip(name))
        lines.append('    {"%s", %dL, %d, mbx_qf_image_%s, mbx_qf_device_image_%s},' %
                     (name, qfmod.image_bytes(q), q.npad, name, name))
    lines.append("};")
    lines.append("static const int mbx_num_qf_types = %d;" % len(QF_TYPES))
    # 1-body evaluators (table-driven), by monomer id
    from mbx_b200.specs import ONEBODY_DISPATCH
    lines.append("struct OneBodyInfo { const char* name; const char* mon; int ncoef; const double* fit; int table; "
                 "int (*launch)(const HolderArgs&, int, int, cudaStream_t); };")
    for name, sp in ONEBODY_SPECS.items():
        lines.append("int mbx_launch_%s_o(const HolderArgs& A, int grid, int block, cudaStream_t s);" % name)
        fit = load_fit(name)
        lines.append("static const double mbx_fit_%s[%d] = {%s};" %
                     (name, len(fit), ", ".join(repr(float(x)) for x in fit)))
    mon_of = {v: k for k, v in ONEBODY_DISPATCH.items()}
    lines.append("static const OneBodyInfo mbx_onebody[] = {%s};" % ", ".join(
        '{"%s", "%s", %d, mbx_fit_%s, %d, mbx_launch_%s_o}' %
        (name, mon_of[name], sp.ncoef, name, tables.index(table_key(name)), name)
        for name, sp in ONEBODY_SPECS.items()))
    lines.append("static const int mbx_num_onebody = %d;" % len(ONEBODY_SPECS))
    # real atoms per monomer id (SetUpMonomers, bblock/sys_tools.cpp:133-254)
    from mbx_b200.specs import MONOMER_ATOMS
    lines.append("struct MonomerInfo { const char* id; int nat; };")
    lines.append("static const MonomerInfo mbx_monomers[] = {%s};" %
                 ", ".join('{"%s", %d}' % (m, n) for m, n in MONOMER_ATOMS.items()))
    lines.append("static const int mbx_num_monomers = %d;" % len(MONOMER_ATOMS))
    write_tu(os.path.join(OUT, "registry.inc"), "\n".join(lines) + "\n")


def main(argv=None, quiet=False):
    """Writes every generated file; returns the translation units to compile."""
    ap = argparse.ArgumentParser()
    ap.add_argument("names", nargs="*", default=list(SPECS))
    args = ap.parse_args(argv)
    os.makedirs(OUT, exist_ok=True)
    prepare_tables(table_names())
    write_registry()
    write_term_tables()
    write_ps1b()
    from mbx_b200.specs import KERNEL_ALIASES
    keep = {"registry.inc", "terms_index.inc", "terms.bin", "terms_blob.cpp", "ps1b.inc"}
    if args.names == list(SPECS):
        args.names = list(SPECS) + list(ONEBODY_SPECS)
    for n in args.names:
        if n in KERNEL_ALIASES:
            continue
        path, leaves, inner = generate(n)
        keep.add(os.path.basename(path))
        if n in SPECS:
            for v in ("pip", "pip_e", "qf"):
                keep.add("%s_%s.cuh" % (n, v))
        keep.update(os.path.basename(p) for p in write_kernels_cu(n))
        if not quiet:
            print("%s: %d leaves, %d inner -> %s" % (n, leaves, inner, path))
    if args.names == list(SPECS) + list(ONEBODY_SPECS):
        # drop the units of an earlier generation (other variants or types)
        for f in os.listdir(OUT):
            if f not in keep:
                os.remove(os.path.join(OUT, f))
    return sorted(os.path.join(OUT, f) for f in os.listdir(OUT) if f.endswith((".cu", ".cpp")))


if __name__ == "__main__":
    main()
