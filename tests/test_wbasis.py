"""The symmetry-adapted form of the polynomials (codegen/wbasis.py) is the
polynomial: value at random variables and random coefficients against the term
table it was derived from, and every term is the product of its two
half-monomials.  CPU only."""
import numpy as np
import pytest

from mbx_b200.codegen import wbasis
from mbx_b200.specs import ONEBODY_SPECS, SPECS
from mbx_b200.tables import load_pip

NAMES = list({s.pip_table: n for n, s in list(SPECS.items()) + list(ONEBODY_SPECS.items())}.values())


def terms_of(table, c, x):
    v = np.where(table.var < 0, len(x), table.var)
    return c[table.k] * table.coef * np.append(x, 1.0)[v].prod(1)


@pytest.mark.parametrize("name", NAMES)
def test_w_polynomial_is_the_polynomial(name):
    table, w = load_pip(name), wbasis.wtable(name)
    rng = np.random.default_rng(3)
    for _ in range(3):
        x = rng.uniform(0.1, 1.2, table.nvars)
        a = rng.normal(size=table.ncoef)
        v = w.W @ x - w.w0
        direct = terms_of(table, a, x)
        t = terms_of(w, w.coefficients(a), v)
        # both are sums of at most nterms products of at most degree + 2
        # factors, each rounded to 2^-53
        bound = (table.degree + 4 + np.log2(table.nterms)) * 2.0 ** -53
        # and every w is rounded relative to its parts: |dw| <= 4 2^-53 (|W| |x|
        # + |w0|), which a term takes in proportion to dw / w of its factors
        dw = 4 * 2.0 ** -53 * (np.abs(w.W) @ np.abs(x) + np.abs(w.w0)) / np.abs(v)
        carried = np.append(dw, 0.0)[np.where(w.var < 0, len(x), w.var)].sum(1)
        assert abs(t.sum() - direct.sum()) <= 8 * bound * (np.abs(direct).sum() + np.abs(t).sum()) + \
            (np.abs(t) * carried).sum()


@pytest.mark.parametrize("name", NAMES)
def test_terms_are_products_of_their_halves(name):
    w = wbasis.wtable(name)
    basis, pairs = w.halves
    assert len(pairs) == w.nterms
    for t, (i, j) in enumerate(pairs):
        assert tuple(sorted(basis[i] + basis[j])) == tuple(w.var[t, :w.deg[t]])
