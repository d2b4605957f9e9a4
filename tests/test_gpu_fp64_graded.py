"""FP64 products whose rows are graded against their columns: the largest elements of a row meet the smallest of a column, so
that a row's power of two says little about the sum.  The digit products keep FP64's error bound there by leaving such
elements to FP64 FMAs, one by one or piece by piece, with and without accumulation."""
import numpy as np
import pytest

from helpers import rel_err
from test_gpu_fp64_products import arrays, products, run

pytestmark = pytest.mark.gpu


def check(x, terms, what):
    """x against extended precision within the bound of an FP64 FMA chain, element by element.  The digits of an element that
    keeps them are off by at most K 2^-58.9 of the two powers of two, and its sum of magnitudes is at least 2^-6 of those:
    K 2^-53 of that sum and one rounding."""
    K = sum(A.shape[1] for _, A, _ in terms)
    ref, mag = np.zeros(x.shape, np.longdouble), np.zeros(x.shape)
    for s, A, B in terms:
        ref += s * (A.astype(np.longdouble) @ B.astype(np.longdouble))
        mag += np.abs(A) @ np.abs(B)
    tol = (K + 1) * 2.0 ** -53 * mag + 2.0 ** -52 * np.abs(ref).astype(float)
    bad = np.abs(x - ref) > tol
    assert not np.any(bad), (what, x.shape, K, int(bad.sum()), float(np.max(np.abs(x - ref)[bad] / tol[bad])))


@pytest.mark.parametrize("emax,lmax", [(5, 5), (6, 4), (7, 7)])
@pytest.mark.parametrize("kind", ["opposed", "spikes", "zeros"])
def test_rows_graded_against_columns(built_lib, emax, lmax, kind):
    from imsrg_gb300 import Engine, make_basis
    eng = Engine(make_basis(emax, lmax=lmax), device=0)
    rng = np.random.default_rng(emax)
    L, R = rng.standard_normal(eng.slab), rng.standard_normal(eng.slab)
    rows = arrays(eng)
    for row in rows:
        for o, n, m in row:
            l, r = L[o:o + n * m].reshape(m, n).T, R[o:o + n * m].reshape(m, n).T
            i, j = np.arange(n)[:, None], np.arange(m)[None]
            if kind == "opposed":  # every element of the products
                l *= np.ldexp(1.0, -(60 * j // max(m, 1)))
                r *= np.ldexp(1.0, -60 + 60 * i // max(n, 1))
            elif kind == "spikes":  # a few of each piece: a row's one large element meets a zero
                l *= np.where(j == i % max(m, 1), 2.0 ** 40, 1.0)
                r *= (i + j) % 23 != 0
            else:  # elements beyond the digits beside exact zeros
                l *= np.where((i + j) % 3 == 0, 2.0 ** 70, np.where((i + j) % 3 == 1, 1.0, 0.0))
                r *= np.where((i + 2 * j) % 3 == 0, 0.0, 1.0)
    got = run(eng, L, R, -1, 1)
    for k, row in enumerate(rows):
        for (w, g), terms in products(L, R, -1, 1, row).items():
            o, n, m = row[g]
            if n * m == 0 or terms[0][1].shape[1] == 0:
                continue
            cols = np.unique(np.linspace(0, m - 1, min(m, 12)).astype(int))
            check(got[w][o:o + n * m].reshape(m, n).T[:, cols], [(s, A, B[:, cols]) for s, A, B in terms], (k, w, g))


@pytest.mark.parametrize("emax", [5, 6])
def test_cross_coupled_products(built_lib, emax):
    from imsrg_gb300 import Engine, make_basis
    eng = Engine(make_basis(emax), device=0)
    rng = np.random.default_rng(emax)
    ops = [eng.new_op(h, rng.standard_normal(eng.slab) * np.ldexp(1.0, rng.integers(-90, 1, eng.slab))) for h in (-1, 1)]
    lcc, rcc, wcc, RES = eng.new_cc(0), eng.new_cc(0), eng.new_cc(1), eng.new_op(1)
    eng.calculate_cross_coupled(ops[0], lcc)
    eng.calculate_cross_coupled(ops[1], rcc)
    eng.commutator_222_ph(lcc, rcc, RES, wcc)
    l, r, w, info = lcc.download(), rcc.download(), wcc.download(), eng.cc_info()
    a = b = 0
    for q, (n, m) in enumerate(zip(info["rlen"], info["nph"])):
        n, m = int(n), int(m)
        if n * m:
            cols = np.unique(np.linspace(0, n - 1, min(n, 12)).astype(int))
            A, B = l[a:a + n * m].reshape(m, n).T, r[a:a + n * m].reshape(m, n)
            check(w[b:b + n * n].reshape(n, n).T[:, cols], [(1, A, B[:, cols])], q)
        a += n * m
        b += n * n


def test_accumulating_products(built_lib, oracles):
    """commutator_vjp: several terms added to one output, some of their elements left to FMAs.  The bound is the one that the
    transposes are held to elsewhere; an element added twice or left out is a hundredth of an array's largest."""
    from imsrg_gb300 import Engine, make_basis
    emax, hL, hR, hRES = 5, -1, 1, 1
    o, eng = oracles(emax), Engine(make_basis(emax), device=0)
    rng = np.random.default_rng(4)
    L, R, Cb = (rng.standard_normal(o.slab) * np.ldexp(1.0, rng.integers(-60, 1, o.slab)) for _ in range(3))
    ref = o.commutator_vjp(L, hL, R, hR, hRES, True, Cb)
    dL, dR, dC = eng.new_op(hL, L), eng.new_op(hR, R), eng.new_op(hRES, Cb)
    out = [eng.new_op(hL), eng.new_op(hR)]
    eng.commutator_vjp(dL, dR, dC, *out, True)
    for got, want in zip(out, ref):
        got = got.download()
        for row in arrays(eng):
            for at, n, m in row:
                if n * m:
                    assert rel_err(got[at:at + n * m], want[at:at + n * m]) < 1e-10
