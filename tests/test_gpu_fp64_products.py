"""The grouped FP64 products (commutator_222_pp_hh's W1 / W2 in FP64): digit products on the tensor cores, and FP64 FMAs
where an operand is not finite.  Compared with extended-precision products of the same arrays, over bases whose channel
sizes fall on both sides of the kernels' tile edges, and over row scales from subnormal to near overflow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLASSES = [(0, 0), (0, 1), (0, 2), (1, 1), (2, 2), (1, 2)]


def arrays(eng):
    """(offset, n1, n2) of gam(1..6) of every channel."""
    b, info = eng.basis, eng.block_info()
    A, P = b.nholes, b.norbits - b.nholes
    at, out = 1 + A * A + P * P + P * A, []
    for q in range(eng.nblocks):
        n = [int(info[k][q]) for k in ("npp", "nph", "nhh")]
        row = []
        for c1, c2 in CLASSES:
            row.append((at, n[c1], n[c2]))
            at += n[c1] * n[c2]
        out.append(row)
    assert at == eng.slab
    return out


def products(L, R, hL, hR, row):
    """The terms of W1 and W2 of one channel: (array, op, [(sign, A, B)]) with A B summed over the inner index."""
    g = [(L[o:o + n * m].reshape(m, n).T, R[o:o + n * m].reshape(m, n).T) for o, n, m in row]
    (Lp, Rp), (Lb, Rb), (Lh, Rh), _, (Lx, Rx), (Ly, Ry) = g
    return {
        ("w1", 0): [(1, Lp, Rp)], ("w1", 4): [(hL, Lh.T, Rh)], ("w1", 2): [(1, Lp, Rh), (-1, Rp, Lh)],
        ("w1", 3): [(hL, Lb.T, Rb)], ("w1", 1): [(1, Lp, Rb), (-1, Rp, Lb)],
        ("w1", 5): [(hL, Lb.T, Rh), (-hR, Rb.T, Lh)],
        ("w2", 4): [(1, Lx, Rx)], ("w2", 0): [(hR, Lh, Rh.T)], ("w2", 2): [(1, Lh, Rx), (-1, Rh, Lx)],
        ("w2", 3): [(hR, Ly, Ry.T)], ("w2", 5): [(1, Ly, Rx), (-1, Ry, Lx)],
        ("w2", 1): [(hR, Lh, Ry.T), (-hL, Rh, Ly.T)],
    }


def run(eng, L, R, hL, hR):
    ops = [eng.new_op(hL, L), eng.new_op(hR, R), eng.new_op(-hL * hR), eng.new_op(1), eng.new_op(1)]
    eng.commutator_222_pp_hh(*ops)
    eng.synchronize()
    return {"w1": ops[3].download(), "w2": ops[4].download()}


def power(x, axis):
    """The power of two above every row's (or column's) largest element."""
    m = np.max(np.abs(x), axis=axis) if x.size else np.zeros(x.shape[1 - axis])
    return np.ldexp(1.0, np.frexp(np.where(m > 0, m, 1.0))[1].astype(int))


@pytest.mark.parametrize("emax,lmax", [(1, 1), (2, 2), (3, 3), (4, 2), (5, 5), (6, 4), (7, 7)])
@pytest.mark.parametrize("kind", ["plain", "graded", "tiny", "large"])
def test_products_match_extended_precision(built_lib, emax, lmax, kind):
    from imsrg_gb300 import Engine, make_basis
    eng = Engine(make_basis(emax, lmax=lmax), device=0)
    rng = np.random.default_rng(emax * 10 + lmax)
    L, R = rng.standard_normal(eng.slab), rng.standard_normal(eng.slab)
    if kind == "graded":  # elements of one row over 60 binary orders
        L *= np.ldexp(1.0, rng.integers(-60, 1, eng.slab))
        R *= np.ldexp(1.0, rng.integers(-60, 1, eng.slab))
    elif kind == "tiny":  # products below the normal range
        L *= 1e-160
        R *= 1e-155
    elif kind == "large":
        L *= 1e150
        R *= 1e150
    hL, hR = -1, 1
    got = run(eng, L, R, hL, hR)
    for row in arrays(eng):
        for (w, g), terms in products(L, R, hL, hR, row).items():
            o, n, m = row[g]
            if n * m == 0 or terms[0][1].shape[1] == 0:
                continue
            cols = np.unique(np.linspace(0, m - 1, min(m, 12)).astype(int))
            x = got[w][o:o + n * m].reshape(m, n).T[:, cols]
            ref, tol = np.zeros((n, len(cols)), np.longdouble), np.zeros((n, len(cols)))
            for s, A, B in terms:
                ref += s * (A.astype(np.longdouble) @ B[:, cols].astype(np.longdouble))
                # digits: each element to 2^-63 of its power of two and the dropped digit products, K 2^-59 of the two
                # powers of two; FP64 FMAs: K 2^-53 of the sum of magnitudes; 2^-1074 a rounding below the normal range
                K = A.shape[1]
                digits = K * 2.0 ** -59 * power(A, 1)[:, None] * power(B[:, cols], 0)[None]
                fma = K * 2.0 ** -53 * (np.abs(A) @ np.abs(B[:, cols]))
                tol += np.maximum(digits, fma) + K * 2.0 ** -1074
            tol += 2.0 ** -52 * np.abs(ref).astype(float)
            assert np.all(np.abs(x - ref) <= tol), (w, g, n, m, float(np.max(np.abs(x - ref) / tol)))


@pytest.mark.parametrize("emax", [3, 6])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_operands(built_lib, emax, bad):
    from imsrg_gb300 import Engine, make_basis
    eng = Engine(make_basis(emax), device=0)
    rng = np.random.default_rng(5)
    L, R = rng.standard_normal(eng.slab), rng.standard_normal(eng.slab)
    rows = arrays(eng)
    q = int(np.argmax([r[0][1] for r in rows]))
    o, n, _ = rows[q][0]
    L[o + n // 2 + n * (n // 3)] = bad  # one element of a pppp array
    for _ in range(2):  # the flag of a call does not outlive it
        got = run(eng, L, R, -1, 1)
        for k, row in enumerate(rows):
            for (w, g), terms in products(L, R, -1, 1, row).items():
                p, a, b = row[g]
                if a * b == 0 or terms[0][1].shape[1] == 0:
                    continue
                x = got[w][p:p + a * b].reshape(b, a).T
                with np.errstate(invalid="ignore"):
                    ref = sum(s * (A @ B) for s, A, B in terms)
                assert np.array_equal(np.isnan(x), np.isnan(ref)), (k, w, g)
                ok = np.isfinite(ref)
                assert np.array_equal(x[~ok & ~np.isnan(ref)], ref[~ok & ~np.isnan(ref)])
                scale = sum(A.shape[1] for _, A, _ in terms) * 40.0
                assert np.all(np.abs(x[ok] - ref[ok]) <= 2.0 ** -50 * scale)
    L[o + n // 2 + n * (n // 3)] = 1.0
    got = run(eng, L, R, -1, 1)
    assert np.all(np.isfinite(got["w1"])) and np.all(np.isfinite(got["w2"]))
