"""The FP64 commutator's gather kernels (122 by pair groups, recoupling by orbit quadruples, the ladder update with the
mirror) against the piecewise entry points, which take a thread per element: bases on both sides of the size where the
commutator changes over, cut and full in l, all signs, operators with and without consistent lower triangles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def by_pieces(eng, L, R, RES):
    lcc, rcc, wcc = eng.new_cc(0), eng.new_cc(0), eng.new_cc(1)
    w1, w2 = eng.new_op(1), eng.new_op(1)
    eng.calculate_cross_coupled(R, rcc)
    eng.calculate_cross_coupled(L, lcc)
    eng.commutator_111(L, R, RES)
    eng.commutator_121(L, R, RES)
    eng.commutator_122(L, R, RES)
    eng.commutator_222_pp_hh(L, R, RES, w1, w2)
    eng.commutator_221(L, R, RES, w1, w2)
    eng.commutator_222_ph(lcc, rcc, RES, wcc)
    return RES.download()


@pytest.mark.parametrize("emax,lmax,A", [(4, 4, 16), (5, 5, 16), (5, 4, 4), (6, 3, 16), (6, 6, 4)])
@pytest.mark.parametrize("hL,hR", [(-1, 1), (-1, -1), (1, 1), (1, -1)])
@pytest.mark.parametrize("mirrored", [True, False])
def test_commutator_matches_pieces(built_lib, oracles, emax, lmax, A, hL, hR, mirrored):
    from imsrg_gb300 import Engine, make_basis
    from oracle.oracle import Oracle
    b = make_basis(emax, A // 2, A // 2, lmax=lmax)
    eng = Engine(b, device=0)
    if mirrored:
        o = Oracle(b)
        L, R = o.random(7, hL), o.random(8, hR)
    else:
        rng = np.random.default_rng(9)
        L, R = rng.standard_normal(eng.slab), rng.standard_normal(eng.slab)
    dL, dR = eng.new_op(hL, L), eng.new_op(hR, R)
    ref = by_pieces(eng, dL, dR, eng.new_op(-hL * hR))
    for _ in range(2):
        out = eng.new_op(-hL * hR)
        eng.commutator(dL, dR, out, e0=False)
        got = out.download()
        # a few hundred FP64 roundings of terms no larger than about the largest element
        assert np.max(np.abs(got[1:] - ref[1:])) <= 4e-13 * np.max(np.abs(ref[1:]))
