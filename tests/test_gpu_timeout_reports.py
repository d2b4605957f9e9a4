"""A bounded wait that runs out is reported by the call that hands the incomplete result to the host, whichever it is, in FP64
and the mixed modes; the next calls of the same context are clean and right.  As in test_gpu_timeout.py the wait runs out
without a fault: a pipeline stage is left unarmed under a short limit."""
import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


def engine(emax, mode):
    from imsrg_gb300 import Engine, make_basis
    return Engine(make_basis(emax), device=0, precision=mode)


def operators(eng, o, size=0.05):
    return eng.new_op(-1, size * o.random(301, -1)), eng.new_op(1, o.random(302, 1)), eng.new_op(1)


def arm(eng):
    assert eng.L.imsrg_set_wait_limit(eng.h, 1_000_000) == 0  # 1 ms
    assert eng.L.imsrg_test_unarmed_stage(eng.h, 1) == 0


def runs_out(eng, call):
    from imsrg_gb300 import ImsrgError
    with pytest.raises(ImsrgError) as e:
        call()
    assert e.value.code == 7 and "bounded wait ran out" in str(e.value)
    eng.synchronize()  # reported once
    assert eng.L.imsrg_set_wait_limit(eng.h, 0) == 0


@pytest.mark.parametrize("mode", ["fp64", "bf16x3"])
@pytest.mark.parametrize("how", ["synchronize", "download", "E0", "norm", "mbpt2"])
def test_commutator(built_lib, oracles, mode, how):
    o, eng = oracles(5), engine(5, mode)
    L, R, RES = operators(eng, o)
    eng.commutator(L, R, RES)
    ref = RES.download()
    arm(eng)
    eng.commutator(L, R, RES)
    runs_out(eng, {"synchronize": eng.synchronize, "download": RES.download, "E0": lambda: RES.E0,
                   "norm": lambda: eng.mat_frob_norm(RES), "mbpt2": lambda: eng.mbpt2(RES)}[how])
    eng.commutator(L, R, RES)
    assert rel_err(RES.download(), ref) < (1e-12 if mode == "fp64" else 1e-6)


@pytest.mark.parametrize("mode", ["fp64", "bf16x3"])
def test_series(built_lib, oracles, mode):
    o, eng = oracles(5), engine(5, mode)
    G, H, HS = operators(eng, o, 1e-3)
    eng.bch_expand(HS, G, H)
    ref = HS.download()
    arm(eng)
    runs_out(eng, lambda: eng.bch_expand(HS, G, H))
    eng.bch_expand(HS, G, H)
    assert rel_err(HS.download(), ref) < (1e-12 if mode == "fp64" else 1e-6)


def test_cross_coupled_download(built_lib, oracles):
    o, eng = oracles(5), engine(5, "fp64")
    L, R, RES = operators(eng, o)
    lcc, rcc, wcc = eng.new_cc(0), eng.new_cc(0), eng.new_cc(1)
    eng.calculate_cross_coupled(L, lcc)
    eng.calculate_cross_coupled(R, rcc)
    arm(eng)
    eng.commutator_222_ph(lcc, rcc, RES, wcc)
    runs_out(eng, wcc.download)


def test_tensor_series_and_download(built_lib):
    eng = engine(4, "fp64")
    rng = np.random.default_rng(3)
    G, Q, Y = eng.new_op(-1, 1e-3 * rng.standard_normal(eng.slab)), eng.new_tensor(4, 0, 1), eng.new_tensor(4, 0, 1)
    x = rng.standard_normal(len(Q.download()))
    Q.upload(x)
    arm(eng)
    runs_out(eng, lambda: eng.bch_tensor(G, Q))
    Q.upload(x)
    arm(eng)
    eng.tensor_commutator(G, Q, Y)
    runs_out(eng, Y.download)


def test_eom_product(built_lib):
    from imsrg_gb300.eom import LadderSpace
    eng = engine(6, "fp64")
    H, s = eng.new_op(1, eng.synthetic_hamiltonian(seed=1)), LadderSpace(eng, 4, 0)
    v = np.random.default_rng(1).standard_normal(s.n)
    ref = s.matvec(H, v)
    arm(eng)  # the captured product takes the new limit
    runs_out(eng, lambda: s.matvec(H, v))
    assert rel_err(s.matvec(H, v), ref) < 1e-12
