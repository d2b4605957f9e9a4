"""A device allocation that fails, whichever of a call's it is: the call says so, what it had prepared half-way is not taken for
ready, and the same call succeeds once there is memory."""
import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


def ops(eng, herms, seed=1):
    rng = np.random.default_rng(seed)
    return [eng.new_op(h, 0.01 * rng.standard_normal(eng.slab)) for h in herms]


def commutator(eng):
    L, R, RES = ops(eng, (-1, 1, 1))
    eng.commutator(L, R, RES)
    return [RES.download()]


def adjoint(eng):
    L, R, C = ops(eng, (-1, 1, 1))
    out = [eng.new_op(-1), eng.new_op(1)]
    eng.commutator_vjp(L, R, C, *out)
    return [x.download() for x in out]


def step(eng):
    H0 = eng.synthetic_hamiltonian(seed=3)
    st = eng.new_op(1, H0), eng.new_op(-1), eng.new_op(-1), eng.new_op(1, H0)
    eng.build_gs_white(st[0], st[2])
    eng.magnus_step(*st, 0.5, 6, 1e-8, allow_unconverged=True)
    return [x.download() for x in st]


def series(eng):
    G, H, HS = ops(eng, (-1, 1, 1))
    eng.bch_expand(HS, G, H)
    return [HS.download()]


def quads(eng):
    G, H, HS = ops(eng, (-1, 1, 1))
    eng.bch_expand_quads(HS, G, H)
    return [HS.download()]


def tensor(eng):
    (G,) = ops(eng, (-1,))
    Q, Y = eng.new_tensor(2, 0, 1), eng.new_tensor(2, 0, 1)
    Q.upload(np.random.default_rng(2).standard_normal(len(Q.download())))
    eng.tensor_commutator(G, Q, Y)
    return [Y.download()]


def eom(eng):
    from imsrg_gb300.eom import LadderSpace
    H, s = eng.new_op(1, eng.synthetic_hamiltonian(seed=1)), LadderSpace(eng, 2, 0)
    return [s.matvec(H, np.random.default_rng(3).standard_normal(s.n)) for _ in range(2)]


def hartree_fock(eng):
    H = eng.new_op(1, eng.synthetic_bare_hamiltonian(seed=1))
    D, info = eng.calc_hf(H)
    return [H.download(), D]


def w2_generator(eng):
    (H,) = ops(eng, (1,))
    H.upload(eng.synthetic_hamiltonian(seed=2))
    ETA = eng.new_op(-1)
    eng.build_gs_w2(H, ETA)
    return [ETA.download()]


def triples(eng):
    H, OM = eng.new_op(1, eng.synthetic_hamiltonian(seed=2)), ops(eng, (-1,))[0]
    return [np.array(eng.restore_triples(H, OM), dtype=np.float64).ravel()[:1]]


@pytest.mark.parametrize("mode,emax,case", [
    ("fp64", 5, commutator), ("bf16x3", 4, commutator), ("fp64", 5, adjoint), ("fp64", 5, step), ("tf32x3", 3, step), ("fp64", 4, series),
    ("fp64", 3, quads), ("fp64", 4, tensor), ("bf16x6", 3, tensor), ("fp64", 4, eom), ("bf16x3", 3, eom), ("fp64", 4, hartree_fock),
    ("fp64", 3, w2_generator), ("fp64", 2, triples)])
def test_every_allocation_in_turn(built_lib, mode, emax, case):
    from imsrg_gb300 import Engine, ImsrgError, make_basis

    def run(eng):
        eng.set_precision(mode)
        return case(eng)

    ref = run(Engine(make_basis(emax), device=0))
    for n in range(1, 60):
        eng = Engine(make_basis(emax), device=0)
        assert eng.L.imsrg_test_memory(eng.h, -1, -n) == 0
        try:
            run(eng)
            failed = False
        except ImsrgError as e:
            assert e.code == 3, (n, e)
            failed = True
        assert eng.L.imsrg_test_memory(eng.h, -1, 0) == 0
        for x, y in zip(ref, run(eng)):
            assert rel_err(y, x) <= (1e-10 if mode == "fp64" else 1e-6), n
        if not failed:
            break
    assert 1 < n < 59


def test_other_precision_that_finds_no_room(built_lib):
    from imsrg_gb300 import Engine, ImsrgError, make_basis
    eng = Engine(make_basis(4), device=0, precision="bf16x3")
    ref = commutator(eng)[0]
    for n in (1, 2, 3, 4):
        assert eng.L.imsrg_test_memory(eng.h, -1, -n) == 0
        with pytest.raises(ImsrgError):
            eng.set_precision("bf16x6")
        assert eng.L.imsrg_test_memory(eng.h, -1, 0) == 0
        assert rel_err(commutator(eng)[0], ref) <= 1e-6  # still in the mode it had
