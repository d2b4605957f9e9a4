"""FP64 without its optional device buffers: digit plans, gather tables and 9j tables that find no room (the kernels that need none
do the call), and buffers given back when a required allocation fails, under captured graphs too."""
import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu

# the other kernels sum a few hundred products in another order
TOL = 1e-12


def engine(emax, limit=None, **more):
    from imsrg_gb300 import Engine, make_basis
    eng = Engine(make_basis(emax, **more), device=0)
    if limit is not None:
        assert eng.L.imsrg_test_memory(eng.h, limit, 0) == 0
    return eng


def refuse_next(eng):
    assert eng.L.imsrg_test_memory(eng.h, -1, 1) == 0


def both(case, *args, **kw):
    a, b = case(engine(*args, **kw)), case(engine(*args, limit=0, **kw))
    for x, y in zip(a, b):
        assert rel_err(y, x) <= TOL


@pytest.mark.parametrize("emax,lmax", [(5, 5), (6, 4)])
def test_commutator_without_room(built_lib, emax, lmax):
    def case(eng):
        rng = np.random.default_rng(2)
        L, R = (eng.new_op(h, rng.standard_normal(eng.slab)) for h in (-1, 1))
        RES = eng.new_op(1)
        eng.commutator(L, R, RES)
        return [RES.download()]
    both(case, emax, lmax=lmax)


def test_adjoint_without_room(built_lib):
    def case(eng):
        rng = np.random.default_rng(3)
        L, R, C = (eng.new_op(h, rng.standard_normal(eng.slab)) for h in (-1, 1, 1))
        out = eng.new_op(-1), eng.new_op(1)
        eng.commutator_vjp(L, R, C, *out)
        return [x.download() for x in out]
    both(case, 5)


@pytest.mark.parametrize("rank,dpar", [(0, 0), (2, 2), (4, 0)])
def test_tensor_commutator_without_room(built_lib, rank, dpar):
    def case(eng):
        rng = np.random.default_rng(4)
        G, Q, Y = eng.new_op(-1, rng.standard_normal(eng.slab)), eng.new_tensor(rank, dpar, 1), eng.new_tensor(rank, dpar, 1)
        Q.upload(rng.standard_normal(len(Q.download())))
        eng.tensor_commutator(G, Q, Y)
        return [Y.download()]
    both(case, 4)


def test_batches_share_their_operands(built_lib):
    def case(eng):
        rng = np.random.default_rng(5)
        G, Q = eng.new_op(-1, rng.standard_normal(eng.slab)), eng.new_tensor(4, 0, 1)
        Q.upload(rng.standard_normal(len(Q.download())))
        out = []
        for _ in range(2):
            Y = eng.new_tensor(4, 0, 1)
            eng.tensor_commutator(G, Q, Y, 64)  # the particle-hole term, several batches of blocks
            out.append(Y.download())
        return out
    both(case, 6, lmax=3)


def test_eom_without_room(built_lib):
    from imsrg_gb300.eom import LadderSpace

    def case(eng):
        H, s = eng.new_op(1, eng.synthetic_hamiltonian(seed=1)), LadderSpace(eng, 4, 0)
        v = np.random.default_rng(6).standard_normal(s.n)
        return [s.matvec(H, v), s.matvec(H, v)]
    both(case, 6)


def test_given_back_and_made_again(built_lib):
    torch = pytest.importorskip("torch")
    from imsrg_gb300.eom import LadderSpace
    eng = engine(5)
    H0 = eng.synthetic_hamiltonian(seed=3)
    H, s = eng.new_op(1, H0), LadderSpace(eng, 4, 0)
    v = np.random.default_rng(7).standard_normal(s.n)
    G0, D0 = eng.new_op(-1), eng.new_op(-1)
    eng.build_gs_white(H, D0)
    HS, G, DG, RES, Q = eng.new_op(1), eng.new_op(-1), eng.new_op(-1), eng.new_op(1), eng.new_tensor(4, 0, 1)
    Q.upload(np.random.default_rng(8).standard_normal(len(Q.download())))
    Y, bars = eng.new_tensor(4, 0, 1), (eng.new_op(-1), eng.new_op(1))

    def everything():
        eng.copy_sq_op(G0, G)
        eng.copy_sq_op(D0, DG)
        eng.magnus_step(HS, G, DG, H, 0.5, max_terms=6, allow_unconverged=True)
        eng.commutator(DG, H, RES)
        eng.tensor_commutator(DG, Q, Y)
        for b in bars:
            eng.clear_sq_op(b)
        eng.commutator_vjp(DG, H, RES, *bars)
        return [HS.download(), RES.download(), Y.download(), *[b.download() for b in bars], s.matvec(H, v)]

    ref = everything()
    kept = []
    for _ in range(2):
        eng.synchronize()
        before = torch.cuda.mem_get_info()[0]
        refuse_next(eng)
        kept.append(eng.new_tensor(2, 0, 1))  # an allocation of every kind of caller would do
        assert torch.cuda.mem_get_info()[0] > before  # more was given back than taken
        for x, y in zip(ref, everything()):
            assert rel_err(y, x) <= 1e-10  # a step's rounding through the White generator's denominators


def test_half_of_the_free_memory(built_lib):
    """No optional buffer above half of what is free: with the limit at the size of the smaller list's operands only that one is
    planned, and the result is the same."""
    def case(limit):
        eng = engine(6, limit)
        rng = np.random.default_rng(9)
        L, R = (eng.new_op(h, rng.standard_normal(eng.slab)) for h in (-1, 1))
        RES = eng.new_op(1)
        eng.commutator(L, R, RES)
        return RES.download()
    ref = case(None)
    for limit in (1 << 22, 1 << 24, 1 << 26):
        assert rel_err(case(limit), ref) <= TOL
