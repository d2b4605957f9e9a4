"""TS_commutator_222_ph over bases whose cross-coupled tensor blocks take more than one batch (and one just within a
batch), against the oracle: FP64 to 1e-10, split-BF16 products to the bound of the other tensor tests."""
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("emax,lmax,rank", [(6, 2, 4), (6, 3, 2), (5, 4, 4)])
def test_particle_hole_term_in_batches(built_lib, emax, lmax, rank):
    from imsrg_gb300 import Engine, make_basis
    from oracle.oracle import Oracle, TensorOracle
    b = make_basis(emax, lmax=lmax)
    o = Oracle(b)
    t = TensorOracle(o, rank, 0)
    A, B = o.random(31, -1), t.random(32, 1)
    ref = t.commutator(A, -1, B, 1, 64)
    for mode, tol in (("fp64", 1e-10), ("bf16x6", 2e-6)):
        eng = Engine(b, device=0, precision=mode)
        dA, dB = eng.new_op(-1, A), eng.new_tensor(rank, 0, 1, B)
        for _ in range(2):  # the batches' buffers are used again
            dR = eng.new_tensor(rank, 0, 1)
            eng.tensor_commutator(dA, dB, dR, 64)
            assert rel_err(dR.download(), ref) < tol, mode
