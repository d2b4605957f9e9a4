"""The two-body basis change on both sides of the sub-block size that a warp takes by itself: few partial waves and many
radial states (sub-blocks up to 6^4 elements), full bases (mostly small ones), coefficients that are no rotation."""
import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


def setup(emax, lmax, A):
    from imsrg_gb300 import Engine, make_basis
    from oracle.oracle import Oracle
    b = make_basis(emax, A // 2, A // 2, lmax=lmax)
    D = np.random.default_rng(4).standard_normal((b.norbits, b.norbits))
    key = np.stack([b.ll, b.jj, b.itzp])
    D[(key[:, :, None] != key[:, None, :]).any(axis=0)] = 0.0
    return Oracle(b), Engine(b, device=0), D


SIZES = [(10, 0, 4), (8, 1, 16), (6, 2, 16), (3, 3, 16), (2, 0, 4)]


@pytest.mark.parametrize("emax,lmax,A", SIZES)
def test_transform_matches_oracle(built_lib, emax, lmax, A):
    o, eng, D = setup(emax, lmax, A)
    R = o.random(11, 1)
    op = eng.new_op(1, R)
    eng.transform_2b_to_hf(op, D)
    # four sums of at most six FP64 terms each
    assert rel_err(op.download(), o.transform_2b_to_hf(R, D)) < 1e-12


@pytest.mark.parametrize("emax,lmax,A", SIZES)
@pytest.mark.parametrize("herm", [1, -1])
def test_round_trip(built_lib, emax, lmax, A, herm):
    o, eng, D = setup(emax, lmax, A)
    # a rotation within each block: the QR of a block-diagonal matrix, in orbit order
    Q = np.zeros_like(D)
    for rows in {tuple(np.flatnonzero(D[i])) for i in range(len(D))}:
        Q[np.ix_(rows, rows)] = np.linalg.qr(D[np.ix_(rows, rows)])[0]
    R = o.random(12, herm)
    op = eng.new_op(herm, R)
    eng.transform_2b_to_hf(op, Q)
    moved = op.download()
    assert rel_err(moved, R) > 1e-2
    eng.transform_2b_to_hf(op, Q.T)
    assert rel_err(op.download(), R) < 1e-12
