"""Contexts side by side in one process: one whose kernels need much shared memory keeps working after one that needs little."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "bf16x3"])
def test_commutator_after_a_smaller_context(built_lib, mode):
    from imsrg_gb300 import Engine, make_basis

    def operators(eng):
        rng = np.random.default_rng(1)
        return [eng.new_op(h, rng.standard_normal(eng.slab)) for h in (-1, 1)] + [eng.new_op(1)]

    a = Engine(make_basis(5), device=0, precision="bf16x3")
    x = operators(a)
    a.set_tuning({**a.autotune(*x), "tiny_cap": 64, "small_cap": 1024})
    a.set_precision(mode)
    a.commutator(*x)
    ref = x[2].download()
    b = Engine(make_basis(5, lmax=2), device=0, precision="bf16x3")
    y = operators(b)
    b.commutator(*y)
    b.set_precision("fp64")
    b.commutator(*y)
    b.synchronize()
    a.commutator(*x)
    assert np.max(np.abs(x[2].download() - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_hartree_fock_after_a_smaller_context(built_lib):
    from imsrg_gb300 import Engine, make_basis
    engines = [Engine(make_basis(e, lmax=l), device=0) for e, l in ((18, 1), (14, 1))]  # blocks of ten and of eight orbits
    out = []
    for k in (0, 1, 0):
        eng = engines[k]
        D = np.eye(eng.basis.norbits)
        op = eng.new_op(1, np.random.default_rng(k).standard_normal(eng.slab))
        eng.transform_2b_to_hf(op, D)
        out.append(op.download())
    assert np.array_equal(out[0], out[2])
