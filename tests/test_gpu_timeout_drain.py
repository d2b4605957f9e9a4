"""A wait limit below the time of a copy: every CTA gives up with copies and MMAs of its own in flight, waits for those under a
limit of its own, and the context goes on with the right results once the limit is back."""
import numpy as np
import pytest

from helpers import rel_err
from test_gpu_timeout_reports import engine, operators, runs_out

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "bf16x3", "bf16x6", "tf32x3"])
def test_step(built_lib, oracles, mode):
    o, eng = oracles(5), engine(5, mode)
    G0, H, HS = operators(eng, o, 1e-3)
    D0, G, DG = eng.new_op(-1, 1e-2 * o.random(303, -1)), eng.new_op(-1), eng.new_op(-1)

    def step():
        eng.copy_sq_op(G0, G)
        eng.copy_sq_op(D0, DG)
        return eng.magnus_step(HS, G, DG, H, 0.5, max_terms=6, allow_unconverged=True)

    step()
    ref = HS.download()
    assert eng.L.imsrg_set_wait_limit(eng.h, 100) == 0
    runs_out(eng, step)
    step()
    assert rel_err(HS.download(), ref) < (1e-12 if mode == "fp64" else 1e-6)


def test_eom_product(built_lib):
    from imsrg_gb300.eom import LadderSpace
    eng = engine(6, "fp64")
    H, s = eng.new_op(1, eng.synthetic_hamiltonian(seed=1)), LadderSpace(eng, 4, 0)
    v = np.random.default_rng(1).standard_normal(s.n)
    ref = s.matvec(H, v)
    assert eng.L.imsrg_set_wait_limit(eng.h, 100) == 0
    runs_out(eng, lambda: s.matvec(H, v))
    assert rel_err(s.matvec(H, v), ref) < 1e-12
