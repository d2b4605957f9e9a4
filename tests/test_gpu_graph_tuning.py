"""A captured Magnus step after its launch tables have changed behind it: another tuning of the mixed modes (accepted, rejected or
broken off half-way), which shares the 122 plan with FP64, and another mixed precision and back.  The step must be the eager one."""
import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


def states(eng):
    H, out = eng.synthetic_hamiltonian(seed=3), []
    for _ in range(2):
        st = (eng.new_op(1, H), eng.new_op(-1), eng.new_op(-1), eng.new_op(1, H))
        eng.build_gs_white(st[0], st[2])
        out.append(st)
    return out


def step_both(eng, st, tol):
    for s, graph in zip(st, (True, False)):
        eng.magnus_step(*s, 0.5, 6, 1e-8, graph=graph, allow_unconverged=True)
    for x, y in zip(*st):
        assert rel_err(x.download(), y.download()) <= tol


@pytest.mark.parametrize("change,accepted", [({"small_cap": 1024, "tiny_cap": 64}, True), ({"small_cap": 64, "tiny_cap": 8}, True),
                                             ({"small_cap": 1024, "gemm_wmax": 256}, False), ({"small_cap": 5000}, False)])
def test_fp64_step_after_tuning(built_lib, oracles, change, accepted):
    from imsrg_gb300 import Engine, ImsrgError, make_basis
    o, eng = oracles(5), Engine(make_basis(5), device=0)
    st = states(eng)
    step_both(eng, st, 1e-11)
    eng.set_precision("bf16x6")
    L, R, RES = eng.new_op(-1, o.random(7, -1)), eng.new_op(1, o.random(8, 1)), eng.new_op(1)
    cfg = dict(eng.autotune(L, R, RES))
    eng.set_precision("fp64")
    step_both(eng, st, 1e-11)  # captured again after the autotuner
    eng.set_precision("bf16x6")
    if accepted:
        eng.set_tuning({**cfg, **change})
    else:
        with pytest.raises(ImsrgError) as e:
            eng.set_tuning({**cfg, **change})
        assert e.value.code == 1
    eng.set_precision("fp64")
    for _ in range(2):
        step_both(eng, st, 1e-11)


def test_mixed_step_after_another_precision(built_lib):
    from imsrg_gb300 import Engine, make_basis
    eng = Engine(make_basis(4), device=0, precision="bf16x3")
    st = states(eng)
    step_both(eng, st, 0.0)
    eng.set_precision("tf32x3")
    filler = [eng.new_op(1, np.full(eng.slab, np.nan)) for _ in range(8)]  # where the old tables lay
    eng.set_precision("bf16x3")
    step_both(eng, st, 0.0)
    del filler
