"""The refinement form's trips run in launched groups, each followed by the
residual replacement: iteration caps that end inside, at and past a group of
eight stop at the cap with the residual of that trip, the same for both ways of
loading the operands, and a tight tolerance with a replacement every few trips
still converges."""
import numpy as np
import pytest

from tealeaf_b200 import problems
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["cg", "ppcg"])
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("cap", [1, 7, 8, 9, 30, 20000])
def test_caps_stop_inside_a_group(cap, precision, solver):
    text = problems.seeded(2, (150, 83), 29, 4, 1, solver=solver, end_step=1, max_iters=cap, error_switch=True,
                           eps_lim=1e30, ppcg_inner_steps=min(10, cap), name="groups").tea_in()
    a, b = Host(text, 2), Host(text, 2)
    try:
        b.lib.tl2d_set_tma(b.chunk, 0)
        ra, rb = (h.refine_step(0, 1e-11, precision, summary=False) for h in (a, b))
        assert ra.iterations == rb.iterations and ra.residual_updates == rb.residual_updates
        assert ra.rel_residual == rb.rel_residual
        assert np.array_equal(a.download("u"), b.download("u"))
        if cap <= 30:
            assert ra.iterations == cap and not ra.converged and ra.rel_residual > 1e-11
        else:
            assert ra.converged and ra.rel_residual <= 1e-11 and ra.residual_updates > 3
    finally:
        a.finalise()
        b.finalise()
