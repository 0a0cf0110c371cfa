"""tl3d_solve_step_backward with settings->max_iters raised above what the chunk
was initialised with: the loops record each trip in tables of that length, so a
solve that converges within it runs as before, and one that does not is an error
and leaves what lies beyond the tables alone."""
import ctypes as C

import numpy as np
import pytest
import torch

from tealeaf_b200 import abi, problems
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu

CELLS = (34, 19, 23)


def _backward(table, max_iters, chip):
    h = Host(problems.seeded(3, CELLS, 11, 4, 0, solver="cg", end_step=1, max_iters=table, name="tables").tea_in(), 3)
    try:
        h.lib.tl3d_set_chip_loop(C.byref(h.chunk), chip)
        h.solve_device(0)
        h.settings.max_iters = max_iters
        n = int(np.prod(h.shape))
        # (a constant g_u is an eigenvector of the operator: one iteration)
        g = torch.from_numpy(np.random.default_rng(3).random(n)).cuda()
        lam, grad = torch.zeros_like(g), torch.zeros_like(g)
        torch.cuda.synchronize()
        its = C.c_int(0)
        rc = h.lib.tl3d_solve_step_backward(C.byref(h.chunk), C.byref(h.settings), g.data_ptr(), h.chunk.vec_u,
                                            lam.data_ptr(), grad.data_ptr(), 1e-10, C.byref(its))
        err = None
        try:
            abi.check(h.lib, 3)
        except abi.SuiteError as exc:
            err = str(exc)
        torch.cuda.synchronize()
        return rc, its.value, err, grad.cpu().numpy()
    finally:
        h.finalise()


@pytest.mark.parametrize("chip", [0, 1])
def test_a_solve_within_the_tables_is_as_with_the_smaller_limit(chip):
    want, got = _backward(400, 400, chip), _backward(400, 4000, chip)
    assert want[0] == got[0] == 0 and want[2] is got[2] is None
    assert 10 < want[1] == got[1] < 400
    assert np.array_equal(want[3], got[3])


@pytest.mark.parametrize("chip", [0, 1])
def test_a_solve_beyond_the_tables_is_an_error(chip):
    rc, its, err, _ = _backward(6, 4000, chip)
    assert rc == 32 and its == 6
    assert "more iterations than the 6 the chunk was initialised with" in err
