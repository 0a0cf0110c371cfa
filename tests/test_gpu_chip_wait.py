"""The waits between the blocks of the persistent CG loops (tealeaf_b200/csrc/
gridsum.cuh), made to run out by a limit of one poll: every block returns, in
all forms of the loops (one to four groups of a block, meshes with ragged
strips and tiles, the preconditioned loop), and the host reports an error. The
blocks' threads meet at barriers, so a block may only be left by all of its
threads at once."""
import ctypes as C

import pytest

from tealeaf_b200 import abi, problems
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu

MESHES = [(2, (64, 64), "none"), (2, (513, 300), "none"), (2, (513, 941), "none"), (2, (1000, 1180), "none"),
          (2, (300, 170), "jac_diag"), (2, (1000, 702), "jac_block"),
          (3, (33, 19, 5), "none"), (3, (48, 47, 50), "none"), (3, (100, 90, 80), "none"), (3, (64, 63, 150), "none")]


def host(dims, cells, pc, **kw):
    return Host(problems.seeded(dims, cells, 11, 4, 0 if dims == 3 else 2, solver="cg", end_step=1, max_iters=400,
                                preconditioner=pc, name="wait", **kw).tea_in(), dims)


def set_limit(h, polls):
    return getattr(h.lib, "tl%dd_set_chip_wait_limit" % h.dims)(C.byref(h.chunk), polls)


@pytest.mark.parametrize("dims,cells,pc", MESHES)
def test_a_wait_that_runs_out_ends_the_solve_with_an_error(dims, cells, pc):
    h = host(dims, cells, pc)
    try:
        for _ in range(10):
            assert set_limit(h, 1) == 0
            with pytest.raises(abi.SuiteError, match="gave up"):
                h.solve_device(0)
    finally:
        h.finalise()


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("polls", [-1, (1 << 22) + 1])
def test_a_limit_out_of_range_is_refused(dims, polls):
    h = host(dims, (12, 10, 8)[:dims], "none")
    try:
        assert set_limit(h, polls) == 36
        with pytest.raises(abi.SuiteError, match="polls must be"):
            abi.check(h.lib, dims)
        h.solve_device(0)
    finally:
        h.finalise()
