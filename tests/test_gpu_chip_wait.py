"""The waits between the blocks of the persistent CG loops (tealeaf_b200/csrc/
gridsum.cuh), made to run out by a limit of one poll: every block returns, in
all forms of the loops (one to four groups of a block, meshes with ragged
strips and tiles, the preconditioned loop), and the host reports an error. The
blocks' threads meet at barriers, so a block may only be left by all of its
threads at once."""
import ctypes as C

import numpy as np
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


@pytest.mark.parametrize("dims,cells,pc", MESHES)
def test_the_error_names_the_loop_and_the_chunk_recovers(dims, cells, pc):
    """The report is the loop's own, not that of the TMA loads, and stays with
    the solve it belongs to: the same chunk's next solve equals a fresh one's."""
    a, b = host(dims, cells, pc), host(dims, cells, pc)
    try:
        assert set_limit(a, 1) == 0
        with pytest.raises(abi.SuiteError, match="error 38: the CG loop on chip did not complete.*after 1 polls"):
            a.solve_device(0)
        assert set_limit(a, 0) == 0
        ra, rb = a.solve_device(0), b.solve_device(0)
        assert ra.iterations == rb.iterations and ra.error == rb.error and ra.summary == rb.summary
        for f in ("u", "p", "r", "w", "energy"):
            assert np.array_equal(a.download(f), b.download(f)), f
    finally:
        a.finalise()
        b.finalise()


def test_the_adjoint_reports_it_too():
    import torch
    h = host(3, (48, 47, 50), "none")
    try:
        box = [2.0, 8.0, 2.0, 8.0, 2.0, 8.0]
        h.solve_device(0)
        n = h.shape[0] * h.shape[1] * h.shape[2]
        g, lam, grad = (torch.ones(n, dtype=torch.float64, device="cuda") for _ in range(3))
        its = C.c_int(0)

        def backward():
            return h.lib.tl3d_solve_step_backward(C.byref(h.chunk), C.byref(h.settings), g.data_ptr(), h.chunk.vec_u,
                                                  lam.data_ptr(), grad.data_ptr(), 1e-8, C.byref(its))

        torch.cuda.synchronize()
        set_limit(h, 1)
        assert backward() == 38
        with pytest.raises(abi.SuiteError, match="error 38"):
            abi.check(h.lib, 3)
        with pytest.raises(abi.SuiteError, match="error 38"):
            h.adjoint_gradient(1, 1, box, 1e-8)
        set_limit(h, 0)
        assert backward() == 0 and its.value > 0
    finally:
        h.finalise()
