"""Where the driver refuses the persistent launch of a CG loop on chip (its
blocks cannot all be resident at once, as in a process that was given part of
the device's SMs), the solve takes the loop of two launches per trip, as larger
meshes do: no error, and the fields, counts and launches of that loop."""
import ctypes as C

import numpy as np
import pytest

from tealeaf_b200 import abi, problems
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu

OFF, ON, REFUSED = 0, 1, 2


def host(dims, cells, mode, pc="none", solver="cg", steps=1):
    h = Host(problems.seeded(dims, cells, 19, 4, 0 if dims == 3 else 2, solver=solver, end_step=steps, max_iters=300,
                             preconditioner=pc, name="refused").tea_in(), dims)
    assert getattr(h.lib, "tl%dd_set_chip_loop" % dims)(C.byref(h.chunk), mode) == 0
    return h


@pytest.mark.parametrize("dims,cells,pc,solver", [
    (2, (64, 64), "none", "cg"), (2, (513, 300), "none", "cg"), (2, (301, 171), "jac_diag", "cg"),
    (2, (300, 170), "jac_block", "cg"), (2, (130, 77), "none", "ppcg"), (2, (130, 77), "none", "cheby"),
    (3, (33, 19, 5), "none", "cg"), (3, (64, 63, 64), "none", "cg"), (3, (37, 19, 23), "none", "ppcg"),
])
def test_a_refused_launch_takes_the_launched_loop(dims, cells, pc, solver):
    a, b = host(dims, cells, REFUSED, pc, solver, 2), host(dims, cells, OFF, pc, solver, 2)
    try:
        for tt in range(2):
            n = [getattr(h.lib, "tl%dd_launch_count" % dims)(C.byref(h.chunk)) for h in (a, b)]
            ra, rb = a.solve_device(tt), b.solve_device(tt)
            n = [getattr(h.lib, "tl%dd_launch_count" % dims)(C.byref(h.chunk)) - m for h, m in zip((a, b), n)]
            assert n[0] == n[1] > 2 * rb.iterations["CG"]
            assert ra.iterations == rb.iterations and ra.error == rb.error and ra.summary == rb.summary
            for f in ("u", "p", "r", "w", "sd", "energy"):
                assert np.array_equal(a.download(f), b.download(f)), (tt, f)
        # and the chunk is as before once its launch is not refused
        assert getattr(a.lib, "tl%dd_set_chip_loop" % dims)(C.byref(a.chunk), ON) == 0
        assert a.solve_device(2).iterations["CG"] > 0
    finally:
        a.finalise()
        b.finalise()


def test_a_refused_adjoint_solve_takes_the_launched_loop():
    box = [2.0, 8.0, 2.0, 8.0, 2.0, 8.0]
    out = []
    for mode in (REFUSED, OFF):
        h = host(3, (48, 30, 26), mode, steps=2)
        try:
            out.append(h.adjoint_gradient(2, 1, box, 1e-10))
        finally:
            h.finalise()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
    assert out[0][2].adjoint_iters == out[1][2].adjoint_iters > 0


@pytest.mark.parametrize("dims", [2, 3])
def test_an_unknown_mode_is_refused(dims):
    h = host(dims, (12, 10, 8)[:dims], ON)
    try:
        assert getattr(h.lib, "tl%dd_set_chip_loop" % dims)(C.byref(h.chunk), 3) == 39
        with pytest.raises(abi.SuiteError, match="error 39"):
            abi.check(h.lib, dims)
    finally:
        h.finalise()
