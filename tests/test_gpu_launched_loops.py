"""The CG loops of two launches per trip, which every mesh too large for the
chip takes, on small meshes (the loop on chip switched off, set_chip_loop) and
past the limit. What is compared runs the two sides' own kernels:

* the preconditioned loop fed by TMA and by per-thread loads, bit for bit
  (k_pcg_ur_tma, k_pcg_ur and the w sweeps), and against the oracle;
* the plain loops fed both ways, 2D and 3D, bit for bit;
* the loops on chip against the launched ones, bit for bit (with jac_block where
  the mesh's strips are whole blocks, so that both loops add the same partial
  sums), smooth and rough densities;
* the adjoint's solves on chip against the launched ones, bit for bit, and the
  launched ones against the CPU adjoint.
"""
import ctypes as C

import numpy as np
import pytest

from tealeaf_b200 import problems
from tealeaf_b200.config import read_config
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu

FIELDS = {2: ("u", "u0", "p", "r", "w", "mi", "kx", "ky", "sd", "energy"),
          3: ("u", "u0", "p", "r", "w", "kx", "ky", "kz", "sd", "energy")}


def text(dims, cells, cap, pc="none", steps=1):
    return problems.seeded(dims, cells, 33, 4, 0 if dims == 3 else 2, solver="cg", end_step=steps, max_iters=cap,
                           preconditioner=pc, name="launched").tea_in()


def host(deck, dims, chip=True, tma=True, rough=False):
    h = Host(deck, dims)
    if not chip:
        getattr(h.lib, "tl%dd_set_chip_loop" % dims)(C.byref(h.chunk), 0)
    if not tma:
        getattr(h.lib, "tl%dd_set_tma" % dims)(C.byref(h.chunk), 0)
    if rough:   # every face coefficient different from its neighbours
        h.upload("density", 0.05 + 20.0 * np.random.default_rng(7).random(h.shape))
    return h


def launches(h):
    return getattr(h.lib, "tl%dd_launch_count" % h.dims)(C.byref(h.chunk))


def assert_equal_steps(a, b, steps, launched):
    """Steps both chunks; `launched`: those of the two whose loop is launched."""
    try:
        for tt in range(steps):
            n0 = {id(h): launches(h) for h in (a, b)}
            ra, rb = a.solve_device(tt), b.solve_device(tt)
            for h in (a, b):
                n = launches(h) - n0[id(h)]
                assert n > 2 * ra.iterations["CG"] if h in launched else n <= 18, n
            assert ra.iterations == rb.iterations and ra.error == rb.error and ra.summary == rb.summary
            for f in FIELDS[a.dims]:
                assert np.array_equal(a.download(f), b.download(f)), (tt, f)
    finally:
        a.finalise()
        b.finalise()


@pytest.mark.parametrize("pc", ["jac_diag", "jac_block"])
@pytest.mark.parametrize("cells,cap,steps", [
    ((300, 170), 20000, 2), ((6, 5), 40, 1), ((130, 77), 20000, 1), ((642, 43), 60, 1),
    ((1300, 1001), 25, 2), ((2050, 1207), 12, 1),
])
def test_preconditioned_sweeps_fed_both_ways_are_bit_identical(cells, cap, steps, pc):
    deck = text(2, cells, cap, pc, steps)
    a, b = host(deck, 2, chip=False), host(deck, 2, chip=False, tma=False)
    assert_equal_steps(a, b, steps, (a, b))


@pytest.mark.parametrize("pc", ["jac_diag", "jac_block"])
@pytest.mark.parametrize("cells,cap,chip", [
    ((97, 61), 20000, False), ((130, 78), 20000, False), ((256, 257), 20000, False),
    ((1300, 1001), 25, True), ((1301, 1002), 25, True), ((1201, 1403), 25, True),
])
def test_launched_preconditioned_cg_against_the_oracle(cells, cap, chip, pc, oracle_lib):
    """Trip counts as the oracle's, the summary within 1e-12 of its."""
    deck = text(2, cells, cap, pc)
    want = oracle_lib.run(*read_config(deck, 2))[0]
    h = host(deck, 2, chip=chip)   # the larger meshes launch their loop by themselves
    try:
        n0 = launches(h)
        got = h.solve_device(0)
        assert launches(h) - n0 > 2 * got.iterations["CG"]
        assert got.iterations == want.iterations
        for x, y in zip(got.summary, want.summary):
            assert abs(x - y) <= 1e-12 * abs(y)
    finally:
        h.finalise()


@pytest.mark.parametrize("rough", [False, True])
@pytest.mark.parametrize("pc,cells,cap", [
    ("none", (300, 157), 20000), ("none", (129, 37), 20000), ("none", (1000, 1180), 25),
    ("jac_diag", (5, 3), 20000), ("jac_diag", (33, 7), 20000), ("jac_diag", (129, 38), 200), ("jac_diag", (1024, 442), 25),
    ("jac_diag", (641, 941), 25), ("jac_diag", (1013, 777), 25), ("jac_diag", (1025, 900), 25),
    ("jac_diag", (1000, 1180), 25),
    ("jac_block", (640, 941), 25), ("jac_block", (640, 942), 25), ("jac_block", (639, 943), 25),
    ("jac_block", (1000, 1180), 25), ("jac_block", (1024, 1181), 25), ("jac_block", (1000, 1178), 1),
])
def test_the_loop_on_chip_equals_the_launched_one(pc, cells, cap, rough):
    """jac_block: strips of 4 and 8 rows, the last block of 4, 1, 2 and 3."""
    deck = text(2, cells, cap, pc)
    a, b = host(deck, 2, rough=rough), host(deck, 2, chip=False, rough=rough)
    assert_equal_steps(a, b, 1, (b,))


@pytest.mark.parametrize("rough", [False, True])
@pytest.mark.parametrize("cells,cap", [((33, 9, 5), 20000), ((38, 19, 23), 20000), ((100, 90, 80), 20),
                                       ((64, 63, 150), 20), ((48, 47, 50), 1)])
def test_the_3d_loop_on_chip_equals_the_launched_one(cells, cap, rough):
    deck = text(3, cells, cap)
    a, b = host(deck, 3, rough=rough), host(deck, 3, chip=False, rough=rough)
    assert_equal_steps(a, b, 1, (b,))


@pytest.mark.parametrize("dims,cells", [(2, (300, 157)), (2, (130, 66)), (3, (38, 19, 23)), (3, (66, 20, 31))])
def test_launched_sweeps_fed_both_ways_are_bit_identical(dims, cells):
    deck = text(dims, cells, 20000, steps=2)
    a, b = host(deck, dims, chip=False), host(deck, dims, chip=False, tma=False)
    assert_equal_steps(a, b, 2, (a, b))


BOX = [2.0, 8.0, 2.0, 8.0, 2.0, 8.0]


def gradient(deck, steps, every, tol, **kw):
    h = host(deck, 3, **kw)
    try:
        return h.adjoint_gradient(steps, every, BOX, tol)
    finally:
        h.finalise()


@pytest.mark.parametrize("cells,cap,steps,every", [
    ((48, 30, 26), 20000, 3, 2), ((37, 19, 23), 20000, 2, 1), ((64, 63, 64), 6, 2, 1), ((64, 63, 64), 7, 2, 1),
    ((48, 30, 26), 1, 1, 1), ((48, 30, 26), 2, 1, 1),
])
def test_adjoint_on_chip_equals_the_launched_one(cells, cap, steps, every):
    """Caps of an even and an odd number of trips end the solves there."""
    deck = text(3, cells, cap, steps=steps)
    J, g, st = gradient(deck, steps, every, 1e-11)
    for tma in (True, False):
        J1, g1, st1 = gradient(deck, steps, every, 1e-11, chip=False, tma=tma)
        assert J1 == J and np.array_equal(g1, g), tma
        assert (st1.forward_iters, st1.adjoint_iters) == (st.forward_iters, st.adjoint_iters)


def test_launched_adjoint_matches_the_cpu_adjoint(oracle_lib):
    """As the adjoint's own test: J within 1e-12, the gradient within 1e-9 of its norm."""
    deck = problems.seeded(3, (20, 18, 16), 33, 6, 0, solver="cg", eps=1e-14, end_step=4, name="adj").tea_in()
    J, g, _ = gradient(deck, 4, 2, 1e-13, chip=False)
    Jc, gc = oracle_lib.adjoint3d(*read_config(deck, 3), BOX, 1e-13)
    assert J == pytest.approx(Jc, rel=1e-12)
    assert np.linalg.norm(g - gc) <= 1e-9 * np.linalg.norm(gc)
