"""The CG loop held on chip (k_cg_chip) against the same loop through run_*
(one launch per sweep): every field, iteration count and summary bit for bit,
at the edges of its tiling -- strips of 2 to 8 rows, single strips and odd
numbers of them, ragged last strips, meshes one column past a warp or a
128-column band, caps of 1 and 2 trips and a solve to convergence."""
import ctypes as C

import numpy as np
import pytest

from tealeaf_b200 import problems
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu

FIELDS2 = ("u", "u0", "p", "r", "w", "kx", "ky", "energy")


def both(dims, cells, cap, steps=1, **kw):
    text = problems.seeded(dims, cells, 11, 4, 0 if dims == 3 else 2, solver="cg", end_step=steps,
                           max_iters=cap, name="chip", **kw).tea_in()
    return Host(text, dims), Host(text, dims)


@pytest.mark.parametrize("cells,cap,steps", [
    ((5, 1), 3, 1), ((2, 3), 20000, 2), ((33, 5), 20000, 2), ((32, 2), 40, 1), ((129, 37), 20000, 2),
    ((65, 4), 1, 1), ((257, 129), 2, 1), ((640, 61), 30, 1), ((1024, 440), 25, 1), ((513, 941), 25, 1),
    ((1000, 700), 25, 1), ((900, 880), 25, 1), ((1025, 900), 25, 1), ((1000, 1180), 25, 1), ((1024, 1184), 25, 1),
])
def test_chip_cg_is_bit_identical(cells, cap, steps):
    a, b = both(2, cells, cap, steps)
    try:
        n0 = b.lib.tl2d_launch_count(C.byref(b.chunk))
        for tt in range(steps):
            ra, rb = a.solve(tt), b.solve_device(tt)
            assert ra.iterations == rb.iterations
            assert ra.error == rb.error
            assert ra.summary == rb.summary
            for f in FIELDS2:
                assert np.array_equal(a.download(f), b.download(f)), (tt, f)
        # the whole loop ran as one launch, not two per trip
        assert b.lib.tl2d_launch_count(C.byref(b.chunk)) - n0 <= 16 * steps
    finally:
        a.finalise()
        b.finalise()


def test_chip_cg_two_chunks_in_turn():
    """Two chunks of different sizes stepped in turn keep their own words."""
    a, b = both(2, (130, 66), 20000, 3)
    c, d = both(2, (70, 300), 20000, 3)
    try:
        for tt in range(3):
            for x, y in ((a, b), (c, d)):
                assert x.solve(tt).iterations == y.solve_device(tt).iterations
                assert np.array_equal(x.download("u"), y.download("u"))
    finally:
        for h in (a, b, c, d):
            h.finalise()


@pytest.mark.parametrize("pc", ["jac_diag", "jac_block"])
@pytest.mark.parametrize("cells,cap", [
    ((5, 3), 20000), ((33, 7), 20000), ((129, 38), 20000), ((1024, 442), 25), ((641, 941), 25), ((1000, 702), 25),
    ((900, 880), 25), ((1025, 900), 25), ((1000, 1181), 25),
])
def test_chip_pcg_against_the_oracle(cells, cap, pc, oracle_lib):
    """The preconditioned loop on chip: trip counts as the oracle's, the
    summary within 1e-12 of its."""
    from tealeaf_b200.config import read_config
    text = problems.seeded(2, cells, 11, 4, 2, solver="cg", end_step=1, max_iters=cap, preconditioner=pc,
                           name="chip").tea_in()
    cfg, states = read_config(text, 2)
    want = oracle_lib.run(cfg, states)[0]
    h = Host(text, 2)
    try:
        n0 = h.lib.tl2d_launch_count(C.byref(h.chunk))
        got = h.solve_device(0)
        assert h.lib.tl2d_launch_count(C.byref(h.chunk)) - n0 <= 18
        assert got.iterations == want.iterations
        for x, y in zip(got.summary, want.summary):
            assert abs(x - y) <= 1e-12 * abs(y)
    finally:
        h.finalise()


FIELDS3 = ("u", "u0", "p", "r", "w", "kx", "ky", "kz", "energy")


@pytest.mark.parametrize("cells,cap,steps", [
    ((5, 1, 1), 3, 1), ((3, 2, 4), 20000, 1), ((33, 9, 5), 20000, 2), ((32, 8, 17), 40, 1), ((65, 17, 33), 60, 2),
    ((48, 48, 48), 1, 1), ((48, 47, 50), 30, 1), ((96, 96, 65), 20, 1), ((97, 90, 100), 20, 1), ((16, 16, 16), 50, 1),
    ((100, 90, 80), 20, 1), ((64, 63, 150), 20, 1), ((120, 100, 77), 20, 1), ((64, 156, 78), 20, 1),
    ((39, 133, 82), 20, 1), ((149, 43, 104), 20, 1), ((133, 32, 98), 20, 1), ((128, 128, 72), 20, 1),
])
def test_chip_cg_3d_is_bit_identical(cells, cap, steps):
    """k3_cg_chip against the two launches per trip of the run_* path: units of
    one to four pencils of 4, 5 and 6 planes, ragged in every direction."""
    a, b = both(3, cells, cap, steps)
    try:
        for tt in range(steps):
            ra, rb = a.solve(tt), b.solve_device(tt)
            assert ra.iterations == rb.iterations
            assert ra.error == rb.error
            assert ra.summary == rb.summary
            for f in FIELDS3:
                assert np.array_equal(a.download(f), b.download(f)), (tt, f)
    finally:
        a.finalise()
        b.finalise()


@pytest.mark.parametrize("dims,cells", [
    (2, (129, 37)), (2, (513, 941)), (2, (1025, 900)), (2, (1000, 1180)), (2, (97, 61)),
    (3, (33, 9, 5)), (3, (39, 133, 82)), (3, (100, 90, 80)), (3, (65, 17, 33)),
])
def test_chip_cg_on_a_rough_density(dims, cells):
    """Every face coefficient different from its neighbours, those on the
    domain's edge included."""
    a, b = both(dims, cells, 30)
    rng = np.random.default_rng(5)
    try:
        rho = 0.05 + 20.0 * rng.random(a.shape)
        for h in (a, b):
            h.upload("density", rho)
        ra, rb = a.solve(0), b.solve_device(0)
        assert ra.iterations == rb.iterations and ra.error == rb.error
        for f in FIELDS2 if dims == 2 else FIELDS3:
            assert np.array_equal(a.download(f), b.download(f)), f
    finally:
        a.finalise()
        b.finalise()
