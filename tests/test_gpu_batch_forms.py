"""The batch's persistent kernel at the edges of its row copies and schedules.

Tile rows that do not divide the height, widths around a tile's 256 columns and
a warp's 64, more problems than blocks, and the two forms of the kernel (arrays
that fit L2, and not): temperatures against the problem's own sequential FP64
solve (FP32 vectors, FP64 stop: the tolerance of the batch's other tests), and
bit-identical results for the same problem and tile height in any company.
"""
import numpy as np
import pytest

from tealeaf_b200 import problems
from tealeaf_b200.batch import Batch
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu

TEMP_RTOL = 1e-6
EDGES = [(2, 3), (63, 16), (64, 17), (65, 1), (1, 70), (255, 33), (256, 15), (257, 32), (320, 47), (513, 5)]


def _step(probs, rows, pick):
    b = Batch([p.tea_in() for p in probs], tile_rows=rows)
    try:
        st = b.step()
        assert st.converged == len(probs)
        it, rr, _ = b.results()
        return [(int(it[k]), float(rr[k]), b.hosts[k].download("energy")) for k in pick], b.summaries()
    finally:
        b.close()


@pytest.mark.parametrize("rows", [16, 5, 2])
def test_tile_edges_match_the_fp64_solve(rows):
    probs = [problems.seeded(2, s, 40 + k, 3, 0, solver="cg", eps=1e-12, end_step=1) for k, s in enumerate(EDGES)]
    _, sums = _step(probs, rows, [])
    for p, s in zip(probs, sums):
        h = Host(p.tea_in(), 2)
        try:
            ref = h.solve_device(0).summary
        finally:
            h.finalise()
        assert s[0] == ref[0] and s[1] == ref[1] and s[2] == ref[2]
        assert abs(s[3] / ref[3] - 1.0) < TEMP_RTOL, (p.cells, s[3], ref[3])


@pytest.mark.parametrize("company", ["streaming", "crowd"])
def test_a_problem_does_not_depend_on_its_company(company):
    if company == "streaming":   # 28 bytes of arrays a cell: beyond L2 together
        probs = problems.batched_2d(1, seed=3, lo=300, hi=700) + problems.batched_2d(3, seed=4, lo=1700, hi=1900)
        pick = [0]
    else:   # more problems than the kernel has blocks
        probs = problems.batched_2d(1300, seed=6, lo=6, hi=14)[:1184]
        pick = [0, 31, 32, 600, 1183]
    got, _ = _step(probs, 16, pick)
    for k, (it, rr, e) in zip(pick, got):
        (it1, rr1, e1), = _step([probs[k]], 16, [0])[0]
        assert it == it1 and rr == rr1
        assert np.array_equal(e, e1)
