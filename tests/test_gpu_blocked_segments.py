"""The z segments of the 3D blocked Chebyshev trips and PPCG inner steps are
cut for the number of x-y tiles: on meshes of few and many tiles, with one to
130 planes, blocked and one-launch-per-step solves leave the same memory
state, bit for bit."""
import numpy as np
import pytest

from tealeaf_b200 import problems
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["cheby", "ppcg"])
@pytest.mark.parametrize("cells", [(30, 20, 1), (28, 21, 2), (29, 20, 65), (31, 9, 130), (150, 130, 7), (90, 61, 64)])
def test_segments_are_bit_identical(cells, solver):
    text = problems.seeded(3, cells, 5, 4, 0, solver=solver, end_step=1, max_iters=47, error_switch=True,
                           eps_lim=1e30, ppcg_inner_steps=5, name="segments").tea_in()
    a, b = Host(text, 3), Host(text, 3)
    try:
        b.lib.tl3d_set_temporal_blocking(b.chunk, 0)
        ra, rb = a.solve_device(0), b.solve_device(0)
        assert ra.iterations == rb.iterations and ra.summary == rb.summary
        for f in ("u", "p", "r", "w", "sd", "energy"):
            assert np.array_equal(a.download(f), b.download(f)), f
    finally:
        a.finalise()
        b.finalise()
