"""The device-resident CG loop of meshes that do not fit on chip applies the u
updates of two trips in one w sweep: for loops that end after an even and an
odd number of trips, and for rows fed by TMA and by per-thread loads, every
field equals that of the run_* path (u updated in every trip), bit for bit."""
import numpy as np
import pytest

from tealeaf_b200 import problems
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu

FIELDS = {2: ("u", "u0", "p", "r", "w", "kx", "ky", "sd", "energy"),
          3: ("u", "u0", "p", "r", "w", "kx", "ky", "kz", "sd", "energy")}


@pytest.mark.parametrize("cap", [1, 2, 3, 4, 5, 24])
@pytest.mark.parametrize("dims,cells", [(2, (1300, 1001)), (2, (1301, 1000)), (3, (128, 120, 90)), (3, (127, 119, 91))])
def test_deferred_updates_are_bit_identical(dims, cells, cap):
    text = problems.seeded(dims, cells, 13, 5, 0, solver="cg", end_step=2, max_iters=cap, name="defer").tea_in()
    a, b = Host(text, dims), Host(text, dims)
    try:
        for tt in range(2):   # the second step starts from whatever buffers the first left
            ra, rb = a.solve(tt), b.solve_device(tt)
            assert ra.iterations == rb.iterations and ra.error == rb.error and ra.summary == rb.summary
            for f in FIELDS[dims]:
                assert np.array_equal(a.download(f), b.download(f)), (tt, f)
        # and the run_* path goes on from them
        ra, rb = a.solve(2), b.solve(2)
        assert ra.error == rb.error and np.array_equal(a.download("u"), b.download("u"))
    finally:
        a.finalise()
        b.finalise()
