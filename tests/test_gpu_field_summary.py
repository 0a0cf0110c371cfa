"""run_field_summary, formed in parallel, against the serial loop it stands
for: the four sums equal, to the last bit, a left-to-right FP64 sum of the same
terms (numpy.cumsum), on fields that cross many binades, put terms half-way
between two values of the running sum, hold zeros, negative and non-finite
values, and on meshes around its tile (256 cells), super-tile (8192 cells)
and serial-loop (up to 12288 cells) sizes."""
import numpy as np
import pytest

from tealeaf_b200 import problems
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu

CELLS = {2: [(1, 1), (16, 16), (257, 1), (96, 128), (97, 127), (128, 129), (640, 333)],
         3: [(16, 16, 1), (24, 32, 16), (23, 24, 25), (33, 40, 67)]}


def fields(kind, shape, rng):
    n = rng.random(shape)
    if kind == "plain":
        return 1.0 + 99.0 * n, n, rng.random(shape)
    if kind == "binades":      # terms over 120 binades, zeros among them
        return np.exp2(np.floor(120.0 * n) - 60.0), np.where(n < 0.3, 0.0, n), np.exp2(40.0 * n)
    if kind == "halves":       # few significant bits: half-way cases in every binade of the sum
        return np.exp2(np.floor(40.0 * n)) * 3.0, np.exp2(-np.floor(30.0 * n)), 1.0 + np.floor(4.0 * n) / 4.0
    if kind == "zeros":        # the running sum stays 0 over long runs
        z = np.zeros(shape)
        z.reshape(-1)[-3:] = 0.7
        return z, n, z.copy()
    if kind == "signs":
        return 1.0 + n, n - 0.5, np.where(n < 0.001, -5.0, n)
    out = 1.0 + n, n.copy(), rng.random(shape)
    out[1].reshape(-1)[n.size // 2] = np.inf
    out[2].reshape(-1)[n.size // 3] = np.nan
    return out


@pytest.mark.parametrize("kind", ["plain", "binades", "halves", "zeros", "signs", "special"])
@pytest.mark.parametrize("dims", [2, 3])
def test_summary_is_the_serial_sum(dims, kind):
    rng = np.random.default_rng(17)
    for cells in CELLS[dims]:
        h = Host(problems.seeded(dims, cells, 3, 2, 0, solver="cg", end_step=1, name="sum").tea_in(), dims)
        try:
            rho, e, u = fields(kind, h.shape, rng)
            vol = np.full(h.shape, 0.3) if kind != "halves" else np.full(h.shape, 0.25)
            for name, f in (("density", rho), ("energy0", e), ("u", u), ("volume", vol)):
                h.upload(name, f)
            got = h.field_summary()
            inner = tuple(slice(h.cfg.halo_depth, -h.cfg.halo_depth) for _ in range(dims))
            v, r, e, u = (f[inner].reshape(-1) for f in (vol, rho, e, u))
            m = v * r
            with np.errstate(invalid="ignore"):
                want = [np.cumsum(t)[-1] for t in (v, m, m * e, m * u)]
            assert np.array_equal(np.array(got), np.array(want), equal_nan=True), (cells, got, want)
        finally:
            h.finalise()
