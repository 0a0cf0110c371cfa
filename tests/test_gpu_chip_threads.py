"""Two host threads, each stepping a 3D chunk of its own whose CG loop runs on
chip with the same kernel (pencils of 4 planes, one to a unit) but a different
number of units per block, so of shared memory: neither launch may depend on
what the other thread is about to launch."""
import threading

import numpy as np
import pytest

from tealeaf_b200 import problems
from tealeaf_b200.host import Host

pytestmark = pytest.mark.gpu

STEPS = 400


def _host(cells):
    return Host(problems.seeded(3, cells, 11, 4, 0, solver="cg", end_step=1, max_iters=2, name="two").tea_in(), 3)


def test_two_threads_launch_the_same_loop_with_different_blocks():
    hosts = [_host((64, 64, 64)), _host((64, 64, 20))]   # two units per block, one
    want = []
    for h in hosts:
        e = h.download("energy")
        h.solve_device(0, summary=False)
        want.append((e, h.download("u")))
    failures = []
    start = threading.Barrier(2)

    def run(h, e, u):
        start.wait()
        try:
            for tt in range(STEPS):
                h.solve_device(tt, summary=False)
            h.upload("energy", e)
            h.solve_device(0, summary=False)
            if not np.array_equal(h.download("u"), u):
                failures.append("u")
        except Exception as exc:
            failures.append(str(exc))

    try:
        threads = [threading.Thread(target=run, args=(h, *w)) for h, w in zip(hosts, want)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failures
    finally:
        for h in hosts:
            h.finalise()
