"""A call that fails for want of device memory leaves nothing half made: whichever
of its allocations is refused, the next call makes what is missing and gives
what a fresh handle gives."""
import pytest

import malloc_limit

pytestmark = pytest.mark.gpu

BODY = """
import numpy as np
import malloc_limit
import mprw
from mprw import workloads as W

lim = malloc_limit.limit()
g, f, p, opt = W.uniform_pulse(n_particles=700)


def calls(tr):
    yield lambda: tr.load_flow(f)
    yield lambda: tr.set_particles(p)
    yield lambda: tr.advance(0.0, 5.0)
    yield lambda: tr.gpkde((200.0, 1.0, 1.0), (1.0, 1.0, 1.0))


def result(tr):
    for c in calls(tr):
        out = c()
    return out[0], tr.get_particles()["lx"]


with mprw.Tracker(g, opt) as tr:
    want = result(tr)
refused = 0
for step in range(4):
    k = 0
    while True:
        k += 1
        tr = mprw.Tracker(g, opt)
        todo = list(calls(tr))
        for c in todo[:step]:
            c()
        before = lim.malloc_limit_refused()
        lim.malloc_limit_refuse(k)
        try:
            todo[step]()
        except mprw.MprwError as e:
            assert "memory" in str(e), e
        lim.malloc_limit_refuse(0)
        hit = lim.malloc_limit_refused() > before
        refused += hit
        got = result(tr)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
        tr.close()
        if not hit:
            break
assert refused > 40, refused
"""


def test_every_refused_allocation_is_made_up_for(gpu_lib, tmp_path):
    malloc_limit.run(BODY, tmp_path)
