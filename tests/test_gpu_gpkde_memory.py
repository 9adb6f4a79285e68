"""What a reconstruction holds on the device: its pass buffers (60 elements of 8
bytes and a mask byte per bin of the grid, twice), nine grids, the counts, two
indexes by bin -- 1,168 bytes a bin -- and the arrays of its active bins, few
here.  On a device with 1,200 left it runs, in either precision."""
import pytest

import malloc_limit

pytestmark = pytest.mark.gpu

BODY = """
import numpy as np
import malloc_limit
import mprw
from mprw import workloads as W
from mprw.model import ACTIVE, FP64, MIXED, Options, Particles

lim = malloc_limit.limit()
nlay, nrow, ncol, n = 50, 100, 100, 2000
g = W.structured_grid(nlay, nrow, ncol)
rng = np.random.default_rng(1)
cell = (rng.integers(20, 24, n) * nrow * ncol + rng.integers(40, 46, n) * ncol + rng.integers(40, 46, n) + 1)
p = Particles(cell=cell.astype(np.int32), lx=rng.random(n), ly=rng.random(n), lz=rng.random(n), t=np.zeros(n),
              status=np.full(n, ACTIVE, np.int32), mass=np.ones(n), id=np.arange(n, dtype=np.uint64),
              rng_ctr=np.zeros(n, np.uint64))
for precision in (FP64, MIXED):
    out = []
    for room in (True, False):
        tr = mprw.Tracker(g, Options(precision=precision))
        tr.set_particles(p)
        if not room:
            lim.malloc_limit_set(lim.malloc_limit_live() + 1200 * nlay * nrow * ncol)
        out.append(tr.gpkde((float(ncol), float(nrow), float(nlay)), (1.0, 1.0, 1.0), precision=precision))
        lim.malloc_limit_set(2 ** 62)
        tr.close()
    assert lim.malloc_limit_refused() == 0
    assert out[0][2] == out[1][2]
    np.testing.assert_array_equal(out[0][0], out[1][0])
"""


def test_a_reconstruction_runs_in_the_memory_its_buffers_take(gpu_lib, tmp_path):
    malloc_limit.run(BODY, tmp_path)
