"""A flow time step that is loaded again takes no more device memory than the
first: it loads on a device that has none left, and a load refused there or
elsewhere leaves the step before it in use, for advances and for the
differentiable walk."""
import pytest

import malloc_limit

pytestmark = pytest.mark.gpu

BODY = """
import copy
import numpy as np
import malloc_limit
import mprw
from mprw import workloads as W

lim = malloc_limit.limit()
g, f, p, opt, _ = W.lognormal_slab(n_particles=4000, nlay=5, nrow=15, ncol=40, seed=3, use_torch=False)
n = g.ncell
rng = np.random.default_rng(5)
cells = copy.copy(f)                       # dispersion by cell
cells.uniform_dispersion = False
cells.alpha_l, cells.alpha_t, cells.dm_eff = rng.uniform(0.2, 0.8, n), rng.uniform(0.02, 0.08, n), np.full(n, 2e-4)
cells.retardation = np.full(n, 1.5)
other = copy.copy(cells)
other.flowja, other.dm_eff, other.retardation = f.flowja * 1.1, np.full(n, 3e-4), np.full(n, 2.0)
bad = []
for field, value in (("flowja", np.nan), ("retardation", 0.0), ("dm_eff", np.inf)):
    b = copy.copy(other)
    setattr(b, field, getattr(b, field).copy())
    getattr(b, field)[5] = value
    b.iboundts = np.zeros(n, np.int32)
    bad.append(b)


def state(tr):
    tr.set_particles(p)
    tr.advance(0.0, 3.0)
    o = tr.get_particles(global_xyz=False)
    return [o[k] for k in ("cell", "status", "lx", "ly", "lz", "t", "rng_ctr")]


def walk(tr):
    tr.adj_setup(np.zeros(n, np.int32), 1, 0.05, 10, 5, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), (40, 15, 5), (2.0, 2.0, 1.0),
                 0.01, seed=1)
    return tr.adj_forward(np.array([0.5, 0.05, 0.25, 1.0]))


want = {}
for name, flow in (("cells", cells), ("other", other)):
    with mprw.Tracker(g, opt) as tr:
        tr.load_flow(flow)
        want[name] = state(tr)
        want[name].append(walk(tr))

for room in (False, True):
    tr = mprw.Tracker(g, opt)
    tr.load_flow(cells)
    if not room:
        lim.malloc_limit_set(lim.malloc_limit_live())
    for b in bad:
        try:
            tr.load_flow(b)
        except mprw.MprwError as e:
            assert "must be" in str(e) or "non-finite" in str(e), e
        else:
            raise AssertionError("a bad step was loaded")
    tr.load_flow(other)
    tr.load_flow(cells)
    for b in bad:
        try:
            tr.load_flow(b)
        except mprw.MprwError as e:
            assert "must be" in str(e) or "non-finite" in str(e), e
        else:
            raise AssertionError("a bad step was loaded")
    lim.malloc_limit_set(2 ** 62)
    got = state(tr)
    got.append(walk(tr))
    for a, b in zip(got, want["cells"]):
        np.testing.assert_array_equal(a, b)
    tr.load_flow(other)
    got = state(tr)
    got.append(walk(tr))
    for a, b in zip(got, want["other"]):
        np.testing.assert_array_equal(a, b)
    tr.close()
"""


def test_a_step_loads_again_without_more_memory(gpu_lib, tmp_path):
    malloc_limit.run(BODY, tmp_path)
