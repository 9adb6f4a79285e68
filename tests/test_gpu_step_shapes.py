"""Launch shapes of the step kernel: few particles run in fewer warps and lanes
per SM, and no particle's result depends on the shape it ran in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mprw
from mprw import workloads as W
from mprw.model import EULERIAN, EXPONENTIAL, FP64, MIXED, Particles

KEYS = ("cell", "status", "lx", "ly", "lz", "t", "rng_ctr")


def _run(g, f, opt, p):
    tr = mprw.Tracker(g, opt)
    tr.load_flow(f)
    tr.set_particles(p)
    steps = tr.advance(0.0, 4.0) + tr.advance(4.0, 6.0)
    o = tr.get_particles(global_xyz=False)
    tr.close()
    return steps, o


def _part(p, sel):
    return Particles(**{k: getattr(p, k)[sel] for k in ("cell", "lx", "ly", "lz", "t", "status", "mass", "id",
                                                        "rng_ctr")})


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("advection", [EULERIAN, EXPONENTIAL])
def test_results_do_not_depend_on_the_launch_shape(gpu_lib, precision, advection):
    n = 61_000 if advection == EULERIAN else 5_000   # past one particle per lane: every warp full
    g, f, p, opt, info = W.lognormal_slab(n_particles=n, nlay=4, nrow=12, ncol=30, seed=9, precision=precision,
                                          use_torch=False)
    opt.advection_kind = advection
    steps, full = _run(g, f, opt, p)
    # the same particles in pieces of 1 to 32 particles per SM and beyond
    cuts = [0, 1, 3, 33, 152, 304, 700, 2_000, 5_000, 20_000, 25_000, 45_000, 61_000]
    cuts = [c for c in cuts if c <= n]
    if cuts[-1] != n:
        cuts.append(n)
    total = 0
    for a, b in zip(cuts[:-1], cuts[1:]):
        s, o = _run(g, f, opt, _part(p, slice(a, b)))
        total += s
        for k in KEYS:
            np.testing.assert_array_equal(o[k], full[k][a:b], err_msg=f"{a}:{b} {k}")
    assert total == steps


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_results_do_not_depend_on_the_processing_order(gpu_lib, precision):
    """Particles are taken heaviest first: by their passes of the previous
    advance, or by the time they have over their cell's time step.  With that
    order and with none: active and pending particles, a second interval, the
    same particles handed over again, a different number of them."""
    n = 130_000   # more than one round of lanes in either precision
    g, f, p, opt, _ = W.lognormal_slab(n_particles=n, nlay=4, nrow=12, ncol=30, seed=13, precision=precision,
                                       use_torch=False)
    rng = np.random.default_rng(3)
    p.status = np.where(rng.random(n) < 0.3, 0, p.status).astype(p.status.dtype)
    p.t = np.where(p.status == 0, rng.uniform(0.0, 7.0, n), 0.0)
    out = []
    for interval in (1, 0):
        tr = mprw.Tracker(g, opt)
        tr.load_flow(f)
        tr.set_tuning(0, interval)
        states = []
        for sel in (slice(0, n), slice(0, n), slice(0, 500)):
            tr.set_particles(_part(p, sel))
            for a, b in ((0.0, 4.0), (4.0, 6.0)):
                states.append((tr.advance(a, b), tr.get_particles(global_xyz=False)))
        tr.close()
        out.append(states)
    for (s0, a), (s1, b) in zip(*out):
        assert s0 == s1 > 0
        for k in KEYS:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
