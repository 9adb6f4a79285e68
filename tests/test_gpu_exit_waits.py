"""EXPONENTIAL advection: a particle that would leave its cell waits, with its
pass unmade, until enough of its warp would leave or it has waited for some
passes.  Its path does not depend on the company it waits in: the same
particles one by one, in small pieces and all together, where most passes end
at a face and where few do (a tenth of the time step), with anisotropic and
axisymmetric dispersion."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mprw
from mprw import workloads as W
from mprw.model import EXPONENTIAL, FP64, MIXED, Particles

KEYS = ("cell", "status", "lx", "ly", "lz", "t", "rng_ctr")


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("axisymmetric", [False, True])
@pytest.mark.parametrize("ts,days", [(0.1, 3.0), (0.005, 0.4)])
def test_paths_do_not_depend_on_the_waiting(gpu_lib, precision, axisymmetric, ts, days):
    n = 2_100
    g, f, p, opt, _ = W.lognormal_slab(n_particles=n, nlay=4, nrow=12, ncol=30, seed=11, precision=precision,
                                       use_torch=False)
    opt.advection_kind = EXPONENTIAL
    opt.ts_param = (ts, ts)
    if axisymmetric:
        f = W.Flow(**{**f.__dict__, "alpha_lv": np.array([0.2]), "alpha_tv": np.array([0.01])})
        opt.dispersion_model = 1

    def run(sel):
        tr = mprw.Tracker(g, opt)
        tr.load_flow(f)
        tr.set_particles(Particles(**{k: getattr(p, k)[sel] for k in ("cell", "lx", "ly", "lz", "t", "status", "mass",
                                                                      "id", "rng_ctr")}))
        steps = tr.advance(0.0, days)
        o = tr.get_particles(global_xyz=False)
        tr.close()
        return steps, o

    steps, full = run(slice(0, n))
    total = 0
    for a, b in ((0, 1), (1, 2), (2, 40), (40, 300), (300, n)):
        s, o = run(slice(a, b))
        total += s
        for k in KEYS:
            np.testing.assert_array_equal(o[k], full[k][a:b], err_msg=f"{a}:{b} {k}")
    assert total == steps > n
