"""mprw_autotune times the processing order that an advance over its interval
would run in, whatever was advanced before: a handle that has advanced over
that interval and one that has never advanced give the same rates.  The
particles are such that the order shows: most have two days of the interval to
go, a few all hundred, and those lie in the last cells, so that by cell the
long ones start when everything else has ended."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mprw
from mprw import workloads as W
from mprw.model import ACTIVE, MIXED, Particles

T = 100.0


def _handle(n):
    g, f = W.uniform_flow(ncol=400, q=0.3, porosity=0.3, alpha_l=0.1, alpha_t=0.01)
    opt = W.uniform_pulse(n_particles=1, precision=MIXED)[3]
    rng = np.random.default_rng(2)
    cell, t = np.full(n, 11, np.int32), np.full(n, T - 2.0)
    late = rng.choice(n, 600, replace=False)
    cell[late], t[late] = 201, 0.0
    p = Particles(cell=cell, lx=np.zeros(n), ly=np.full(n, 0.5), lz=np.full(n, 0.5), t=t,
                  status=np.full(n, ACTIVE, np.int32), mass=np.ones(n), id=np.arange(n, dtype=np.uint64),
                  rng_ctr=np.zeros(n, np.uint64))
    tr = mprw.Tracker(g, opt)
    tr.load_flow(f)
    tr.set_particles(p)
    return tr, p


def test_autotune_times_the_order_its_interval_runs_in(gpu_lib):
    n = 2_000_000
    best = {}
    for name in ("fresh", "advanced"):
        rates = []
        for _ in range(3):
            tr, p = _handle(n)
            if name == "advanced":
                tr.advance(0.0, T)
                tr.set_particles(p)
            rates.append(tr.autotune(0.0, T)["trial_rates_per_ms"][0])
            tr.close()
        best[name] = max(rates)
    # (by cell: 0.68)
    assert best["fresh"] > 0.85 * best["advanced"], best
