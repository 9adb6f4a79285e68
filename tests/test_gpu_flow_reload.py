"""Flow steps loaded one after another on one handle: buffers are kept between
loads, so every load must give what a fresh handle gives, whichever optional
arrays it has and whatever was loaded (or refused) before."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mprw
from mprw import workloads as W

KEYS = ("cell", "status", "lx", "ly", "lz", "t", "rng_ctr", "gx", "gy", "gz")


def _variants():
    g, f, p, opt, _ = W.lognormal_slab(n_particles=3000, nlay=4, nrow=9, ncol=30, seed=3, use_torch=False)
    n = g.ncell
    rng = np.random.default_rng(1)
    out = [f]
    v = copy.copy(f)                                   # per-cell dispersion, masses bounded by cells
    v.uniform_dispersion = False
    v.alpha_l, v.alpha_t, v.dm_eff = rng.uniform(0.2, 0.8, n), rng.uniform(0.02, 0.08, n), np.full(n, 1e-4)
    v.icboundts = rng.integers(0, 2, n).astype(np.int32)
    out.append(v)
    v = copy.copy(f)                                   # convertible cells below their heads, boundary flows
    v.celltype = np.ones(n, np.int32)
    v.heads = g.botm + 0.4 * np.repeat(np.arange(1, 2), n) + 0.3 * rng.uniform(0.0, 1.0, n)
    v.boundary_flows = np.zeros(6 * n)
    v.boundary_flows[0] = 0.1
    out.append(v)
    v = copy.copy(f)                                   # no heads, no sources or sinks
    v.heads = v.source_flow = v.sink_flow = None
    v.porosity = rng.uniform(0.2, 0.3, n)
    out.append(v)
    return g, p, opt, out


def _run(tr, p):
    tr.set_particles(p)
    tr.advance(0.0, 3.0)
    return tr.get_particles()


def test_reloaded_steps_match_fresh_handles(gpu_lib):
    g, p, opt, flows = _variants()
    ref = []
    for f in flows:
        with mprw.Tracker(g, opt) as tr:
            tr.load_flow(f)
            ref.append(_run(tr, p))
    bad = copy.copy(flows[0])
    bad.flowja = bad.flowja.copy()
    bad.flowja[7] = np.nan
    tr = mprw.Tracker(g, opt)
    for k in (0, 1, 2, 3, 1, 0, 3, 2, 2):
        tr.load_flow(flows[k])
        if k % 2:
            with pytest.raises(mprw.MprwError, match="non-finite"):
                tr.load_flow(bad)
        o = _run(tr, p)
        for key in KEYS:
            np.testing.assert_array_equal(o[key], ref[k][key], err_msg=f"{k} {key}")
    tr.close()
    b = mprw.Batch([g, g], opt)                        # members: slices of the batch's arrays
    for ks in ((0, 1), (2, 3), (1, 0)):
        for m, k in enumerate(ks):
            b.load_flow(m, flows[k])
        b.set_particles([p, p])
        b.advance(0.0, 3.0)
        for m, k in enumerate(ks):
            o = b.members[m].get_particles()
            for key in KEYS:
                np.testing.assert_array_equal(o[key], ref[k][key], err_msg=f"batch {ks} {key}")
    b.close()


@pytest.mark.parametrize("field,value,what", [("porosity", 0.0, "porosity"), ("retardation", np.inf, "porosity"),
                                              ("heads", np.nan, "NaN head"), ("sink_flow", np.inf, "non-finite"),
                                              ("ja", 0, "JA entry"), ("ja", 10 ** 6, "JA entry")])
def test_bad_steps_are_refused(gpu_lib, field, value, what):
    g, p, opt, flows = _variants()
    tr = mprw.Tracker(g, opt)
    tr.load_flow(flows[0])
    good = _run(tr, p)
    for at in (0, -1):
        bad = copy.copy(flows[0])
        a = np.array(getattr(bad, field), copy=True)
        a[at] = value
        setattr(bad, field, a)
        with pytest.raises(mprw.MprwError, match=what):
            tr.load_flow(bad)
    o = _run(tr, p)
    for key in KEYS:
        np.testing.assert_array_equal(o[key], good[key], err_msg=key)
    tr.close()
