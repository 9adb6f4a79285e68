"""The density scatter and the gathers at the grid shapes where their loops
turn over: spans of one cell, of a few, of more than a warp (32) and of more
layers than the row cache takes at once; grids narrower than the kernels
(windows folded at both edges), odd sizes, one, two and three dimensions.
FP64 against the numpy restatement on the same particles (1e-9 of the
largest density and the same number of loops, as test_gpu_gpkde), FP32
against FP64 (1e-3 of the largest density, as there)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mprw
from mprw import workloads as W
from mprw.model import ACTIVE, MIXED
from oracle import gpkde_oracle as GO

# (ncol, nrow, nlay), bin size along x, particles
SHAPES = [
    ((97, 1, 1), 1.0, 700),
    ((33, 7, 3), 1.0, 500),
    ((5, 3, 2), 1.0, 400),
    ((12, 10, 40), 1.0, 900),
    ((70, 5, 9), 0.5, 800),
]


@pytest.mark.parametrize("dims,bin_x,n", SHAPES)
def test_reconstruction_at_the_edges_of_the_loops(gpu_lib, dims, bin_x, n):
    ncol, nrow, nlay = dims
    g, f, p, opt, _ = W.lognormal_slab(n_particles=n, nlay=nlay, nrow=nrow, ncol=ncol, seed=4, use_torch=False)
    dom, bins = (float(ncol), float(nrow), float(nlay)), (bin_x, 1.0, 1.0)
    tr = mprw.Tracker(g, opt)
    tr.load_flow(f)
    tr.set_particles(p)
    tr.advance(0.0, 0.5)
    out = tr.get_particles()
    act = out["status"] == ACTIVE
    co = np.stack([out["gx"], out["gy"], out["gz"]], 1)[act]
    assert co.shape[0] >= 50  # particles left in the grid
    dens, hist, loops = tr.gpkde(dom, bins, n_opt_loops=3)
    d32, _, _ = tr.gpkde(dom, bins, n_opt_loops=3, precision=MIXED)
    tr.close()
    G = GO.GPKDE(dom, bins, n_opt_loops=3)
    ref, _ = G.compute_density(co, np.ones(co.shape[0]))
    assert loops == G.loops
    np.testing.assert_allclose(dens, ref.transpose(2, 1, 0), rtol=0, atol=1e-9 * ref.max())
    np.testing.assert_allclose(d32, dens, rtol=0, atol=1e-3 * dens.max())


@pytest.mark.parametrize("dims,n", [((61, 37, 9), 150_000), ((31, 29, 17), 20_000), ((523, 40, 1), 120_000)])
def test_needed_elements_of_the_gathers(gpu_lib, dims, n):
    """FP64 gathers over the elements that are read: more active bins than the
    16,384 from which the passes run down lists of them (and fewer, where
    they do not), plumes over odd grids whose windows fold at every face."""
    ncol, nrow, nlay = dims
    g, f, p, opt, _ = W.lognormal_slab(n_particles=8, nlay=nlay, nrow=nrow, ncol=ncol, seed=5, use_torch=False)
    p = W.release_in_box(g, n, 0.0, float(ncol), 0.0, float(nrow), float(g.botm[-1]), float(g.top[0]), seed=6)
    dom, bins = (float(ncol), float(nrow), float(nlay)), (1.0, 1.0, 1.0)
    tr = mprw.Tracker(g, opt)
    tr.load_flow(f)
    tr.set_particles(p)
    tr.advance(0.0, 0.01)
    out = tr.get_particles()
    act = out["status"] == ACTIVE
    co = np.stack([out["gx"], out["gy"], out["gz"]], 1)[act]
    dens, hist, loops = tr.gpkde(dom, bins, n_opt_loops=1)
    tr.close()
    assert ((hist > 0).sum() >= 16384) == (n > 100_000)
    G = GO.GPKDE(dom, bins, n_opt_loops=1)
    ref, _ = G.compute_density(co, np.ones(co.shape[0]))
    assert loops == G.loops
    np.testing.assert_allclose(dens, ref.transpose(2, 1, 0), rtol=0, atol=1e-9 * ref.max())


def test_small_reconstruction_on_a_stream_and_on_the_default_stream(gpu_lib):
    """Below the bins from which the loop runs on the device the host drives
    it, as a kept graph on a stream that can be captured and launch by launch
    on the legacy default stream: the same loops, the same bits, also for a
    second reconstruction that finds the kept graph."""
    g, f, p, opt = W.uniform_pulse(n_particles=5000)
    tr = mprw.Tracker(g, opt)
    tr.load_flow(f)
    tr.set_particles(p)
    for t0, t1 in ((0.0, 20.0), (20.0, 40.0)):
        tr.advance(t0, t1)
        d0, h0, l0 = tr.gpkde((200.0, 1.0, 1.0), (1.0, 1.0, 1.0))
        tr.set_stream(1)  # cudaStreamLegacy
        d1, h1, l1 = tr.gpkde((200.0, 1.0, 1.0), (1.0, 1.0, 1.0))
        tr.set_stream(0)
        assert l0 == l1 > 0
        np.testing.assert_array_equal(h0, h1)
        assert np.array_equal(d0.view(np.uint64), d1.view(np.uint64))
    tr.close()


@pytest.mark.parametrize("n", [1, 2, 3])
def test_few_particles_in_fp32(gpu_lib, n):
    """The FP32 scatter's fixed-point cell products at their largest scale:
    one particle's kernel spans from its centre to its last cell every
    magnitude from 2^60 units down, some below 2^23 (rounded) and most above
    (shifted).  Against FP64 to 1e-3 of the maximum and the mass to 1e-4, as
    test_gpu_gpkde."""
    g, f, p, opt, _ = W.lognormal_slab(n_particles=8, nlay=9, nrow=21, ncol=21, seed=7, use_torch=False)
    p = W.release_in_box(g, n, 9.0, 12.0, 9.0, 12.0, float(g.botm[-1]), float(g.top[0]), seed=8)
    tr = mprw.Tracker(g, opt)
    tr.load_flow(f)
    tr.set_particles(p)
    tr.advance(0.0, 0.001)
    d64, h64, l64 = tr.gpkde((21.0, 21.0, 9.0), (1.0, 1.0, 1.0), n_opt_loops=0)
    d32, h32, l32 = tr.gpkde((21.0, 21.0, 9.0), (1.0, 1.0, 1.0), n_opt_loops=0, precision=MIXED)
    tr.close()
    np.testing.assert_array_equal(h32, h64)
    assert h64.sum() == n and d64.max() > 0
    np.testing.assert_allclose(d32, d64, rtol=0, atol=1e-3 * d64.max())
    assert abs(d32.sum() - d64.sum()) < 1e-4 * n
