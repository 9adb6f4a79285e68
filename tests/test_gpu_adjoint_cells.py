"""The differentiable walk and its adjoint on cell sizes that are not powers
of two (quotients instead of exact reciprocals), narrow domains (many wall
reflections) and particle counts around a warp, against torch's autograd of
the restatement."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import mprw
from adjoint_cases import base_theta, block_zones
from mprw import workloads as W
from mprw.model import ACTIVE, EULERIAN, MIN_ADV_DISP, Flow, Options
from oracle import adjoint_oracle as A


@pytest.mark.parametrize("d", [(1.0, 1.0, 1.0), (0.7, 1.3, 0.3), (2.0, 0.9, 0.25)])
@pytest.mark.parametrize("n", [1, 31, 33])
def test_adjoint_on_odd_cells(gpu_lib, d, n):
    nlay, nrow, ncol, eps, dt, nsteps = 3, 4, 9, 0.05, 0.1, 25
    g = W.structured_grid(nlay, nrow, ncol, *d)
    K = W.lognormal_field(nlay, nrow, ncol, 1.0, 10.0, 10.0, 2.0, seed=4)
    s = W.steady_heads(g, K, use_torch=False)
    nc = g.ncell
    f = Flow(ia=s["ia"], ja=s["ja"], flowja=s["flowja"], porosity=np.full(nc, 0.25), retardation=np.ones(nc),
             iboundts=np.ones(nc, np.int32), alpha_l=np.array([0.5]), alpha_t=np.array([0.05]),
             dm_eff=np.array([1e-4]), heads=s["heads"], source_flow=s["source_flow"], sink_flow=s["sink_flow"])
    opt = Options(time_step_kind=MIN_ADV_DISP, ts_param=(0.1, 0.1), advection_kind=EULERIAN, stop_weak_sinks=True)
    size = (ncol * d[0], nrow * d[1], nlay * d[2])
    p = W.release_in_box(g, n, 0.2 * size[0], 0.8 * size[0], 0.0, size[1], 0.0, size[2], seed=n, status=ACTIVE)
    zones = block_zones(g)
    grid = dict(origin=(0.0, 0.0, 0.0), bin_size=d, n_bins=(ncol, nrow, nlay), h=tuple(1.5 * v for v in d))
    tr = mprw.Tracker(g, opt)
    tr.load_flow(f)
    tr.set_particles(p)
    tr.adj_setup(zones, 8, dt, nsteps, 10, grid["origin"], d, grid["n_bins"], grid["h"], eps, seed=11)
    th0 = base_theta()
    rho = tr.adj_forward(th0)
    w = np.random.default_rng(n).standard_normal(rho.shape)
    grad = tr.adj_backward(w)
    q = tr.get_particles()
    tr.close()
    ns = A.node_setup(g, f, opt, zones, 8)
    th = torch.tensor(th0, requires_grad=True)
    nodes = A.node_fields(ns, th, 8, d, eps)
    x0 = torch.tensor(np.stack([q["gx"], q["gy"], q["gz"]], 1))
    ref = A.deposit(A.walk(ns, nodes, x0, A.philox_walk_normals(11, p.id, nsteps), dt, (0.0, 0.0, 0.0), d, eps),
                    torch.ones(n, dtype=torch.float64), **grid)
    # the tolerances of the walk's test on unit cells
    np.testing.assert_allclose(rho, ref.detach().numpy(), rtol=0, atol=1e-12 * rho.max())
    (g_ref,) = torch.autograd.grad((ref * torch.tensor(w)).sum(), th)
    np.testing.assert_allclose(grad, g_ref.numpy(), rtol=0, atol=1e-9 * np.abs(g_ref.numpy()).max())
