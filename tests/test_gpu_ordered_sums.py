"""Weighted histograms: per-bin sums and totals equal the sequential sums in
particle order to the bit, whatever the weights (ties, changes of binade,
zeros, tiny, huge and negative weights) and the particle count (edges of the
summation tiles, runs of one to thousands of particles per bin)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mprw
from mprw import workloads as W
from mprw.model import ACTIVE, BOUNDARY, Options, Particles
from oracle import gpkde_oracle as GO


def _weights(kind, n, rng):
    if kind == "uniform":
        return rng.uniform(0.1, 2.0, n)
    if kind == "tenth":
        return np.full(n, 0.1)
    if kind == "ties":          # half units of the running sum's binade, among others
        w = np.where(rng.random(n) < 0.5, 2.0 ** -53, 2.0 ** -52) * rng.integers(1, 4, n)
        w[0] = 1.0
        return w
    if kind == "dynamic":       # many orders of magnitude, zeros and subnormals
        w = 10.0 ** rng.uniform(-40.0, 20.0, n)
        w[rng.random(n) < 0.1] = 0.0
        w[rng.random(n) < 0.05] = 5e-324
        return w
    if kind == "rising":
        return 1.001 ** np.arange(n) if n < 100_000 else np.arange(1.0, n + 1.0)
    w = rng.uniform(0.1, 2.0, n)  # one negative weight late in the order
    w[-max(1, n // 3)] = -0.05
    return w


@pytest.mark.parametrize("n", [1, 7, 9, 2047, 2049, 70_000])
@pytest.mark.parametrize("kind", ["uniform", "tenth", "ties", "dynamic", "rising", "negative"])
def test_ordered_sums_are_sequential(gpu_lib, kind, n):
    rng = np.random.default_rng(n)
    g = W.structured_grid(2, 9, 40)
    lx, ly, lz = rng.uniform(0.0, 1.0, (3, n))
    # a third of the particles in one cell: long runs beside short ones
    cell = np.where(rng.random(n) < 0.33, 17, rng.integers(1, g.ncell + 1, n)).astype(np.int32)
    status = np.where(rng.random(n) < 0.2, BOUNDARY, ACTIVE).astype(np.int32)
    status[0] = ACTIVE
    mass = _weights(kind, n, rng)
    tr = mprw.Tracker(g, Options())
    tr.set_particles(Particles(cell=cell, lx=lx, ly=ly, lz=lz, t=np.zeros(n), status=status, mass=mass))
    o = tr.get_particles()
    act = status == ACTIVE
    xyz = np.stack([o["gx"], o["gy"], o["gz"]], 1)[act]
    for origin, size, nb in (((0.0, 0.0, 0.0), (1.0, 1.0, 1.0), (40, 9, 2)),
                             ((5.0, 0.0, 0.0), (2.0, 0.0, 0.0), (10, 1, 1))):
        c, _, eff = tr.histogram(origin, size, nb)
        ref, _, reff = GO.histogram_weighted(xyz, mass[act], origin, size, nb)
        assert eff == reff
        np.testing.assert_array_equal(c, ref)
    tr.close()
