"""The time-series GPKDE's ways to its kernel taps: a table of them, values
cached per block, or every tap evaluated where it is used (long grids, kernels
of thousands of bins), against the numpy restatement; and its record
statistics and histogram at block edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mprw
from oracle import series_oracle as SO


def _check(t, w, **kw):
    got, ref = mprw.gpkde_series(t, w, **kw), SO.gpkde_series(t, w, **kw)
    assert got["n_bins"] == ref["n_bins"] and got["loops"] == ref["loops"]
    # counts: fixed-point sums; density: the same taps in another order (the
    # tolerances of the other series tests)
    np.testing.assert_allclose(got["counts"], ref["counts"], rtol=0, atol=1e-12 * ref["counts"].max())
    np.testing.assert_allclose(got["density"], ref["density"], rtol=0, atol=1e-10 * ref["density"].max())


@pytest.mark.parametrize("bins,factor", [(600, 3.0),      # table
                                         (600, 260.0),    # the initial kernel wider than the table
                                         (2300, 3.0),     # no table
                                         (2300, 720.0)])  # no table, kernels wider than a block's cache
def test_tap_paths(gpu_lib, bins, factor):
    rng = np.random.default_rng(bins)
    t = rng.lognormal(np.log(60.0), 0.3, 40)
    _check(t, rng.uniform(0.5, 1.5, t.size), domain_size=200.0, bin_size=200.0 / bins, bin_format=2,
           init_selection=1, init_factor=factor, n_opt_loops=2, skip_error=True)


@pytest.mark.parametrize("n", [1, 255, 257, 8193, 78_000])
@pytest.mark.parametrize("fmt", [0, 3])
@pytest.mark.parametrize("bins", [50, 9000])   # histogram in shared memory, and past its size with two grids
def test_statistics_and_histogram(gpu_lib, n, fmt, bins):
    rng = np.random.default_rng(n)
    t, w = rng.uniform(0.0, 90.0, n), rng.uniform(0.5, 1.5, n)
    kw = dict(domain_size=90.0, bin_size=90.0 / bins, bin_format=2, eff_format=fmt, only_histogram=True)
    got, ref = mprw.gpkde_series(t, w, **kw), SO.gpkde_series(t, w, **kw)
    assert got["n_bins"] == ref["n_bins"] == bins
    np.testing.assert_allclose(got["counts"], ref["counts"], rtol=0, atol=1e-12 * ref["counts"].max())
