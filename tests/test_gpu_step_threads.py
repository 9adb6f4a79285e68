"""Handles in several host threads: the step kernel's launches of few particles
take less shared memory per block than those of many, and neither may have the
other's refused."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import mprw
from mprw import workloads as W


def test_handles_with_few_and_many_particles_advance_side_by_side(gpu_lib):
    trackers, errors = [], []
    for n in (3, 8_000, 70_000):   # one warp per SM, four, all
        g, f, p, opt = W.uniform_pulse(n_particles=n)
        tr = mprw.Tracker(g, opt)
        tr.load_flow(f)
        tr.set_particles(p)
        trackers.append(tr)
    start = threading.Barrier(len(trackers))

    def many_short_advances(tr):
        start.wait()
        try:
            for k in range(3000):
                tr.advance(1e-6 * k, 1e-6 * (k + 1))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=many_short_advances, args=(tr,)) for tr in trackers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for tr in trackers:
        o = tr.get_particles(global_xyz=False)
        assert np.isfinite(o["lx"]).all() and np.all(o["rng_ctr"] > 0)
        tr.close()
