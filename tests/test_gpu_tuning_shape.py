"""mprw_autotune with few particles: every block count gives the same launch, and
the default is kept rather than the luckiest of equal trials."""
import pytest

pytestmark = pytest.mark.gpu

import mprw
from mprw import workloads as W
from mprw.model import MIXED


def test_equal_launches_keep_the_default(gpu_lib):
    g, f, p, opt = W.uniform_pulse(n_particles=5000, precision=MIXED)
    tr = mprw.Tracker(g, opt)
    tr.load_flow(f)
    tr.set_particles(p)
    default = tr.tuning()["blocks_per_sm"]
    assert default > 1
    assert [tr.autotune(0.0, 2.0)["blocks_per_sm"] for _ in range(8)] == [default] * 8
    tr.close()
