"""The order of the objects of one leaf, at the lengths where the way they are
sorted changes: one, two or four ids a lane of a warp, whole blocks from 129
on, and the network from 513 on."""
import numpy as np
import pytest

from glint_pipeline_gb300 import Configuration, DeviceBench
from glint_pipeline_gb300.tracegen import TraceGenerator
from oracle.bindings import Oracle, make_config
from test_gpu_parity import compare_meetings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision_mode", [0, 1])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1024, 1025])
def test_one_leaf(n, precision_mode):
    """All objects start in the root, a map too small to be split: one leaf of n."""
    gen = TraceGenerator(0x5E6 + n, n, 0, extent_m=40.0, n_hotspots=1, sigma_m=10.0, hotspot_frac=0.5)
    box, pts = gen.box(), gen.steps(3)
    args = dict(num_objects=n, num_meeting_buckets=1 << 23, grid_capacity=n, grid_amplify=1.0)
    o = Oracle(make_config(**args), box, pts[0])
    g = DeviceBench(Configuration(precision_mode=precision_mode, **args), box, pts[0])
    for t in range(3):
        o.step(pts[t], t)
        st = g.step(pts[t], t)
        c = o.counts()
        assert (st.checks, st.candidates, st.contacts) == (c.grid_check_counter, c.candidates, c.contacts), f"step {t}"
        if t == 0:
            assert st.candidates == n * (n - 1) // 2
        compare_meetings(o.meetings(), g.meetings(), t)
    g.close()
    o.close()


@pytest.mark.parametrize("capacity", [20, 70, 200, 400])
def test_dense_leaves(capacity):
    """Leaves of all lengths up to twice the buffer and beyond, over several
    steps: full buffers keep their first objects by id, whatever the route."""
    n = 6000
    gen = TraceGenerator(0x1EAF + capacity, n, 0, extent_m=1500.0, n_hotspots=4, sigma_m=8.0, hotspot_frac=0.8)
    box, pts = gen.box(), gen.steps(6)
    args = dict(num_objects=n, num_meeting_buckets=1 << 21, grid_capacity=capacity, grid_amplify=1.5)
    o = Oracle(make_config(**args), box, pts[0])
    g = DeviceBench(Configuration(precision_mode=1, **args), box, pts[0])
    for t in range(6):
        o.step(pts[t], t)
        st = g.step(pts[t], t)
        c = o.counts()
        assert (st.checks, st.candidates, st.contacts) == (c.grid_check_counter, c.candidates, c.contacts), f"step {t}"
        compare_meetings(o.meetings(), g.meetings(), t)
    g.close()
    o.close()
