"""The refine stage's pair enumeration and screening against the oracle, at
the leaf sizes and map sizes where they can go wrong: leaves of one, two and
about 32 members and their neighbours, leaf buffers far larger than a warp,
work items of few and many checks, and maps so wide that the longitude scale
leaves its expansion around the map's middle."""
import numpy as np
import pytest

from glint_pipeline_gb300 import Configuration, DeviceBench
from glint_pipeline_gb300.tracegen import TraceGenerator
from oracle.bindings import Oracle, make_config
from test_gpu_parity import compare_meetings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision_mode", [0, 1])
@pytest.mark.parametrize("capacity,amplify,extent,sigma,chunk", [
    (1, 2.0, 2000.0, 60.0, 0),        # leaves of one and two members
    (16, 2.0, 2000.0, 60.0, 1),       # up to 32, one check per work item
    (33, 1.0, 2000.0, 60.0, 33),      # up to 33, full buffers drop objects
    (64, 1.0, 3000.0, 120.0, 64),
    (600, 2.0, 4000.0, 200.0, 500),   # hundreds of members
    (50, 2.0, 200000.0, 40.0, 0),     # a map 200 km wide: coarse offsets in sparse leaves
    (50, 2.0, 4000000.0, 40.0, 0),    # 4000 km: beyond the expansion of the longitude scale
])
def test_refine_matches_oracle(capacity, amplify, extent, sigma, chunk, precision_mode):
    n, steps = 4001, 12
    gen = TraceGenerator(0x5EED + capacity, n, 0, extent_m=extent, n_hotspots=3, sigma_m=sigma, hotspot_frac=0.9)
    box, pts = gen.box(), gen.steps(steps)
    args = dict(num_objects=n, num_meeting_buckets=1 << 20, grid_capacity=capacity, grid_amplify=amplify)
    o = Oracle(make_config(**args), box, pts[0])
    g = DeviceBench(Configuration(precision_mode=precision_mode, refine_chunk=chunk, **args), box, pts[0])
    contacts = total = 0
    for t in range(steps):
        o.step(pts[t], t)
        st = g.step(pts[t], t)
        c = o.counts()
        assert (st.checks, st.candidates, st.contacts) == (c.grid_check_counter, c.candidates, c.contacts), f"step {t}"
        assert (st.num_taken_buckets, st.num_active_meetings) == (c.num_taken_buckets, c.num_active_meetings)
        assert st.ambiguous == 0
        m = g.meetings()
        compare_meetings(o.meetings(), m, t)
        contacts += int(st.contacts)
        total += len(m)
    assert contacts > 0 and total > 0
    g.close()
    o.close()


@pytest.mark.parametrize("precision_mode", [0, 1])
@pytest.mark.parametrize("n,chunk", [(40, 0), (2000, 0), (6000, 0), (10000, 0), (16000, 0), (40000, 0),
                                     (2000, 1), (6000, 2)])
def test_items_by_number_and_by_cursor(n, chunk, precision_mode):
    """Work items from a handful to several times the warps of a launch: four,
    two and one warps an item, and items taken from the cursor.  About four
    members a leaf, so that n / 4 leaves and their extra chunks cross 1216, 2432
    and 4864."""
    gen = TraceGenerator(0xA11 + n, n, 0, extent_m=6.0 * n ** 0.5, n_hotspots=5, sigma_m=1.2 * n ** 0.5, hotspot_frac=0.5)
    box, pts = gen.box(), gen.steps(4)
    args = dict(num_objects=n, num_meeting_buckets=1 << 20, grid_capacity=6, grid_amplify=2.0)
    o = Oracle(make_config(**args), box, pts[0])
    g = DeviceBench(Configuration(precision_mode=precision_mode, refine_chunk=chunk, **args), box, pts[0])
    for t in range(4):
        o.step(pts[t], t)
        st = g.step(pts[t], t)
        c = o.counts()
        assert (st.checks, st.candidates, st.contacts) == (c.grid_check_counter, c.candidates, c.contacts), f"step {t}"
        compare_meetings(o.meetings(), g.meetings(), t)
    assert n < 1000 or int(st.contacts) > 0
    g.close()
    o.close()
