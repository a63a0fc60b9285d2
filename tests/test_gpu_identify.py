"""Identify and the scans at the sizes where their tiles end: tables of one
bucket more or less than a whole number of tiles, on both sides of the small
table's shorter spans, and object counts around a scan tile's 4096; and both
ways of touching an entry, over enough steps for both parities."""
import numpy as np
import pytest

from glint_pipeline_gb300 import Configuration, DeviceBench
from glint_pipeline_gb300.tracegen import TraceGenerator
from oracle.bindings import Oracle, make_config
from test_gpu_parity import compare_meetings, compare_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,buckets", [
    (4095, 1024 * 12 - 1), (4096, 1024 * 12), (4097, 1024 * 12 + 1), (8193, 30011),
    (4000, (1 << 23) - 1), (4000, 1 << 23), (4000, (1 << 23) + 8193),
    (3000, 1 << 26), (3000, (1 << 26) + 1),  # touches by stamp, by tag
])
def test_identify_matches_oracle(n, buckets):
    steps = 14
    gen = TraceGenerator(0x1DE + n, n, 0, extent_m=2500.0, n_hotspots=4, sigma_m=150.0)
    box, pts = gen.box(), gen.steps(steps)
    args = dict(num_objects=n, num_meeting_buckets=buckets)
    o = Oracle(make_config(**args), box, pts[0])
    g = DeviceBench(Configuration(precision_mode=1, **args), box, pts[0])
    total = 0
    for t in range(steps):
        o.step(pts[t], t)
        st = g.step(pts[t], t)
        c = o.counts()
        assert (st.num_taken_buckets, st.num_active_meetings) == (c.num_taken_buckets, c.num_active_meetings)
        m = g.meetings()
        compare_meetings(o.meetings(), m, t)
        total += len(m)
    compare_state(o, g)
    assert total > 0
    g.close()
    o.close()
