"""The schema update with more events in a step than one round of its block
handles (1024), splits and merges mixed, and the high-water marks that bound
its passes: schema, both free stacks and the leaf counts against the oracle."""
import pytest

from glint_pipeline_gb300 import Configuration, DeviceBench
from glint_pipeline_gb300.tracegen import TraceGenerator
from oracle.bindings import Oracle, make_config
from test_gpu_parity import compare_meetings, compare_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,capacity,delay", [(60_000, 2, 1), (60_000, 3, 2), (3_000, 40, 1)])
def test_schema_matches_oracle(n, capacity, delay):
    steps = 10
    gen = TraceGenerator(0x5C4E + capacity, n, 0, extent_m=6000.0, n_hotspots=6, sigma_m=400.0)
    box, pts = gen.box(), gen.steps(4 * steps)[::4]  # four seconds a step: more objects change leaves
    args = dict(num_objects=n, num_meeting_buckets=1 << 21, grid_capacity=capacity, schema_update_delay=delay)
    o = Oracle(make_config(**args), box, pts[0])
    g = DeviceBench(Configuration(precision_mode=1, **args), box, pts[0])
    most = 0
    for t in range(steps):
        o.step(pts[t], t)
        st = g.step(pts[t], t)
        compare_meetings(o.meetings(), g.meetings(), t)
        compare_state(o, g)
        if st.splits and st.merges:
            most = max(most, int(st.splits + st.merges))
    assert most > (1024 if capacity <= 3 else 0)
    g.close()
    o.close()
