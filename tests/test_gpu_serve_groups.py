"""More running queries than one scan's 32-bit sums can count the objects of:
the marks of 4400 slots of a million objects are listed by two scans, one after
the other, and every query's result is the one it has in a small batch."""
import numpy as np
import pytest

from glint_pipeline_gb300 import Configuration, DeviceBench, Server
from glint_pipeline_gb300.tracegen import TraceGenerator

pytestmark = pytest.mark.gpu


def test_slots_beyond_one_scan():
    n, slots, steps = 1_000_000, 4400, 8
    assert slots * n > 1 << 32
    gen = TraceGenerator(0x5CA, n, 0, extent_m=9000.0, n_hotspots=4, sigma_m=400.0)
    box, pts = gen.box(), gen.steps(steps)
    g = DeviceBench(Configuration(num_objects=n, num_meeting_buckets=1 << 26, precision_mode=1, min_meet_time=1,
                                  kv_capacity=1 << 25), box, pts[0])
    for t in range(steps):
        g.step(pts[t], t)
    assert g.flush().kv_count > 0
    rng = np.random.default_rng(11)
    queries = [(rng.choice(n, 3, replace=False).astype(np.uint32), 1 + i % 3, 0, 0) for i in range(slots)]
    want, _ = g.query(queries)
    srv = Server(g, max_slots=slots)
    assert srv.slots == slots
    tickets = [srv.submit(*q) for q in queries]
    for _ in range(3):
        srv.step()
    reached = 0
    for i, t in enumerate(tickets):
        got = srv.poll(t)
        assert got is not None
        for h in range(queries[i][1]):
            np.testing.assert_array_equal(got[0][h], want[i][h], err_msg=f"query {i} hop {h + 1}")
            reached += len(got[0][h])
    assert reached > slots
    srv.close()
    g.close()
