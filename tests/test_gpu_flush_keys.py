"""The flush's sort keys, counted from the map's corner, where the corner is
unusual: maps at the western end of the longitudes (whose coordinates round down
to nothing), across zero in both axes, in the south, and a map far larger than
the objects' part of it; and oversize objects among them."""
import numpy as np
import pytest

from glint_pipeline_gb300 import Configuration, DeviceBench
from glint_pipeline_gb300.tracegen import TraceGenerator
from oracle.bindings import Store
from test_gpu_flush import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("corner,widen,dprob", [
    ((-180.0, -60.0), 0.0, 100.0),
    ((-0.02, -0.02), 0.0, 100.0),
    ((179.95, 40.0), 0.0, 2e-9),     # most objects over the area bound: the oversize part
    ((10.0, -33.0), 9.0, 100.0),     # 9 degrees of empty map on every side
])
def test_flush_matches_oracle_on_any_map(corner, widen, dprob):
    n, steps = 20_000, 24
    gen = TraceGenerator(0xF1, n, 0, extent_m=4000.0, n_hotspots=5, sigma_m=300.0)
    box, pts = gen.box(), gen.steps(steps)
    move = np.array(corner) - box[:2]
    pts = pts + move
    box = np.concatenate([box[:2] + move - widen, box[2:] + move + widen])
    pts = np.clip(pts, box[:2], box[2:])
    g = DeviceBench(Configuration(num_objects=n, num_meeting_buckets=1 << 18, precision_mode=1, kv_capacity=1 << 22,
                                  dProbFalse=dprob, min_meet_time=3), box, pts[0])
    st = Store(n, box, first_end_time_min=3, kv_capacity=1 << 22, dProbFalse=dprob, max_meet_time=4096)
    keys = 0
    for t in range(steps):
        g.step(pts[t], t)
        st.add_meetings(g.meetings())
        if t in (11, 23):
            info = g.flush()
            rc, oi = st.flush(t)
            assert rc == 0
            compare(g.store(), st.result(oi), oi, f"flush at {t}")
            keys += int(info.kv_count + info.oversize_kv_count)
    assert keys > 0
    g.close()
    st.close()
