"""Steps replayed from the captured graph: points at changing addresses, on
and off a 16-byte boundary, steps queued without waiting between them, host and
device points mixed, and key appends after a flush that was refused."""
import numpy as np
import pytest

from glint_pipeline_gb300 import Configuration, DeviceBench, GlintError
from glint_pipeline_gb300.tracegen import TraceGenerator
from oracle.bindings import Oracle, make_config
from test_gpu_parity import compare_meetings, compare_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [False, True])
def test_graph_steps_match_oracle(use_graph):
    torch = pytest.importorskip("torch")
    n, steps = 3001, 24
    gen = TraceGenerator(0x6A7, n, 0, extent_m=2000.0, n_hotspots=3, sigma_m=100.0)
    box, pts = gen.box(), gen.steps(steps)
    args = dict(num_objects=n, num_meeting_buckets=1 << 18)
    o = Oracle(make_config(**args), box, pts[0])
    g = DeviceBench(Configuration(precision_mode=1, use_graph=use_graph, **args), box, pts[0])
    # one buffer, each step's points at an address of its own; odd steps are
    # only 8-byte aligned
    room = torch.zeros(steps * (2 * n + 2), dtype=torch.float64, device="cuda")
    at = []
    for t in range(steps):
        first = t * (2 * n + 2) + (t & 1)
        room[first:first + 2 * n] = torch.from_numpy(pts[t].reshape(-1))
        at.append(room.data_ptr() + 8 * first)
    torch.cuda.synchronize()
    refused = total = 0
    for t in range(steps):
        o.step(pts[t], t)
        if t % 6 == 2:
            g.step(pts[t], t)             # host points
        else:
            g.step_device(at[t], t)
            if t % 6 == 3:                # the next step is queued behind it
                continue
            g.sync()
        compare_meetings(o.meetings(), g.meetings(), t)
        total += len(g.meetings())
        if t == 12:
            # a window of few keys leaves files without any: refused, and the
            # keys stay pending
            before = int(g.sync().kv_count)
            with pytest.raises(GlintError):
                g.flush()
            refused += 1
            assert before > 0
    compare_state(o, g)
    assert total > 0 and refused == 1
    g.close()
    o.close()
