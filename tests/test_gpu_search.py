"""The active search by object (short lists beside the table) and by bucket,
and the switch between them, against the oracle: a loaded table whose entries
sit far from their home slots, lists around the switch, more entries than one
block orders, repeated and unknown ids, and a resumed context."""
import numpy as np
import pytest

from glint_pipeline_gb300 import Configuration, DeviceBench
from glint_pipeline_gb300.tracegen import TraceGenerator
from oracle.bindings import Oracle, make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,extent,sigma,buckets,counts,steps", [
    (20_000, 4000.0, 500.0, 30_011, (1, 3, 14, 15, 16), 30),      # loaded: by object up to 15 ids
    (20_000, 4000.0, 500.0, 1 << 20, (1, 500, 524, 525), 16),     # either side of B / 2000
    (6_000, 2000.0, 25.0, 1 << 24, (2_048, 2_049), 14),           # more than 4096 entries: by bucket after all
    (5_000, 2000.0, 60.0, 1 << 22, (0, 1, 2_000), 14),            # full leaf buffers drop objects
])
def test_search_matches_oracle(tmp_path, n, extent, sigma, buckets, counts, steps):
    gen = TraceGenerator(0x5EA + n, n, 0, extent_m=extent, n_hotspots=4, sigma_m=sigma)
    box, pts = gen.box(), gen.steps(steps)
    args = dict(num_objects=n, num_meeting_buckets=buckets, min_meet_time=2)
    cfg = Configuration(precision_mode=1, **args)
    o, g = Oracle(make_config(**args), box, pts[0]), DeviceBench(cfg, box, pts[0])
    rng = np.random.default_rng(n)
    found = 0

    def check(bench, t):
        nonlocal found
        everyone = o.active_search(np.arange(n, dtype=np.uint32))
        for k in counts:
            # half of them objects with active meetings, with repeats and an unknown id
            pids = rng.choice(n, k, replace=False).astype(np.uint32)
            if len(everyone) and k > 1:
                pids[: k // 2] = rng.choice(everyone["pid"], k // 2)
                pids[-1] = n + 7
            want = o.active_search(pids)
            assert bench.active_search(pids).tobytes() == want.tobytes(), f"step {t}, {k} ids"
            assert bench.active_search(pids, cap=2).tobytes() == want[:2].tobytes()
            found += len(want)

    for t in range(steps):
        o.step(pts[t], t)
        g.step(pts[t], t)
        if t >= 4 and t % 3 == 1:
            check(g, t)
    assert found > (4 * 4096 if n == 6_000 else 0)
    path = str(tmp_path / "snap")
    g.snapshot(path)
    g.close()
    r = DeviceBench.resume(path, cfg)
    check(r, "resumed")
    r.close()
    o.close()
