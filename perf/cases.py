"""Measured cases: what a user of the framework has it do, through its public
entry points, from the smallest regions to the largest.

Every case is one of five kinds:

step     one pass advances a context by its timesteps and takes the meetings
         of each (the per-timestep contact tracing path)
batch    one pass advances many independent regions by one timestep
query    one pass answers contact-trace queries over kept store blocks
compact  one pass steps and flushes a few windows, merges their blocks and
         asks the merged store
search   one pass lists the active contacts of given objects

The trajectories are walks on a street grid: blocks of 100 m, speeds 0.5-2
m/s, a tenth of the objects standing, starts at Gaussian hotspots or uniform,
at the densities of the repository's own workloads.  A context moves forwards
and backwards through its prepared steps, so it can be stepped without end.
Every output is whole numbers: meeting and search records are returned as
their 32-bit words (ids, times and the bits of their f32 boxes), because the
path's results are exact.
"""
import math

import numpy as np
import torch

import glint_pipeline_gb300 as gp
from glint_pipeline_gb300.batch import Batch

BLOCK_M = 100.0
LON0, LAT0 = -87.9, 41.6
DEG_LAT = 360.0 / 40076000.0
DEG_LON = DEG_LAT / math.cos(math.radians(LAT0))


def listed():
    return [
        # a village on a graph-replayed step: latency and launches decide
        dict(name="village_2k_graph", kind="step", objects=2_000, extent_m=2000.0, screened=True, call="graph",
             buckets=1 << 17, spots=8, sigma_m=200.0, spot_frac=0.7),
        # the drop-in call on a dense small town: host points in, meetings
        # out, the reference's default of two buckets per object
        dict(name="town_20k_plain_host", kind="step", objects=20_000, extent_m=4000.0, screened=False, call="host",
             buckets=40_009, spots=8, sigma_m=500.0, spot_frac=0.7),
        # a county: 100k objects sparse over the 40 km box, the small workload
        # of the repository's plain form
        dict(name="county_100k_plain_host", kind="step", objects=100_000, extent_m=40000.0, screened=False,
             call="host", buckets=200_000, spots=8, sigma_m=500.0, spot_frac=0.7),
        # a city stepped from device-resident points, FP64 on every pair
        dict(name="city_1m_plain", kind="step", objects=1_000_003, extent_m=12649.0, screened=False, call="device",
             buckets=1 << 24, spots=8, sigma_m=500.0, spot_frac=0.7),
        # the same city as a live feed: pipelined from page-locked host memory
        dict(name="city_1m_pipe", kind="step", objects=1_000_003, extent_m=12649.0, screened=True, call="pipe",
             buckets=1 << 26, spots=8, sigma_m=500.0, spot_frac=0.7),
        # extreme skew: a fifth of the objects in five spots of 50 m
        dict(name="core_2m_skew", kind="step", objects=2_000_000, extent_m=40000.0, screened=True, call="device",
             buckets=1 << 28, spots=5, sigma_m=50.0, spot_frac=0.2),
        # a metropolis at full size: two timesteps and the flush of their
        # meetings into the store
        dict(name="metro_10m_flush", kind="step", objects=10_000_000, extent_m=40000.0, screened=True, call="device",
             buckets=1 << 30, spots=8, sigma_m=500.0, spot_frac=0.7, steps=2, flush=True),
        # sixteen regions of uneven population in one timestep graph
        dict(name="regions_16", kind="batch", regions=16, smallest=1_000, largest=400_000),
        # an outbreak team's question: everyone within two hops of 1000 cases
        dict(name="query_2hop_1k_seeds", kind="query", objects=3_000_000, extent_m=21909.0, blocks=16, count=1,
             seeds=1000, hops=2, windows=False, served=False),
        # a served mix: many small and large questions at once, with windows
        dict(name="served_mix_64", kind="query", objects=1_000_000, extent_m=12649.0, blocks=24, count=64, seeds=300,
             hops=3, windows=True, served=True),
        # three windows of a city, flushed, merged into one block and asked
        dict(name="compact_2m", kind="compact", objects=2_000_000, extent_m=17889.0, blocks=3, split=24),
        # who are these objects meeting right now
        dict(name="search_2m_256", kind="search", objects=2_000_000, extent_m=17889.0, buckets=1 << 27, pids=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "batch", "query", "compact", "search"])
    if kind == "step":
        n = _log(rng, 2_000, 1_200_000)
        dense = rng.random() < 0.7
        ext = 40000.0 * math.sqrt(n / 1e7) * rng.uniform(1.0, 1.6) if dense else rng.uniform(10000.0, 40000.0)
        c = dict(kind=kind, objects=n, extent_m=max(2000.0, round(ext, 1)), screened=rng.random() < 0.6,
                 call=rng.choice(["host", "device", "graph", "pipe"]), spots=rng.choice([5, 8]),
                 sigma_m=rng.choice([200.0, 500.0]), spot_frac=rng.choice([0.2, 0.7]))
        c["buckets"] = n * 64 + rng.randrange(1000) if rng.random() < 0.5 else 1 << (n * 50).bit_length()
        # a flush needs keys in every one of its 100 files
        if dense and rng.random() < 0.5 and n >= 500_000:
            c["steps"], c["flush"] = rng.randint(2, 4), True
        return c
    if kind == "batch":
        return dict(kind=kind, regions=rng.randint(3, 16), smallest=1_000, largest=_log(rng, 20_000, 400_000))
    if kind == "query":
        n = _log(rng, 100_000, 2_000_000)
        served = rng.random() < 0.5
        return dict(kind=kind, objects=n, extent_m=round(40000.0 * math.sqrt(n / 1e7), 1), blocks=rng.randint(2, 16),
                    count=_log(rng, 4, 96) if served else rng.randint(1, 4), seeds=_log(rng, 1, 1000),
                    hops=rng.randint(1, 3), windows=rng.random() < 0.5, served=served)
    if kind == "compact":
        n = _log(rng, 300_000, 2_000_000)
        return dict(kind=kind, objects=n, extent_m=round(40000.0 * math.sqrt(n / 1e7), 1), blocks=rng.randint(2, 3),
                    split=rng.randint(8, 24))
    n = _log(rng, 5_000, 1_000_000)
    return dict(kind="search", objects=n, extent_m=max(2000.0, round(40000.0 * math.sqrt(n / 1e7), 1)),
                buckets=64 * n + rng.randrange(1000), pids=_log(rng, 1, 4000))


# ---- trajectories ---------------------------------------------------------


def _walk(n, extent_m, steps, seed, spots=8, sigma_m=500.0, spot_frac=0.7):
    """(box, points[steps, n, 2] on the GPU): n objects walking the streets of
    a square of extent_m metres for `steps` seconds."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda")
    extent = max(2, int(extent_m // BLOCK_M)) * BLOCK_M
    centre = torch.rand((spots, 2), generator=g, **f64) * (0.8 * extent) + 0.1 * extent
    which = torch.randint(0, spots, (n,), generator=g, device="cuda")
    at = centre[which] + torch.randn((n, 2), generator=g, **f64) * sigma_m
    anywhere = torch.rand((n, 2), generator=g, **f64) * extent
    u = torch.rand((n, 4), generator=g, **f64)
    at = torch.where(u[:, :1] < spot_frac, at, anywhere).clamp_(0.0, extent)
    axis = (u[:, 1] < 0.5).long()                       # 0 moves along x, 1 along y
    p = torch.where(axis == 0, at[:, 0], at[:, 1])      # along the street
    q = torch.where(axis == 0, at[:, 1], at[:, 0])      # the street
    q = (q / BLOCK_M).round() * BLOCK_M
    d = torch.where(u[:, 2] < 0.5, 1.0, -1.0).to(torch.float64)
    v = torch.rand((n,), generator=g, **f64) * 1.5 + 0.5
    v = torch.where(u[:, 3] < 0.1, torch.zeros_like(v), v)
    del at, anywhere, u, which
    out = torch.empty((steps, n, 2), **f64)
    for t in range(steps):
        x = torch.where(axis == 0, p, q)
        y = torch.where(axis == 0, q, p)
        out[t, :, 0] = x * DEG_LON + LON0
        out[t, :, 1] = y * DEG_LAT + LAT0
        k = p / BLOCK_M
        nxt = torch.where(d > 0, k.floor() + 1.0, k.ceil() - 1.0) * BLOCK_M
        nxt = nxt.clamp(0.0, extent)
        gap = (nxt - p) * d
        turn = v >= gap
        rest = (v - gap).clamp_(min=0.0)
        go = torch.rand((n,), generator=g, **f64)
        flip = turn & (go < 0.5)                        # into the crossing street
        p2, q2 = torch.where(flip, q, nxt), torch.where(flip, nxt, q)
        nd = torch.where((go * 4.0).floor() % 2 == 0, 1.0, -1.0).to(torch.float64)
        nd = torch.where(p2 <= 0.0, torch.ones_like(nd), torch.where(p2 >= extent, -torch.ones_like(nd), nd))
        p = torch.where(turn, p2 + rest * nd, p + v * d)
        q = torch.where(turn, q2, q)
        d = torch.where(turn, nd, d)
        axis = torch.where(flip, 1 - axis, axis)
    box = [LON0, LAT0, LON0 + extent * DEG_LON, LAT0 + extent * DEG_LAT]
    return box, out


def _turn(k, steps):
    """forwards and backwards through 0 .. steps - 1"""
    k %= 2 * (steps - 1)
    return k if k < steps else 2 * (steps - 1) - k


# ---- outputs ---------------------------------------------------------------

COUNTS = ("checks", "border_objects", "cross_checks", "candidates", "contacts", "new_keys", "num_taken_buckets",
          "num_active_meetings", "meetings", "splits", "merges", "leaves", "nodes", "dropped_objects",
          "meeting_log_size", "kv_count", "flushed")


def _counts(st):
    return np.array([int(getattr(st, f)) for f in COUNTS], dtype=np.int64)


def _words(rec):
    """records as their 32-bit words"""
    return rec.view(np.int32).reshape(len(rec), rec.dtype.itemsize // 4)


def _records(n):
    """a page-locked buffer for a step's meetings; the program keeps it, so
    what lies past a step's own records is an earlier step's"""
    out = gp.pinned_empty((max(1024, n),), gp.MEETING_DTYPE)
    out.view(np.uint8)[:] = 0
    return out


# ---- step ------------------------------------------------------------------


def _config(case, **more):
    n = case["objects"]
    return gp.Configuration(num_objects=n, num_meeting_buckets=case["buckets"],
                            precision_mode=1 if case["screened"] else 0, auto_flush=True,
                            kv_restriction=1 << 26 if case.get("flush") else max(1 << 20, 8 * n), store_keep=1, **more)


def _prepare_step(case, seed):
    n, steps = case["objects"], 8 if case["objects"] > 2_000_000 else 24
    box, pts = _walk(n, case["extent_m"], steps, seed, case["spots"], case["sigma_m"], case["spot_frac"])
    first = pts[0].cpu().numpy()
    call = case["call"]
    bench = gp.DeviceBench(_config(case, use_graph=call == "graph"), box, first)
    s = dict(case=case, bench=bench, n_steps=steps, t=0, per_pass=case.get("steps", 1), call=call,
             out=[_records(n) for _ in range(case.get("steps", 1))])
    if call in ("host", "pipe"):
        s["host"] = gp.pinned_empty((steps, n, 2), np.float64)
        torch.from_numpy(s["host"]).copy_(pts)
    else:
        s["pts"] = pts
    if call == "graph":
        s["feed"] = torch.empty_like(pts[0])
        s["stream"] = torch.cuda.ExternalStream(bench.stream)
    torch.cuda.synchronize()
    if call == "pipe":
        s["pipe"] = gp.Pipe(bench)
        s["pipe"].submit(s["host"][0], 0)
        s["t"] = 1
    # past the first steps, where every contact is new and none can end
    for _ in range(9):
        _one_step(s)
    return s


def _one_step(s, j=0):
    """one timestep: its statistics, and its meetings into buffer j"""
    bench, t, call = s["bench"], s["t"], s["call"]
    s["t"] = t + 1
    k = _turn(t, s["n_steps"])
    if call == "pipe":
        # the next step's points go in while the last one's meetings come out
        s["pipe"].submit(s["host"][k], t)
        st, m = s["pipe"].result(t - 1)
        # the view lives as long as the pipe: the consumer takes a copy
        s["out"][0][: len(m)] = m
        return st
    if call == "host":
        st = bench.step(s["host"][k], t)
        bench.meetings(out=s["out"][j])
        return st
    if call == "graph":
        with torch.cuda.stream(s["stream"]):
            s["feed"].copy_(s["pts"][k], non_blocking=True)
        bench.step_device(s["feed"].data_ptr(), t)
    else:
        bench.step_device(s["pts"][k].data_ptr(), t)
    st = bench.sync()
    bench.meetings(out=s["out"][j])
    return st


def _run_step(s):
    got = []
    for j in range(s["per_pass"]):
        got += [_counts(_one_step(s, j)), _words(s["out"][j])]
    if s["case"].get("flush"):
        info = s["bench"].flush()
        got.append(np.array([info.kv_count, info.key_bytes, info.oversize_kv_count, info.sid_count,
                             info.oversize_oid_count, info.end_time_min], dtype=np.int64))
    return got


# ---- batch -----------------------------------------------------------------


def _prepare_batch(case, seed):
    R = case["regions"]
    lo, hi = math.log(case["smallest"]), math.log(case["largest"])
    pops = [int(math.exp(lo + (hi - lo) * (r + 0.37) / R)) for r in range(R)]
    cfgs, boxes, pts = [], [], []
    for r, n in enumerate(pops):
        ext = float(np.clip(40000.0 * math.sqrt(n / 1e7), 2000.0, 40000.0))
        box, p = _walk(n, ext, 16, seed * 64 + r)
        cfgs.append(gp.Configuration(num_objects=n, num_meeting_buckets=1 << (64 * n - 1).bit_length(),
                                     precision_mode=1, auto_flush=True, kv_restriction=max(1 << 20, 8 * n),
                                     store_keep=1))
        boxes.append(box)
        pts.append(p)
    batch = Batch(cfgs, boxes, [p[0].cpu().numpy() for p in pts])
    s = dict(case=case, batch=batch, pts=pts, feed=[torch.empty_like(p[0]) for p in pts], t=0,
             streams=[torch.cuda.ExternalStream(batch.stream(r)) for r in range(R)],
             out=[_records(n) for n in pops])
    torch.cuda.synchronize()
    for _ in range(9):
        _run_batch(s)
    return s


def _run_batch(s):
    batch, t = s["batch"], s["t"]
    s["t"] = t + 1
    k = _turn(t, 16)
    for f, p, st in zip(s["feed"], s["pts"], s["streams"]):
        with torch.cuda.stream(st):
            f.copy_(p[k], non_blocking=True)
    batch.step([f.data_ptr() for f in s["feed"]], t)
    stats = batch.sync()
    got = [np.stack([_counts(st) for st in stats])]
    for reg, out in zip(batch.regions, s["out"]):
        reg.meetings(out=out)
        got.append(_words(out))
    return got


# ---- a store of kept blocks --------------------------------------------------


def _store(case, seed, keep):
    """a context that has flushed case["blocks"] windows of eight steps after
    four first ones, and its points"""
    n, per = case["objects"], 8
    box, pts = _walk(n, case["extent_m"], 24, seed)
    cfg = gp.Configuration(num_objects=n, num_meeting_buckets=64 * n, precision_mode=1, store_keep=keep,
                           min_meet_time=2, kv_restriction=16 * n)
    bench = gp.DeviceBench(cfg, box, pts[0].cpu().numpy())
    torch.cuda.synchronize()
    for t in range(case["blocks"] * per + 4):
        bench.step_device(pts[_turn(t, 24)].data_ptr(), t)
        bench.sync()
        if t >= 4 and (t - 4) % per == per - 1:
            bench.flush()
    return bench, pts


def _prepare_query(case, seed):
    bench = _store(case, seed, case["blocks"])[0]
    rng = np.random.default_rng(seed)
    last = case["blocks"] * 8 + 4
    qs = []
    for i in range(case["count"]):
        n = case["seeds"] if case["count"] == 1 else int(math.exp(rng.uniform(0.0, math.log(max(2, case["seeds"])))))
        seeds = rng.choice(case["objects"], size=n, replace=False).astype(np.uint32)
        hops = case["hops"] if case["count"] == 1 else int(rng.integers(1, case["hops"] + 1))
        t0, t1 = (0, 0)
        if case["windows"]:
            w = int(rng.integers(4, last))
            t0 = int(rng.integers(0, max(1, last - w)))
            t1 = t0 + w
        qs.append((seeds, hops, t0, t1))
    s = dict(case=case, bench=bench, queries=qs, rows=np.zeros((len(qs), case["objects"]), dtype=np.int32))
    if case["served"]:
        s["server"] = gp.Server(bench, max_slots=32)
    return s


def _run_query(s):
    """the ids reached, hop after hop, in each query's row, and each hop's
    count (the keys that a late hop reads depend on where its scan stops: they
    are not returned)"""
    rows, sizes = s["rows"], np.zeros((len(s["queries"]), 8), dtype=np.int64)

    def take(i, hops):
        at = 0
        for h, ids in enumerate(hops):
            rows[i, at:at + len(ids)] = ids
            at += len(ids)
            sizes[i, h] = len(ids)

    if not s["case"]["served"]:
        for i, hops in enumerate(s["bench"].query(s["queries"])[0]):
            take(i, hops)
        return [rows, sizes]
    srv = s["server"]
    tickets = {srv.submit(*q): i for i, q in enumerate(s["queries"])}
    while tickets:
        srv.step()
        for t in list(tickets):
            r = srv.poll(t, cap=s["case"]["objects"])
            if r is not None:
                take(tickets.pop(t), r[0])
    return [rows, sizes]


def _prepare_compact(case, seed):
    bench, pts = _store(dict(case, blocks=0), seed, 2 * case["blocks"] + 2)
    rng = np.random.default_rng(seed)
    s = dict(case=case, bench=bench, pts=pts, t=4, rows=np.zeros((1, case["objects"]), dtype=np.int32),
             asked=[(rng.choice(case["objects"], size=500, replace=False).astype(np.uint32), 1, 0, 0)])
    _run_compact(s)
    return s


def _run_compact(s):
    bench, k = s["bench"], s["case"]["blocks"]
    for _ in range(k):
        for _ in range(4):
            bench.step_device(s["pts"][_turn(s["t"], 24)].data_ptr(), s["t"])
            bench.sync()
            s["t"] += 1
        bench.flush()
    info = bench.compact(bench.store_blocks() - k, k, s["case"]["split"])
    sizes = [int(info[x]) for x in ("CTF_count", "blocks", "kv_count", "key_bytes", "padding", "oversize_kv_count",
                                    "sid_count", "x_part", "y_part")]
    hit = bench.query(s["asked"])[0][0][0]
    s["rows"][0, :len(hit)] = hit
    return [np.array(sizes, dtype=np.int64), np.array([len(hit)]), s["rows"]]


# ---- active search -----------------------------------------------------------


def _prepare_search(case, seed):
    n = case["objects"]
    box, pts = _walk(n, case["extent_m"], 12, seed)
    cfg = gp.Configuration(num_objects=n, num_meeting_buckets=case["buckets"], precision_mode=1, auto_flush=True,
                           kv_restriction=max(1 << 20, 8 * n), store_keep=1)
    bench = gp.DeviceBench(cfg, box, pts[0].cpu().numpy())
    torch.cuda.synchronize()
    for t in range(12):
        bench.step_device(pts[t].data_ptr(), t)
        bench.sync()
    rng = np.random.default_rng(seed)
    pids = rng.choice(n, size=min(n, case["pids"]), replace=False).astype(np.uint32)
    return dict(case=case, bench=bench, pids=pids, found=np.zeros(256 * case["pids"] + 4096, gp.SEARCH_DTYPE))


def _run_search(s):
    got = s["bench"].active_search(s["pids"])
    n = min(len(got), len(s["found"]))
    s["found"][:n] = got[:n]
    return [np.array([len(got)]), _words(s["found"])]


# ---- the interface -------------------------------------------------------------

_PREPARE = dict(step=_prepare_step, batch=_prepare_batch, query=_prepare_query, compact=_prepare_compact,
                search=_prepare_search)
_RUN = dict(step=_run_step, batch=_run_batch, query=_run_query, compact=_run_compact, search=_run_search)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


def _contacts(n, extent_m, spots=8, sigma_m=500.0, spot_frac=0.7):
    """contacts per step, estimated: ten per unit of squared line density,
    summed over the spots (at most fifty for an object: leaf buffers are
    bounded) and the open area"""
    own = n * spot_frac / spots
    return spots * min(10.0 * (own / sigma_m) ** 2, 50.0 * own) + 10.0 * (n * (1.0 - spot_frac) / extent_m) ** 2


def work(case):
    """Bytes of one pass: a step reads 16 bytes of points per object, reads
    and writes the 32-byte record of every contact and writes a 32-byte record
    per meeting (about a thirtieth of the contacts); a flush reads and writes
    its keys and boxes; a query reads the keys (about 15 bytes) of what it
    reaches; a compaction pass is its steps, and the flush and merge of their
    keys; a search reads the
    stamp of every bucket and the record of every live meeting."""
    k = case["kind"]
    if k == "step":
        n = case["objects"]
        c = _contacts(n, case["extent_m"], case["spots"], case["sigma_m"], case["spot_frac"])
        one = 16.0 * n + 64.0 * c + 32.0 * c / 30
        steps = case.get("steps", 1)
        return {"bytes": steps * (one + (2 * 47.0 * c / 30 if case.get("flush") else 0.0)), "flops": 0}
    if k == "batch":
        lo, hi, R = math.log(case["smallest"]), math.log(case["largest"]), case["regions"]
        pops = [math.exp(lo + (hi - lo) * (r + 0.5) / R) for r in range(R)]
        return {"bytes": sum(16.0 * n + 65.0 * _contacts(n, max(2000.0, 40000.0 * math.sqrt(n / 1e7)))
                             for n in pops), "flops": 0}
    c = _contacts(case["objects"], case["extent_m"])
    if k in ("query", "compact"):
        if k == "compact":
            steps = 4 * case["blocks"]
            return {"bytes": steps * (16.0 * case["objects"] + 64.0 * c + 4 * 47.0 * c / 5), "flops": 0}
        keys = case["blocks"] * 8 * c / 5
        share = min(1.0, case["count"] * case["seeds"] * 20.0 ** (case["hops"] - 1) / case["objects"])
        return {"bytes": 15.0 * keys * share + 4.0 * case["objects"] * share, "flops": 0}
    return {"bytes": case["buckets"] + 32.0 * 1.35 * c, "flops": 0}


def exact(case, seed):
    """None: every output is whole numbers and bits, which stay equal."""
    return None
