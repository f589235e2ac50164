"""Workloads of the co-occurrence pipeline, from single small steps to the 10M-object stream.

A case is a dict of plain values. Its "kind" says which public calls it makes:

  step            plain steps (stc_step_device, or stc_step from host memory), one drain at the end
  window          one pipelined window (stc_step_window) of page-locked host input, meetings drained beside it
  lsm             ingest windows, each flushed into a block, then the blocks compacted into one
  count_queries   a batch of object and box queries over flushed blocks, counted (stc_query_batch)
  contact_queries a serving-size batch of object queries that return their contacts
  sort            the library's radix sort of 32-bit pairs (stc_sort_pairs_u32)

Positions are the seeded street walkers of the repository's benchmark. A stream of steps is made
once and walked forwards and backwards, so that objects never jump and a pass over one period
always finds the same work. A pass covers one whole period.
"""
import ctypes
import math

import numpy as np
import torch

from stcdb_gb300._lib import load_library
from stcdb_gb300.pipeline import QUERY_BOX, QUERY_DTYPE, QUERY_OBJECT, MEETING_DTYPE, Pipeline, StcConfig
from stcdb_gb300.tracegen import DeviceTraceGenerator, TraceConfig

BOX_M = 40000.0  # side of the default street grid, 200 x 200 streets


def _stream(kind, objects, *, hot=0, hot_frac=0.0, sigma_m=300.0, box_m=BOX_M, grid_n=200, reach=10.0, min_meet=5,
            grid_capacity=200, amplify=2.0, buckets=0, steps=8, **more):
    c = dict(kind=kind, objects=objects, hot=hot, hot_frac=hot_frac, sigma_m=sigma_m, box_m=box_m, grid_n=grid_n,
             reach=reach, min_meet=min_meet, grid_capacity=grid_capacity, amplify=amplify, steps=steps)
    c.update(more)
    c["buckets"] = buckets or max(4 * _live_pairs(c), 4 * objects)
    # meetings that end within one period, at most, per pair within reach
    c.setdefault("ends", 2.0 if min_meet <= 3 else 0.6)
    return c


def _live_pairs(c):
    """Pairs within reach in one step, about: the benchmark's workloads have 67M (10M objects spread
    over the streets, reach 10 m), 20M to 35M (1M objects, 70% in 1000 hotspots of 300 m, reach
    10 m) and 370M to 590M (1M objects, 90% in 200 hotspots of 150 m, reach 20 m), and pairs grow
    with the square of the objects."""
    n = float(c["objects"])
    spread = (1.0 - c["hot_frac"]) ** 2 * 0.54 * n * n * c["reach"] / (c["grid_n"] * c["box_m"])
    if not c["hot"]:
        return int(spread) + 1
    share = 7e-5 if c["hot"] >= 500 else 1.8e-4  # Zipf weights: fewer hotspots hold more each
    scale = (c["reach"] / 10.0) * (300.0 / c["sigma_m"]) * (1000.0 / max(c["hot"], 1) if c["hot"] < 100 else 1.0)
    return int(spread + (c["hot_frac"] * n) ** 2 * share * min(scale, 12.0)) + 1


def listed():
    return [
        # A small deployment, or a test run: 20k objects handed over from host memory second by
        # second. Launches and host work count.
        dict(_stream("step", 20_000, hot=20, hot_frac=0.7, sigma_m=150.0, box_m=3000.0, grid_n=16, min_meet=3,
                     grid_capacity=50, buckets=1 << 20, steps=10, host=True), name="step_20k_host"),
        # The CPU-runnable configuration: 100k objects uniform over the streets.
        dict(_stream("step", 100_000, buckets=800_000, steps=10), name="step_100k"),
        # A ragged mid-size city: odd object and slot counts, another reach and leaf capacity.
        dict(_stream("step", 700_001, reach=13.0, min_meet=4, grid_capacity=120, buckets=3_000_017, steps=8),
             name="step_700k_odd"),
        # The hotspot model at 1M objects: dense leaves, many contacts an object.
        dict(_stream("step", 1_000_000, hot=1000, hot_frac=0.7, amplify=8.0, buckets=1 << 28, steps=8),
             name="step_hotspot_1m"),
        # The headline stream: 10M objects, positions already on the device.
        dict(_stream("step", 10_000_000, buckets=1 << 28, steps=8), name="step_uniform_10m"),
        # Uneven ingest windows: a short window of a few hundred thousand objects, half of them in
        # hotspots, from page-locked host memory.
        dict(_stream("window", 300_007, hot=1000, hot_frac=0.5, reach=12.0, amplify=8.0, buckets=1 << 24, steps=10),
             name="window_300k"),
        # The same call at 3M objects: the host link carries 48 MB a step.
        dict(_stream("window", 3_000_000, buckets=1 << 26, steps=8), name="window_3m"),
        # Ingest with the memtable on, two blocks flushed and compacted; the merged block then
        # answers counting queries and a few contact look-ups.
        dict(_stream("lsm", 60_000, hot=20, hot_frac=0.7, sigma_m=150.0, box_m=4000.0, grid_n=20, min_meet=3,
                     amplify=8.0, buckets=1 << 23, steps=8, blocks=2, split=7),
             name="lsm_60k"),
        # The same on the stress model (90% of objects in 200 hotspots, reach 20 m, minimum meeting
        # 3): tens of millions of keys a block.
        dict(_stream("lsm", 300_000, hot=200, hot_frac=0.9, sigma_m=150.0, reach=20.0, min_meet=3, amplify=32.0,
                     buckets=1 << 28, steps=8, blocks=2, split=10, ends=1.0), name="lsm_stress_300k"),
        # An analyst's batch: object and box counts over several retained blocks.
        dict(_stream("count_queries", 200_000, hot=200, hot_frac=0.7, reach=15.0, min_meet=3, amplify=16.0,
                     buckets=1 << 24, steps=8, blocks=4, queries=2048), name="count_queries_2k"),
        # What a serving batch holds at 20,000 queries a second: a few dozen contact look-ups.
        dict(_stream("contact_queries", 200_000, hot=200, hot_frac=0.7, reach=15.0, min_meet=3, amplify=16.0,
                     buckets=1 << 24, steps=8, blocks=4, queries=32), name="contact_queries_32"),
        # The sort on its own, as the flush and the compaction run it: tens of millions of pairs.
        dict(kind="sort", n=40_000_000, bits=32, name="sort_40m"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "window", "lsm", "count_queries", "contact_queries", "sort"])
    if kind == "sort":
        return dict(kind="sort", n=_log(rng, 1000, 60_000_000) | 1, bits=rng.randint(9, 32))
    dense = rng.random() < 0.5 or kind in ("lsm", "count_queries", "contact_queries")
    reach = round(rng.uniform(5.0, 20.0), 1)
    more = dict(reach=reach, min_meet=rng.randint(2, 5), grid_capacity=rng.choice([50, 64, 100, 128, 200, 256]),
                steps=rng.choice([6, 8, 10]))
    if dense:
        hi = {"step": 900_000, "window": 600_000}.get(kind, 250_000)
        n = _log(rng, 10_000, hi) | 1
        hot = rng.choice([1000, 700, 500])
        more.update(hot=hot, hot_frac=round(rng.uniform(0.2, 0.7), 2), sigma_m=float(rng.randint(200, 400)),
                    amplify=16.0)
        if kind not in ("step", "window") or n < 60_000:
            # a district: the same crowd on fewer streets, so that there are meetings
            more.update(box_m=8000.0, grid_n=40, hot=20, sigma_m=150.0)
            n = min(n, 80_001)
    else:
        n = _log(rng, 10_000, 4_000_000 if kind == "step" else 2_000_000) | 1
        more.update(amplify=4.0)
    if kind == "step":
        more["host"] = rng.random() < 0.3 and n < 500_000
    elif kind == "lsm":
        more.update(blocks=rng.randint(2, 3), split=rng.randint(3, 10))
    elif kind == "count_queries":
        more.update(blocks=rng.randint(1, 5), queries=_log(rng, 16, 4000))
    elif kind == "contact_queries":
        more.update(blocks=rng.randint(1, 5), queries=_log(rng, 1, 64))
    c = _stream(kind, n, **more)
    c["buckets"] = int(max(3 * _live_pairs(c), 2 * n) * rng.uniform(1.0, 4.0)) | 1
    return c


# ---- what a program has before the call ---------------------------------------------------------


def _positions(case, seed):
    """One period of positions on the device, (steps, objects, 2) f64, and the map box."""
    n, period = case["objects"], case["steps"]
    forward = period // 2 + 1  # steps 0 .. forward - 1, then back to 1
    g = DeviceTraceGenerator(TraceConfig(num_objects=n, grid_n=case["grid_n"], box_m=case["box_m"],
                                         n_hotspots=case["hot"], hot_frac=case["hot_frac"], sigma_m=case["sigma_m"],
                                         seed=seed + 1))
    xy = torch.empty((period, n, 2), dtype=torch.float64, device="cuda")
    g.next_into(xy.data_ptr(), forward)
    box = g.map_box(100.0)
    g.close()
    for k in range(forward, period):
        xy[k] = xy[period - k]
    torch.cuda.synchronize()
    return xy, box


def _pinned_like(xy):
    host = torch.empty(xy.shape, dtype=xy.dtype, pin_memory=True)
    host.copy_(xy)
    return host


class _Stream:
    """A pipeline in the middle of its stream: the table holds the meetings of the steps so far."""

    def __init__(self, case, seed):
        self.case, self.period = case, case["steps"]
        kind, n = case["kind"], case["objects"]
        lsm = kind in ("lsm", "count_queries", "contact_queries")
        # room for the meetings that end in one period, two directed keys each
        rows = int(case["ends"] * _live_pairs(case)) + 8192
        cfg = StcConfig(num_objects=n, reach_distance=case["reach"], min_meet_time=case["min_meet"],
                        grid_capacity=case["grid_capacity"], grid_amplify=case["amplify"],
                        num_meeting_buckets=case["buckets"], emit_capacity=2 * rows,
                        kv_restriction=2 * rows if lsm else 0, kv_capacity=3 * rows if lsm else 0,
                        ctb_retain=case.get("blocks", 0) + 1)
        self.xy, box = _positions(case, seed)
        self.box = [float(v) for v in box]
        self.pipe = Pipeline(cfg, box, self.xy[0].cpu().numpy())
        self.meetings = torch.empty((rows, 8), dtype=torch.int32, pin_memory=True)
        self.out = self.meetings.numpy().view(MEETING_DTYPE).reshape(-1)
        self.table = None if lsm else torch.zeros((rows, 8), dtype=torch.int32, device="cuda")
        self.filled = 0
        self.t = 0
        for _ in range(2):  # two periods: every pair has been met and left once
            self.window()

    def window(self):
        """One period as a pipelined window of device positions; the meetings that ended in it."""
        got = self.pipe.step_window((self.xy.data_ptr(), self.period), self.t, out=self.out)
        self.t += self.period
        return got

    def answer(self, count):
        """The first `count` drained meetings in (end, pid_lo, pid_hi) order, as 32-bit words, in the
        stream's device table (its rows behind them are zero): the library's order within a step is
        unspecified, and a pair ends at most once a step."""
        m = self.meetings[:count].to("cuda", non_blocking=True)
        key = ((m[:, 3].long() - (self.t - self.period - 1)) << 48) | (m[:, 0].long() << 24) | m[:, 1].long()
        torch.index_select(m, 0, torch.argsort(key), out=self.table[:count])
        if self.filled > count:
            self.table[count:self.filled].zero_()
        self.filled = count
        return self.table


def _counters(pipe):
    s = pipe.stats()
    return np.array([s.leaves, s.schema_nodes, s.overflow_objects, s.checking_units, s.border_units, s.hits,
                     s.new_candidates, s.taken_buckets, s.splits, s.merges], dtype=np.int64)


class _Steps(_Stream):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        self.host = self.xy.cpu().numpy() if case["host_input"] else None

    def run(self):
        for k in range(self.period):
            if self.host is not None:
                self.pipe.step(self.host[k], self.t + k)
            else:
                self.pipe.step_device(self.xy[k].data_ptr(), self.t + k)
        self.t += self.period
        got = self.pipe.drain_some(self.out)
        return {"meetings": self.answer(len(got)), "counters": _counters(self.pipe)}


class _Window(_Stream):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        self.pinned = _pinned_like(self.xy)
        self.host = self.pinned.numpy()

    def run(self):
        got = self.pipe.step_window(self.host, self.t, out=self.out)
        self.t += self.period
        return {"meetings": self.answer(len(got)), "counters": _counters(self.pipe)}


def _queries(st, seed, count, boxes):
    """Object look-ups and, with `boxes`, 40% box counts of up to a twentieth of the map a side."""
    rng = np.random.default_rng(seed)
    q = np.zeros(count, QUERY_DTYPE)
    q["kind"] = QUERY_OBJECT
    q["pid"] = rng.integers(0, st.case["objects"], count)
    q["t_start"] = 0
    q["t_end"] = 0xFFFFFFFF
    if boxes:
        b = rng.random(count) < 0.4
        x0, y0, x1, y1 = st.box
        cx, cy = rng.uniform(x0, x1, count), rng.uniform(y0, y1, count)
        w, h = rng.uniform(0.001, 0.05, count) * (x1 - x0), rng.uniform(0.001, 0.05, count) * (y1 - y0)
        q["kind"][b] = QUERY_BOX
        q["box"][b] = np.stack([cx - w, cy - h, cx + w, cy + h], axis=1)[b]
        late = rng.random(count) < 0.5
        q["t_start"][late] = max(st.t - st.period, 0)
    return q


class _Contacts:
    """Contact look-ups and their answers: how many each query has, then the contacts in (query,
    target, end) order (the library's order within an answer is unspecified), 7 words each, in an
    array whose rows behind them are zero."""

    def __init__(self, st, seed, count):
        self.pipe = st.pipe
        self.queries = _queries(st, seed, count, False)
        self.rows = np.zeros((8192 + 2048 * count, 7), dtype=np.int64)
        self.filled = 0

    def run(self):
        per_query = self.pipe.query_batch(self.queries)
        lengths = np.array([len(r) for r in per_query], dtype=np.int64)
        rows = np.concatenate(per_query)
        at = np.repeat(np.arange(len(lengths), dtype=np.int64), lengths)
        order = np.argsort((at << 54) | (rows["target"].astype(np.int64) << 28) | rows["end"].astype(np.int64))
        self.rows[:len(rows)] = rows[order].view(np.int64).reshape(-1, 7)
        self.rows[len(rows):self.filled] = 0
        self.filled = len(rows)
        return {"lengths": lengths, "contacts": self.rows}


class _Lsm(_Stream):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        self.pipe.flush()
        self.queries = _queries(self, seed, 2048, True)
        self.contacts = _Contacts(self, seed, 128)

    def run(self):
        first = None
        for _ in range(self.case["blocks"]):
            self.window()
            self.pipe.flush()
            if first is None:
                first = self.pipe.ctb_info().index
        merged, _ = self.pipe.compact(first, self.case["blocks"], self.case["split"])
        info = self.pipe.block_info(merged)
        said = np.array([info.kv_count, info.ctf_kv_count, info.oversize_kv_count, info.key_bytes, info.sid_count],
                        dtype=np.int64)
        # over the merged block and the last pass's, which is still retained
        return {"info": said, "counts": self.pipe.query_counts(self.queries).astype(np.int64),
                **self.contacts.run()}


class _Queries(_Stream):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        self.pipe.flush()
        for _ in range(case["blocks"] - 1):
            self.window()
            self.pipe.flush()
        if case["kind"] == "count_queries":
            self.queries = _queries(self, seed, case["queries"], True)
        else:
            self.queries, self.contacts = None, _Contacts(self, seed, case["queries"])

    def run(self):
        if self.queries is None:
            return self.contacts.run()
        return self.pipe.query_counts(self.queries).astype(np.int64)


class _Sort:
    def __init__(self, case, seed):
        f = load_library("libstc").stc_sort_pairs_u32
        f.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_size_t, ctypes.c_uint32, ctypes.c_uint32]
        f.restype = ctypes.c_int
        self.f, self.n, self.bits = f, case["n"], case["bits"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.keys = torch.randint(-(1 << 31), 1 << 31, (self.n,), dtype=torch.int32, device="cuda", generator=g)
        self.values = torch.arange(self.n, dtype=torch.int32, device="cuda")
        self.keys_out, self.values_out = torch.empty_like(self.keys), torch.empty_like(self.values)

    def run(self):
        if self.f(self.keys.data_ptr(), self.values.data_ptr(), self.keys_out.data_ptr(), self.values_out.data_ptr(),
                  self.n, self.bits, 0) != 0:
            raise RuntimeError("stc_sort_pairs_u32 failed")
        return self.keys_out, self.values_out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        return _Sort(case, seed)
    if kind == "step":
        return _Steps(dict(case, host_input=bool(case.get("host"))), seed)
    if kind == "window":
        return _Window(case, seed)
    if kind == "lsm":
        return _Lsm(case, seed)
    return _Queries(case, seed)


def run(state):
    return state.run()


def work(case):
    if case["kind"] == "sort":
        return {"bytes": 16.0 * case["n"], "flops": 0.0}  # each pair read once and written once
    n, live = case["objects"], _live_pairs(case)
    if case["kind"] in ("count_queries", "contact_queries"):
        # each query's record, and a few hundred 14-byte keys and 56-byte answers for it
        return {"bytes": case["queries"] * (48.0 + 8.0 + 100.0 * (14.0 + 56.0)), "flops": 0.0}
    # a step reads its positions and reads and writes the 32-byte record of each pair within reach
    step = 16.0 * n + 64.0 * live
    total = step * case["steps"] * case.get("blocks", 1)
    if case["kind"] == "lsm":
        # about a tenth of the pairs end in a step: two 32-byte keys each, packed once in the
        # block's flush and once in the compaction
        total += case["steps"] * case["blocks"] * 0.1 * live * 2 * (32.0 + 3 * 14.0)
    # a distance test of each pair within reach
    return {"bytes": total, "flops": 8.0 * live * case["steps"] * case.get("blocks", 1)}


def exact(case, seed):
    """Every output is whole numbers and record bytes (object ids, step times, float boxes bit for
    bit, packed keys, counts), which stay equal; there is no rounding to hold against 64 bits."""
    return None
