"""The work that users of the engine have it do, as timed cases.

A case is one use of the operator API (select -> aggregate, hash join, probe
of a resident table, select -> join -> group-by, join -> sink, a batch of
queries, a burst of served requests), with its sizes and options.  Sizes are
those of the benchmark configurations where they name one (2^22-row select,
2^22-key / 2^26-row join, 2^24-key / 2^27-row pipeline over 4096 Zipf groups,
the batched mix's log-uniform sizes) and otherwise odd numbers between them.

  listed()             the cases
  draw(rng)            another case of the same ranges
  prepare(case, seed)  inputs on the GPU and the operators a program keeps
  run(state)           one pass and its outputs
  work(case)           the bytes and operations a pass cannot do without
  exact(case, seed)    the same outputs by plain torch in 64 bits
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "multigpu-vector_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

GROUP_ROW = np.dtype([("group", np.int32), ("pad", np.int32), ("sum", np.int64), ("count", np.int64)])
FILTERS = 1000  # filter columns are uniform in [0, 1000)


def listed():
    return [
        # A dashboard-sized column: open, one launch and the read-back are all there is.
        {"name": "select_small", "kind": "select", "rows": 10_007, "percent": 50, "offset": 0},
        # The select configuration: one 4 Mi-row buffer, half of the rows qualify.
        {"name": "select_buffer", "kind": "select", "rows": 1 << 22, "percent": 50, "offset": 0},
        # A lookup against a small dimension table, built and probed once.
        {"name": "join_small", "kind": "join", "build": 1_000, "probe": 4_099, "dups": False, "offset": 0},
        # A join on a key that repeats on the build side, over column slices that start at an odd row.
        {"name": "join_repeated_keys", "kind": "join", "build": 300_007, "probe": 2_000_003, "dups": True, "offset": 1},
        # Both sides of the join one 4 Mi-row buffer: the build is most of it.
        {"name": "join_buffer", "kind": "join", "build": 1 << 22, "probe": 1 << 22, "dups": False, "offset": 0},
        # The join configuration's probe side against its resident table.
        {"name": "probe_large", "kind": "probe", "build": 1 << 22, "probe": 1 << 26, "offset": 0},
        # One interactive query over a small fact table.
        {"name": "query_small", "kind": "query", "build": 2_011, "probe": 40_009, "percent": 30, "groups": 60,
         "radix_bits": 0, "hit": 90},
        # A median query of the batched mix's upper half, one at a time.
        {"name": "query_ordinary", "kind": "query", "build": 400_009, "probe": 5_000_011, "percent": 45, "groups": 5_003,
         "radix_bits": 0, "hit": 90},
        # The pipeline configuration: radix-partitioned build, 10 % of the probe rows qualify.
        {"name": "query_large", "kind": "query", "build": 1 << 24, "probe": 1 << 27, "percent": 10, "groups": 4096,
         "radix_bits": 8, "hit": 100},
        # A join whose matches are wanted themselves (row number, key, payload), on the GPU.
        {"name": "materialise", "kind": "materialise", "build": 1_000_003, "probe": 8_000_009},
        # The batched mix: queries of uneven sizes in one launch.
        {"name": "batch", "kind": "batch", "queries": 64, "mix": 4, "build_log2": 22, "probe_log2": 24, "groups_log2": 16},
        # A burst of requests over one resident table that differ in their filter bound.
        {"name": "serve_burst", "kind": "serve", "requests": 64, "build": 1 << 20, "probe": 1 << 24, "groups": 1000},
    ]


def draw(rng):
    def size(lo, hi):  # log-uniform, odd or even as it falls
        return int(round(2 ** rng.uniform(math.log2(lo), math.log2(hi))))

    kind = rng.choice(["select", "select", "join", "join", "probe", "query", "query", "query", "materialise", "batch",
                       "serve"])
    offset = rng.choice([0, 0, 0, 1, 3, 8])
    if kind == "select":
        return {"kind": kind, "rows": size(1 << 12, 1 << 27), "percent": rng.randint(1, 99), "offset": offset}
    if kind == "join":
        return {"kind": kind, "build": size(1 << 8, 1 << 22), "probe": size(1 << 10, 1 << 26),
                "dups": rng.random() < 0.25, "offset": offset}
    if kind == "probe":
        return {"kind": kind, "build": size(1 << 10, 1 << 22), "probe": size(1 << 16, 1 << 26), "offset": offset}
    if kind == "query":
        probe = size(1 << 12, 1 << 27)
        return {"kind": kind, "build": size(1 << 8, 1 << 24), "probe": probe,
                "percent": rng.randint(1, 90) if probe < 1 << 25 else rng.randint(1, 20),
                "groups": size(1 << 4, 1 << 16), "radix_bits": rng.choice([0, 0, 6, 8]), "hit": rng.choice([90, 100])}
    if kind == "materialise":
        return {"kind": kind, "build": size(1 << 10, 1 << 22), "probe": size(1 << 12, 1 << 24)}
    if kind == "batch":
        return {"kind": kind, "queries": rng.randint(4, 64), "mix": rng.randint(0, 1 << 20), "build_log2": 21,
                "probe_log2": 23, "groups_log2": rng.choice([10, 16])}
    return {"kind": kind, "requests": rng.randint(8, 64), "build": size(1 << 12, 1 << 20),
            "probe": size(1 << 16, 1 << 24), "groups": size(1 << 5, 1 << 10)}


# ---- inputs -----------------------------------------------------------------------

class _Columns:
    """Seeded int32 columns on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def uniform(self, n, lo, hi, offset=0):
        """n values in [lo, hi); with an offset, a slice that starts `offset` rows into its column."""
        c = torch.randint(lo, hi, (n + offset,), generator=self.g, device="cuda", dtype=torch.int32)
        return c[offset:]

    def build_keys(self, n, dups, offset=0):
        if dups:
            return self.uniform(n, 0, max(1, n // 2), offset)
        c = torch.empty(n + offset, dtype=torch.int32, device="cuda")
        c[offset:] = torch.randperm(n, generator=self.g, device="cuda", dtype=torch.int32)
        return c[offset:]

    def probe_keys(self, n, build, hit, offset=0):
        """`hit` percent uniform over [0, build), the others above it."""
        keys = self.uniform(n, 0, build, offset)
        if hit < 100:
            miss = torch.randint(0, 100, (n,), generator=self.g, device="cuda", dtype=torch.int8) >= hit
            keys[miss] = self.uniform(int(miss.sum()), build, (1 << 31) - 1)
        return keys

    def zipf(self, n, groups):
        """Zipf(1) group ids in [0, groups)."""
        w = 1.0 / torch.arange(1, groups + 1, device="cuda", dtype=torch.float64)
        cdf = torch.cumsum(w, 0)
        out = torch.empty(n, dtype=torch.int32, device="cuda")
        for lo in range(0, n, 1 << 24):
            m = min(n, lo + (1 << 24)) - lo
            u = torch.rand(m, generator=self.g, device="cuda", dtype=torch.float64) * cdf[-1]
            out[lo:lo + m] = torch.searchsorted(cdf, u, out_int32=True).clamp_(max=groups - 1)
        return out

    def query(self, build, probe, groups, hit, dups=False):
        """(build keys, [probe key, filter, group, value])."""
        return self.build_keys(build, dups), [self.probe_keys(probe, build, hit), self.uniform(probe, 0, FILTERS),
                                              self.zipf(probe, groups), self.uniform(probe, 0, 1 << 16)]


def _mix(case):
    """Sizes of a batch's queries, (build, probe, bound, groups): log-uniform as in the batched configuration, from
    2^10, 2^12 and 2^4 up to the case's largest; 1 % to 90 % of the probe rows qualify."""
    r = random.Random(case["mix"])

    def size(lo, hi):
        return int(2 ** r.uniform(lo, hi))

    return [(size(10, case["build_log2"]), size(12, case["probe_log2"]), r.randint(10, 900) - 1,
             size(4, case["groups_log2"])) for _ in range(case["queries"])]


def _bounds(case, seed):
    """Filter bounds of a burst's requests: 1 % to 20 % of the rows qualify."""
    r = random.Random(seed)
    return [r.randint(9, 199) for _ in range(case["requests"])]


def _inputs(case, seed):
    c = _Columns(seed)
    kind = case["kind"]
    if kind == "select":
        # the filter is uniform in [0, 2^31); the bound keeps `percent` of it
        return {"filter": c.uniform(case["rows"], 0, (1 << 31) - 1, case["offset"]),
                "value": c.uniform(case["rows"], 0, 1 << 20, case["offset"])}
    if kind in ("join", "probe"):
        off = case["offset"]
        return {"bk": c.build_keys(case["build"], case.get("dups", False), off),
                "bp": c.uniform(case["build"], 0, 1 << 20, off),
                "pk": c.probe_keys(case["probe"], case["build"], 90, off),
                "pp": c.uniform(case["probe"], 0, 1 << 20, off)}
    if kind == "query":
        bk, cols = c.query(case["build"], case["probe"], case["groups"], case["hit"])
        return {"bk": bk, "cols": cols}
    if kind == "materialise":
        return {"bk": c.build_keys(case["build"], False), "bp": c.uniform(case["build"], 0, 1 << 20),
                "pk": c.probe_keys(case["probe"], case["build"], 90),
                "row": torch.arange(case["probe"], dtype=torch.int32, device="cuda")}
    if kind == "batch":
        return {"queries": [c.query(nb, npr, g, 90) for nb, npr, _, g in _mix(case)]}
    bk, cols = c.query(case["build"], case["probe"], case["groups"], 90)
    return {"bk": bk, "cols": cols, "bounds": _bounds(case, seed)}


def _select_bound(case):
    return (1 << 31) * case["percent"] // 100 - 1


def _query_bound(case):
    return FILTERS * case["percent"] // 100 - 1


# ---- one pass ---------------------------------------------------------------------

_context = None


def _ctx():
    global _context
    import mgv

    if _context is None:
        _context = mgv.Context(torch.cuda.current_device())
    return _context


class _State:
    """Inputs, operators and what a program keeps with them; the operators go with it."""

    def __init__(self, case, inputs):
        self.kind = case["kind"]
        self.case = case
        self.x = inputs
        self.owned = []

    def own(self, *objects):
        self.owned.extend(objects)

    def __del__(self):
        for o in self.owned:
            try:
                o.destroy()
            except Exception:  # interpreter shutdown
                pass


def prepare(case, seed):
    import mgv

    ctx = _ctx()
    s = _State(case, _inputs(case, seed))
    x = s.x
    if s.kind == "select":
        s.head, s.agg = mgv.create_sum_select_pipeline(ctx, _select_bound(case), 0, 1)
        s.own(s.head, s.agg)
    elif s.kind in ("join", "probe"):
        _, s.build, s.head, s.agg = mgv.create_count_join_1G_pipeline(ctx, case["build"])
        s.own(s.head, s.agg, s.build)
        if s.kind == "probe":
            _build(s.build, [x["bk"], x["bp"]], case["build"])
    elif s.kind == "query":
        s.bhead, s.build, s.head, s.groupby = mgv.create_join_groupby_pipeline(
            ctx, case["build"], case["groups"], _query_bound(case), case["radix_bits"])
        s.own(s.head, s.head.parent, s.groupby, s.bhead)
        if s.bhead is not s.build:
            s.own(s.build)
        s.rows = np.zeros(case["groups"], dtype=GROUP_ROW)
    elif s.kind == "materialise":
        rows = mgv.DEFAULT_BUFFER_ROWS
        s.pool = mgv.Pool(ctx, -(-case["probe"] // rows) + 1, rows, 3)
        s.sink = mgv.Op.sink(ctx, s.pool)
        s.build = mgv.Op.hash_build(ctx, 0, 1, case["build"])
        s.head = mgv.Op.hash_probe(ctx, 0, s.build, s.sink)
        s.out = [torch.empty(case["probe"], dtype=torch.int32, device="cuda") for _ in range(3)]
        s.own(s.head, s.sink, s.build, s.pool)
        _build(s.build, [x["bk"], x["bp"]], case["build"])
    elif s.kind == "batch":
        descs = [mgv.query_desc(bk, nb, *cols, npr, bound, g)
                 for (bk, cols), (nb, npr, bound, g) in zip(x["queries"], _mix(case))]
        s.batch = mgv.Batch(ctx, descs)
        s.max_groups = [g for _, _, _, g in _mix(case)]
        s.rows = np.zeros(sum(s.max_groups), dtype=GROUP_ROW)
        s.own(s.batch)
    else:
        s.server = mgv.Server(ctx, 40 << 30)
        s.own(s.server)
        s.table = s.server.add_table(x["bk"], case["build"])
        s.rows = np.empty((case["requests"], case["groups"]), dtype=GROUP_ROW)
    torch.cuda.synchronize()  # a server's streams do not wait for the default stream
    return s


def _build(op, cols, rows):
    op.open()
    op.consume_columns(cols, rows)
    op.close()


def _push(head, cols, rows):
    head.open()
    head.consume_columns(cols, rows)
    head.close()


def _groups(op, rows):
    """A closed group-by's rows into the program's result buffer, in group order; unused rows are zero."""
    import mgv

    used = ctypes.c_size_t()
    mgv.check(mgv.load().mgv_op_result(op.h, rows.ctypes.data, rows.nbytes, ctypes.byref(used)), "mgv_op_result")
    rows[used.value // GROUP_ROW.itemsize:] = 0
    return rows.view(np.int64).reshape(-1, 3)


def run(s):
    x, case = s.x, s.case
    if s.kind == "select":
        _push(s.head, [x["filter"], x["value"]], case["rows"])
        return s.agg.result()
    if s.kind == "join":
        _build(s.build, [x["bk"], x["bp"]], case["build"])
        _push(s.head, [x["pk"], x["pp"]], case["probe"])
        return s.agg.result()
    if s.kind == "probe":
        _push(s.head, [x["pk"], x["pp"]], case["probe"])
        return s.agg.result()
    if s.kind == "query":
        _push(s.bhead, [x["bk"]], case["build"])
        _push(s.head, x["cols"], case["probe"])
        return _groups(s.groupby, s.rows)
    if s.kind == "materialise":
        _push(s.head, [x["pk"], x["row"]], case["probe"])
        n = s.sink.result()
        for c, out in enumerate(s.out):
            s.sink.sink_read(c, out.data_ptr(), n)
        # the matches come in no order: a program that wants them per probe row puts them there by row number
        key, row, pay = (o[:n] for o in s.out)
        row = row.long()
        keys = torch.full((case["probe"],), -1, dtype=torch.int32, device="cuda")
        pays = torch.full((case["probe"],), -1, dtype=torch.int32, device="cuda")
        return n, keys.index_copy_(0, row, key), pays.index_copy_(0, row, pay)
    if s.kind == "batch":
        return _run_batch(s)
    return _run_burst(s)


def _run_batch(s):
    import mgv

    s.batch.run()
    lib, n, slot = mgv.load(), ctypes.c_uint64(), 0
    counts = np.empty(len(s.max_groups), dtype=np.int64)
    for q, most in enumerate(s.max_groups):  # every query's rows into its part of one result buffer
        mgv.check(lib.mgv_batch_result(s.batch.h, q, 0, s.rows.ctypes.data + GROUP_ROW.itemsize * slot, most,
                                       ctypes.byref(n)), "mgv_batch_result")
        s.rows[slot + n.value:slot + most] = 0
        counts[q] = n.value
        slot += most
    return counts, s.rows.view(np.int64).reshape(-1, 3)


def _run_burst(s):
    """All requests submitted at once, then waited for; groups come back unordered and are put in their places."""
    import mgv

    case, x = s.case, s.x
    tickets = [s.server.submit(s.table, *x["cols"], case["probe"], b, case["groups"]) for b in x["bounds"]]
    lib, n, lat = mgv.load(), ctypes.c_uint64(), ctypes.c_double()
    sums = np.zeros((case["requests"], case["groups"]), dtype=np.int64)
    counts = np.zeros((case["requests"], case["groups"]), dtype=np.int64)
    for i, ticket in enumerate(tickets):
        rows = s.rows[i]
        mgv.check(lib.mgv_server_wait(s.server.h, ticket, 60000, rows.ctypes.data, len(rows), ctypes.byref(n),
                                      ctypes.byref(lat)), "mgv_server_wait")
        got = rows[:n.value]
        sums[i, got["group"]] = got["sum"]
        counts[i, got["group"]] = got["count"]
    return sums, counts


# ---- floors and values --------------------------------------------------------------

def work(case):
    """Every input column read once and every result written once; comparisons, hashes and adds as operations."""
    kind = case["kind"]
    if kind == "select":
        return {"bytes": 8 * case["rows"] + 16, "flops": 2 * case["rows"]}
    if kind == "join":
        return {"bytes": 8 * case["build"] + 8 * case["probe"] + 16, "flops": 4 * (case["build"] + case["probe"])}
    if kind == "probe":
        return {"bytes": 8 * case["build"] + 8 * case["probe"] + 16, "flops": 4 * case["probe"]}
    if kind == "query":
        return _query_work(case["build"], case["probe"], case["groups"])
    if kind == "materialise":
        return {"bytes": 8 * case["build"] + 16 * case["probe"], "flops": 4 * case["probe"]}
    if kind == "batch":
        each = [_query_work(nb, npr, g) for nb, npr, _, g in _mix(case)]
        return {"bytes": sum(w["bytes"] for w in each), "flops": sum(w["flops"] for w in each)}
    return {"bytes": 4 * case["build"] + 16 * case["probe"] + 20 * case["requests"] * case["groups"],
            "flops": 6 * case["probe"]}


def _query_work(build, probe, groups):
    return {"bytes": 4 * build + 16 * probe + 20 * groups, "flops": 4 * build + 6 * probe}


def exact(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "select":
        keep = x["filter"] <= _select_bound(case)
        return int(keep.sum()), int(x["value"][keep].sum(dtype=torch.int64))
    if kind in ("join", "probe"):
        hit, key = _hits(x["pk"], case["build"])
        n = torch.bincount(x["bk"], minlength=case["build"])
        pay = torch.zeros(case["build"], dtype=torch.int64, device="cuda")
        pay.index_add_(0, x["bk"].long(), x["bp"].long())
        m = n[key]
        return int(m.sum()), int((pay[key] + m * x["pp"][hit]).sum())
    if kind == "query":
        return _result_rows(*_query_groups(x["bk"], x["cols"], _query_bound(case), case["groups"]))
    if kind == "materialise":
        hit, key = _hits(x["pk"], case["build"])
        pay = torch.empty(case["build"], dtype=torch.int32, device="cuda")
        pay[x["bk"].long()] = x["bp"]
        keys = torch.where(hit, x["pk"], -1)
        pays = torch.full_like(keys, -1)
        pays[hit] = pay[key]
        return int(hit.sum()), keys, pays
    if kind == "batch":
        each = [_query_groups(bk, cols, bound, g) for (bk, cols), (_, _, bound, g) in zip(x["queries"], _mix(case))]
        return (np.array([np.count_nonzero(c) for _, c in each]),
                np.concatenate([_result_rows(s, c) for s, c in each]))
    each = [_query_groups(x["bk"], x["cols"], b, case["groups"]) for b in x["bounds"]]
    return np.stack([s for s, _ in each]), np.stack([c for _, c in each])


def _hits(pk, build):
    hit = pk < build
    return hit, pk[hit].long()


def _query_groups(bk, cols, bound, groups):
    """SUM(value) and COUNT of every group of select(filter <= bound) -> join -> group-by."""
    key, filt, group, value = cols
    n = torch.bincount(bk, minlength=len(bk))
    keep = (filt <= bound) & (key < len(bk))
    m = n[key[keep].long()]
    g = group[keep].long()
    count = torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, g, m)
    total = torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, g, m * value[keep])
    return total.cpu().numpy(), count.cpu().numpy()


def _result_rows(sums, counts):
    """The groups found, {group, sum, count} in group order, in a buffer of one row per possible group."""
    g = np.flatnonzero(counts)
    rows = np.zeros((len(counts), 3), dtype=np.int64)
    rows[:len(g)] = np.stack([g, sums[g], counts[g]], axis=1)
    return rows
