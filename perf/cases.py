"""Performance cases of the hash GROUP BY / hash join engine, as its users call it.

Every pass is a whole query through the public Python binding of the C ABI
(query-engine_gb300/qeg): an operator is created, fed its columns, finished and
its result fetched. GROUP BY results have no defined row order, so each pass
ends with the ORDER BY key that a program wanting a stable answer runs on it
(numpy on host results, torch on device results), into result buffers that the
program keeps: as long as the case's expected group count with some room, the
rows past the result's own stay zero. Tables are resident in HBM unless the
case says "host".
"""
import ctypes
import json
import math
import os
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(REPO, "query-engine_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(REPO, "query-engine_gb300"))

SESSION_NS = 23_400 * 10 ** 9  # one 6.5 h trading session
T0 = 1_700_000_000 * 10 ** 9
MINUTE_NS = 60 * 10 ** 9


def listed():
    return [
        # One 2048-row batch of a host operator tree (the reference's batch
        # size), nullable key and value: the smallest call, all latency.
        {"name": "groupby_host_2k", "kind": "groupby", "rows": 2048, "groups": 64, "dist": "uniform", "s": 0.0,
         "keys": 1, "set": "f64", "nulls": True, "host": True},
        # The plain aggregate: 1M rows over 1,024 int64 keys, nullable F64.
        {"name": "groupby_1m", "kind": "groupby", "rows": 1 << 20, "groups": 1024, "dist": "uniform", "s": 0.0,
         "keys": 1, "set": "f64", "nulls": True, "host": False},
        # Skewed ids (clicks per user): Zipf(1.1) over 64M int64 keys.
        {"name": "groupby_zipf_256m", "kind": "groupby", "rows": 256 << 20, "groups": 64 << 20, "dist": "zipf",
         "s": 1.1, "keys": 1, "set": "int_f64", "nulls": False, "host": False},
        # Near-unique ids without a heavy head (orders per customer).
        {"name": "groupby_uniform_48m", "kind": "groupby", "rows": 48_000_000, "groups": 10_000_000,
         "dist": "uniform", "s": 0.0, "keys": 1, "set": "f64", "nulls": False, "host": False},
        # Composite key (store, product), ragged row count, nullable price.
        {"name": "groupby_two_keys_20m", "kind": "groupby", "rows": 20_000_003, "groups": 20_000, "dist": "zipf",
         "s": 0.9, "keys": 2, "set": "sales", "nulls": True, "host": False},
        # The headline join: COUNT/SUM over 256M probe rows, 16M dense unique
        # build keys, half of the probe rows match, 2% NULL keys.
        {"name": "join_sum_dense", "kind": "join_sum", "build": 16 << 20, "probe": 256 << 20, "keys": "dense",
         "dup": 1},
        # The same sink over sparse 64-bit ids: a hash table beyond L2.
        {"name": "join_sum_sparse", "kind": "join_sum", "build": 8 << 20, "probe": 128 << 20, "keys": "sparse",
         "dup": 1},
        # Fact table LEFT JOIN dimension, all columns materialised.
        {"name": "join_rows_left", "kind": "join_rows", "build": 2_000_000, "probe": 20_000_001, "keys": "sparse",
         "left": True, "host": False},
        # A dashboard refresh: 64 uneven GROUP BY queries in one batch.
        {"name": "batch_64q", "kind": "batch", "queries": 64, "max_rows": 10_000_000, "max_groups": 100_000},
        # One-minute bars of a day of trades.
        {"name": "window_50m", "kind": "window", "rows": 50_000_000, "symbols": 10_000, "minutes": 1},
        # The quote in force at every trade.
        {"name": "asof_20m", "kind": "asof", "trades": 20_000_000, "quotes": 5_000_000, "symbols": 10_000},
        # Fused filter -> join on symbol strings -> GROUP BY sector.
        {"name": "pipeline_200m", "kind": "pipeline", "rows": 200_000_000, "symbols": 10_000, "sectors": 32},
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | rng.choice((0, 1))

    kind = rng.choice(("groupby", "groupby", "groupby", "join_sum", "join_rows", "batch", "window", "asof",
                       "pipeline"))
    if kind == "groupby":
        host = rng.random() < 0.25
        rows = size(1000, 1 << 18) if host else size(1 << 14, 256 << 20)
        zipf = rng.random() < 0.5
        return {"kind": kind, "rows": rows, "groups": size(4, min(64 << 20, rows)),
                "dist": "zipf" if zipf else "uniform", "s": round(rng.uniform(0.5, 1.4), 2) if zipf else 0.0,
                "keys": 2 if rows <= 50_000_000 and rng.random() < 0.25 else 1,
                "set": rng.choice(("f64", "int_f64", "sales")), "nulls": rows <= 100_000_000 and rng.random() < 0.5,
                "host": host}
    if kind == "join_sum":
        build = size(1000, 16 << 20)
        return {"kind": kind, "build": build, "probe": size(max(build, 100_000), 256 << 20),
                "keys": rng.choice(("dense", "sparse")), "dup": rng.choice((1, 1, 4))}
    if kind == "join_rows":
        host = rng.random() < 0.25
        build = size(100, 100_000 if host else 4_000_000)
        return {"kind": kind, "build": build, "probe": size(2000, 500_000 if host else 40_000_000),
                "keys": rng.choice(("dense", "sparse", "two")), "left": rng.random() < 0.5, "host": host}
    if kind == "batch":
        return {"kind": kind, "queries": rng.randint(8, 96), "max_rows": size(20_000, 10_000_000),
                "max_groups": size(100, 100_000)}
    if kind == "window":
        return {"kind": kind, "rows": size(100_000, 100_000_000), "symbols": size(10, 10_000),
                "minutes": rng.choice((1, 1, 5, 30))}
    if kind == "asof":
        trades = size(100_000, 30_000_000)
        return {"kind": kind, "trades": trades, "quotes": size(20_000, 10_000_000), "symbols": size(10, 10_000)}
    return {"kind": kind, "rows": size(100_000, 200_000_000), "symbols": size(100, 10_000),
            "sectors": rng.randint(4, 64)}


# ---- inputs ------------------------------------------------------------------
def generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def zipf_ranks(n, domain, s, g):
    """n ranks in [0, domain) with Zipf(s) frequencies: an exact table for the
    first 2^18 ranks, the integral of x^-s beyond it."""
    head = min(domain, 1 << 18)
    cdf = np.cumsum(np.arange(1, head + 1, dtype=np.float64) ** -s)
    lo, hi = head + 0.5, domain + 0.5
    tail = (math.log(hi / lo) if s == 1.0 else (hi ** (1 - s) - lo ** (1 - s)) / (1 - s)) if domain > head else 0.0
    top = float(cdf[-1])
    table = torch.from_numpy(cdf).cuda()
    out = torch.empty(n, dtype=torch.int64, device="cuda")
    for a in range(0, n, 1 << 25):
        b = min(n, a + (1 << 25))
        u = torch.rand(b - a, generator=g, device="cuda", dtype=torch.float64).mul_(top + tail)
        r = torch.searchsorted(table, u).clamp_(max=head - 1)
        if tail:
            t = (u - top).clamp_(min=0)
            x = torch.exp(t).mul_(lo) if s == 1.0 else t.mul_(1 - s).add_(lo ** (1 - s)).pow_(1.0 / (1 - s))
            r = torch.where(u > top, x.sub_(0.5).long().clamp_(head, domain - 1), r)
        out[a:b] = r
    return out


def ranks(n, domain, dist, s, g):
    if dist == "zipf":
        return zipf_ranks(n, domain, s, g)
    return torch.randint(0, domain, (n,), generator=g, device="cuda", dtype=torch.int64)


def spread(r, bits):
    """Ids of ranks: an odd-multiplier bijection of [0, 2^bits)."""
    return r.mul(0x2545F4914F6CDD1D | 1).bitwise_and_((1 << bits) - 1)


def pack_bits(valid):
    """Validity words (64-bit, LSB first, padding bits set) of a boolean mask."""
    n = valid.numel()
    pad = (-n) % 64
    if pad:
        valid = torch.cat([valid, torch.ones(pad, dtype=torch.bool, device=valid.device)])
    b = valid.view(-1, 8).to(torch.uint8)
    w = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device=valid.device)
    return (b * w).sum(dim=1, dtype=torch.uint8).contiguous().view(torch.int64)


def unpack_bits(words, n):
    b = words.view(torch.uint8).unsqueeze(1) >> torch.arange(8, dtype=torch.uint8, device=words.device)
    return (b & 1).view(-1)[:n].bool()


def mask(n, share, g):
    return torch.rand(n, generator=g, device="cuda") >= share


_context = None


def context():
    """A program keeps one context for all its queries."""
    global _context
    if _context is None:
        import qeg

        _context = qeg.Context(0)
    return _context


def column(values, valid=None, type=None, code_map=None, host=False):
    import qeg

    words = None if valid is None else pack_bits(valid)
    if host:
        values = values.cpu().numpy()
        words = None if words is None else words.cpu().numpy().view(np.uint64)
    return qeg.Col(values, words, type, code_map)


def result_buffers(cols, rows):
    """Device buffers for a join's output columns: values and validity words."""
    return [(torch.zeros(rows, dtype=c.values.dtype, device="cuda"),
             torch.zeros((rows + 63) // 64, dtype=torch.int64, device="cuda")) for c in cols]


def key_bits(domain):
    return max(4, (domain - 1).bit_length() + 1)


def groupby_columns(case, seed):
    """(key tensors, value tensors, validity masks by column) of a GROUP BY."""
    g = generator(seed)
    n, dom = case["rows"], case["groups"]
    r = ranks(n, dom, case["dist"], case["s"], g)
    if case["keys"] == 2:  # (store I32, product I32): about a twentieth as many stores as products
        stores = max(2, int(math.sqrt(dom / 20.0)) + 1)
        keys = [(r % stores).to(torch.int32), spread(r.div(stores, rounding_mode="floor"), 24).to(torch.int32)]
    else:
        keys = [spread(r, key_bits(dom))]
    del r
    if case["set"] == "f64":
        vals = [torch.rand(n, generator=g, device="cuda", dtype=torch.float64).mul_(1000)]
    elif case["set"] == "int_f64":
        vals = [torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int64),
                torch.randn(n, generator=g, device="cuda", dtype=torch.float64).mul_(1e3)]
    else:  # sales: quantity I32, price F64
        vals = [torch.randint(1, 100, (n,), generator=g, device="cuda", dtype=torch.int32),
                torch.randn(n, generator=g, device="cuda", dtype=torch.float64).mul_(0.3).add_(3.0).exp_()]
    cols = keys + vals
    valid = [None] * len(cols)
    if case["nulls"]:
        valid[-1] = mask(n, 0.05, g)
        if case["host"] and case["keys"] == 1:
            valid[0] = mask(n, 0.02, g)
    return cols, valid


def groupby_aggs(case):
    import qeg

    k = case["keys"]
    if case["set"] == "f64":
        return [(qeg.COUNT_STAR, 0), (qeg.SUM, k), (qeg.AVG, k), (qeg.MIN, k), (qeg.MAX, k)]
    if case["set"] == "int_f64":
        return [(qeg.COUNT_STAR, 0), (qeg.SUM, k), (qeg.SUM, k + 1), (qeg.MIN, k), (qeg.MAX, k)]
    return [(qeg.COUNT_STAR, 0), (qeg.SUM, k), (qeg.AVG, k + 1), (qeg.MIN, k + 1), (qeg.MAX, k + 1),
            (qeg.COUNT, k + 1)]


def join_keys(case, seed):
    """Build and probe key tensors, masks and probe payload of a join: unique
    (or `dup` times repeated) build ids in random order, half of the probe ids
    among them."""
    g = generator(seed)
    nb, npr = case["build"], case["probe"]
    distinct = max(1, nb // case.get("dup", 1))
    bits = 48 if case["keys"] == "sparse" else 0
    b = torch.randperm(nb, generator=g, device="cuda", dtype=torch.int64).remainder_(distinct)
    p = torch.empty(npr, dtype=torch.int64, device="cuda")
    for a in range(0, npr, 1 << 26):
        z = min(npr, a + (1 << 26))
        p[a:z] = torch.randint(0, 2 * distinct, (z - a,), generator=g, device="cuda", dtype=torch.int64)
    if bits:
        b, p = spread(b, bits), spread(p, bits)
    return b, p, mask(nb, 0.02, g), mask(npr, 0.02, g), g


def ticks(rows, symbols, g):
    sym = zipf_ranks(rows, symbols, 1.0, g).to(torch.int32)
    step = SESSION_NS // rows
    ts = torch.arange(rows, device="cuda", dtype=torch.int64).mul_(step).add_(T0)
    ts += torch.randint(0, step, (rows,), generator=g, device="cuda")
    return sym, ts


def price(n, g):
    return torch.randn(n, generator=g, device="cuda", dtype=torch.float64).mul_(0.3).add_(4.6).exp_()


def batch_shape(case):
    """Row offsets and key domains: rows log-spaced over [1e3, max_rows], domains
    over [4, max_groups], paired at random; every other query is Zipf."""
    nq = case["queries"]
    at = (np.arange(nq) + 0.5) / nq
    sizes = np.exp(np.log(1e3) + at * (np.log(case["max_rows"]) - np.log(1e3))).astype(np.int64)
    doms = np.exp(np.log(4) + at * (np.log(case["max_groups"]) - np.log(4))).astype(np.int64)
    rng = np.random.RandomState(nq)
    sizes = rng.permutation(sizes)
    doms = rng.permutation(doms)
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64), doms, rng.uniform(0.5, 1.5, nq)


def batch_columns(case, seed):
    g = generator(seed)
    offs, doms, s = batch_shape(case)
    n = int(offs[-1])
    key = torch.empty(n, dtype=torch.int32, device="cuda")
    for q in range(case["queries"]):
        a, z = int(offs[q]), int(offs[q + 1])
        r = ranks(z - a, int(doms[q]), "zipf" if q & 1 else "uniform", float(s[q]), g)
        x = spread(r, 32)
        key[a:z] = torch.where(x >= (1 << 31), x - (1 << 32), x).to(torch.int32)
    return offs, key, torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def pipeline_columns(case, seed):
    g = generator(seed)
    n, ns = case["rows"], case["symbols"]
    tmap = torch.randperm(ns, generator=g, device="cuda").to(torch.int32)  # trades code -> value id
    bmap = torch.randperm(ns, generator=g, device="cuda").to(torch.int32)  # symbol-table code -> value id
    code_of = torch.argsort(tmap).to(torch.int32)
    sym = code_of[zipf_ranks(n, ns, 1.0, g)]
    return {"sym": sym, "price": price(n, g),
            "qty": torch.randint(1, 10001, (n,), generator=g, device="cuda", dtype=torch.int32),
            "tmap": tmap, "bmap": bmap, "bsym": torch.arange(ns, dtype=torch.int32, device="cuda"),
            "sector": torch.randint(0, case["sectors"], (ns,), generator=g, device="cuda", dtype=torch.int32)}


def prepare(case, seed):
    import qeg

    st = {"case": case, "ctx": context()}
    kind = case["kind"]
    if kind == "groupby":
        cols, valid = groupby_columns(case, seed)
        st["cols"] = [column(c, v, None, None, case["host"]) for c, v in zip(cols, valid)]
        st["aggs"] = groupby_aggs(case)
        st.update(room={}, rows=rooms(case))
    elif kind == "join_sum":
        b, p, bv, pv, g = join_keys(case, seed)
        val = torch.randint(0, 1 << 20, (case["probe"],), generator=g, device="cuda", dtype=torch.int64)
        st.update(build=column(b, bv), key=column(p, pv), val=column(val))
    elif kind == "join_rows":
        h = case["host"]
        b, p, bv, pv, g = join_keys(case, seed)
        bp = price(case["build"], g)
        bq = torch.randint(1, 10001, (case["build"],), generator=g, device="cuda", dtype=torch.int32)
        amount = torch.randint(0, 1 << 40, (case["probe"],), generator=g, device="cuda", dtype=torch.int64)
        bk, pk = [(b, bv)], [(p, pv)]
        if case["keys"] == "two":
            bk, pk = ([((t % 1009).to(torch.int32), v), (t.div(1009, rounding_mode="floor"), None)]
                      for t, v in ((b, bv), (p, pv)))
        st["probe"] = [column(t, v, host=h) for t, v in pk] + [column(amount, host=h)]
        st["build"] = [column(t, v, host=h) for t, v in bk] + [column(bp, host=h), column(bq, host=h)]
        st["on"] = list(range(len(pk)))
        if not h:
            st["bufs"] = result_buffers(st["probe"] + st["build"], case["probe"])
    elif kind == "batch":
        offs, key, val = batch_columns(case, seed)
        with open(os.path.join(REPO, "query-engine_gb300", "batch_tuning.json")) as f:
            tuned = json.load(f)
        torch.cuda.synchronize()
        st["aggs"] = [(qeg.COUNT_STAR, 0), (qeg.SUM, 1), (qeg.AVG, 1), (qeg.MIN, 1), (qeg.MAX, 1)]
        st["batch"] = qeg.Batch(st["ctx"], offs, qeg.Col(key), qeg.Col(val), st["aggs"],
                                tuning=[tuple(t) for t in tuned["tuning"]],
                                block_threads=int(tuned.get("block_threads", 0)))
        st.update(room={}, rows=rooms(case))
    elif kind == "window":
        g = generator(seed)
        sym, ts = ticks(case["rows"], case["symbols"], g)
        qty = torch.randint(1, 10001, (case["rows"],), generator=g, device="cuda", dtype=torch.int32)
        st["cols"] = [column(sym), column(ts, None, qeg.TS), column(price(case["rows"], g)), column(qty)]
        st.update(room={}, rows=rooms(case))
    elif kind == "asof":
        g = generator(seed)
        sym, ts = ticks(case["trades"], case["symbols"], g)
        qsym, qts = ticks(case["quotes"], case["symbols"], g)
        bid = price(case["quotes"], g)
        st["probe"] = [column(sym), column(ts, None, qeg.TS), column(price(case["trades"], g)),
                       column(torch.randint(1, 10001, (case["trades"],), generator=g, device="cuda",
                                            dtype=torch.int32))]
        st["build"] = [column(qsym), column(qts, None, qeg.TS), column(bid), column(bid + 0.01)]
        st["bufs"] = result_buffers(st["probe"] + st["build"], case["trades"])
    else:
        t = pipeline_columns(case, seed)
        st["probe"] = [column(t["sym"], None, qeg.STR, t["tmap"]), column(t["price"]), column(t["qty"])]
        st["build"] = [column(t["bsym"], None, qeg.STR, t["bmap"]), column(t["sector"])]
    torch.cuda.synchronize()  # the library reads the columns on its own stream
    return st


# ---- one pass ------------------------------------------------------------------
def kept(x, room):
    """A host column in a zeroed buffer of `room` rows."""
    y = np.zeros(max(room, len(x)), x.dtype)
    y[:len(x)] = x
    return y


def ordered_host(res, nkeys, room):
    """ORDER BY the key columns (NULLs first) of a result fetched to the host:
    the row count, then values and validity of each column in `room` rows."""
    by = []
    for v, ok in reversed(res[:nkeys]):
        by += [v, ok]
    order = np.lexsort(by)
    return [len(order)] + [kept(x[order], room) for v, ok in res for x in (v, ok)]


def ordered_device(st, cols, key):
    """ORDER BY `key` of a device result's columns, into the state's result
    buffers (allocated with the first result): the row count, then each column."""
    n, room = key.numel(), st["room"]
    order = torch.argsort(key)
    out = [n]
    for i, v in enumerate(cols):
        if i not in room or room[i].numel() < n:
            room[i] = torch.zeros(max(n, st["rows"]), dtype=v.dtype, device="cuda")
        out.append(room[i])
        torch.index_select(v, 0, order, out=room[i][:n])
    return out


def run(st):
    import qeg

    case, ctx, kind = st["case"], st["ctx"], st["case"]["kind"]
    if kind == "groupby":
        nk = case["keys"]
        if case["host"]:
            return ordered_host(qeg.groupby(ctx, st["cols"], list(range(nk)), st["aggs"], batch_rows=2048), nk,
                                st["rows"])
        a = qeg.Aggregate(ctx, [c.type for c in st["cols"]], list(range(nk)), st["aggs"])
        try:
            a.consume(st["cols"])
            a.finish()
            res = a.fetch_torch()
            key = res[0][0]
            if nk == 2:
                key = (key.long() << 34) + (res[1][0].long() + (1 << 33))
            cols = [v for v, _ in res]
            if case["nulls"]:  # the aggregates that a group of NULL values leaves NULL
                cols += [unpack_bits(res[c][1], key.numel()) for c in (nk + 2, nk + 3)]
            return ordered_device(st, cols, key)
        finally:
            a.close()
    if kind == "join_sum":
        j = qeg.Join(ctx, [qeg.I64, qeg.I64], [qeg.I64], [0], [0])
        try:
            j.build([st["build"]])
            j.build_finish()
            j.probe_count_sum(st["key"], st["val"])
            count, total = j.count_sum()
            return [count, 0 if total is None else total]
        finally:
            j.close()
    if kind in ("join_rows", "asof"):
        pt, bt = [c.type for c in st["probe"]], [c.type for c in st["build"]]
        if kind == "asof":
            j = qeg.AsofJoin(ctx, pt, bt, [0], [0], 1, 1, qeg.LEFT)
        else:
            j = qeg.Join(ctx, pt, bt, st["on"], st["on"], qeg.LEFT if case["left"] else qeg.INNER)
        try:
            j.build(st["build"])
            j.build_finish()
            n = j.probe(st["probe"])
            if case.get("host"):
                return [n] + [kept(x, case["probe"]) for v, ok in j.fetch(0, n) for x in (v, ok)]
            j.fetch_device(0, n, st["bufs"])
            return [n] + [x for v, w in st["bufs"] for x in (v, w)]
        finally:
            j.close()
    if kind == "batch":
        return run_batch(st)
    if kind == "window":
        w = qeg.Window(ctx, [c.type for c in st["cols"]], [0], 1, case["minutes"] * MINUTE_NS,
                       [(qeg.COUNT_STAR, 0), (qeg.SUM, 3), (qeg.MIN, 2), (qeg.MAX, 2), (qeg.AVG, 2)])
        try:
            w.consume(st["cols"])
            w.finish()
            res = w.fetch_torch()
        finally:
            w.close()
        return ordered_device(st, [v for v, _ in res], (res[0][0].long() << 48) + (res[1][0] - T0 + MINUTE_NS * 60))
    _, res = qeg.filter_join_agg(ctx, st["probe"], st["build"], 0, 0, 4,
                                 [(qeg.COUNT_STAR, 0), (qeg.AVG, 1), (qeg.SUM, 2)], filter_col=1,
                                 filter_op=qeg.CMP_GT, filter_value=100.0, capacity=case["sectors"])
    return ordered_host(res, 1, case["sectors"])


def run_batch(st):
    """Runs the batch and fetches every query's result into device tensors,
    ordered by (query, key)."""
    import qeg

    b = st["batch"]
    b.run()
    groups = b.finish().astype(np.int64)
    total = int(groups.sum())
    types = {qeg.I32: torch.int32, qeg.I64: torch.int64, qeg.F64: torch.float64}
    cols = [torch.empty(total, dtype=types[t], device="cuda") for t in b.result_types]
    torch.cuda.synchronize()  # the library writes them on its own stream
    outs = (qeg.OutColumn * len(cols))()
    at = 0
    for q, n in enumerate(groups.tolist()):
        for i, c in enumerate(cols):
            outs[i] = qeg.OutColumn(c.data_ptr() + at * c.element_size(), None, None)
        status = qeg.lib().qeg_batch_fetch(b.p, q, ctypes.byref(outs))
        if status != 0:
            raise qeg.QegError(status, "batch fetch")
        at += n
    counts = torch.from_numpy(groups).cuda()
    query = torch.repeat_interleave(torch.arange(len(groups), device="cuda"), counts, output_size=total)
    return [groups] + ordered_device(st, cols, (query << 32) + cols[0].long())


# ---- what a pass cannot do without ----------------------------------------------
def expected_groups(n, domain, dist, s):
    """Expected distinct values of n draws."""
    if dist != "zipf":
        return domain * -math.expm1(n * math.log1p(-1.0 / domain)) if domain > 1 else 1.0
    edge = np.unique(np.round(np.geomspace(1, domain + 1, 4000)).astype(np.int64))
    mid, width = np.sqrt(edge[:-1] * (edge[1:] - 1.0)), np.diff(edge).astype(np.float64)
    w = mid ** -s
    return float((width * -np.expm1(-n * w / (w * width).sum())).sum())


def result_rows(case):
    """Expected rows of a GROUP BY's result."""
    kind = case["kind"]
    if kind == "groupby":
        return expected_groups(case["rows"], case["groups"], case["dist"], case["s"])
    if kind == "batch":
        offs, doms, s = batch_shape(case)
        n = np.diff(offs.astype(np.int64))
        return sum(expected_groups(int(n[q]), int(doms[q]), "zipf" if q & 1 else "uniform", float(s[q]))
                   for q in range(len(n)))
    buckets = max(1, 390 // case["minutes"])
    return buckets * expected_groups(case["rows"] / buckets, case["symbols"], "zipf", 1.0)


def rooms(case):
    """Rows of the result buffers: the expected count and some room."""
    return int(1.05 * result_rows(case)) + 1000


def work(case):
    kind = case["kind"]
    bit = 1 / 8
    if kind == "groupby":
        n = case["rows"]
        row = {"f64": 8, "int_f64": 16, "sales": 12}[case["set"]] + 8 + (bit if case["nulls"] else 0)
        out = {"f64": 40, "int_f64": 40, "sales": 48}[case["set"]] + 8
        return {"bytes": n * row + out * result_rows(case), "flops": 0}
    if kind == "join_sum":
        return {"bytes": case["build"] * (8 + bit) + case["probe"] * (16 + bit), "flops": 0}
    if kind == "join_rows":
        key = 12 if case["keys"] == "two" else 8
        rows = case["probe"] * (1.0 if case["left"] else 0.49)
        return {"bytes": case["build"] * (key + 12 + bit) + case["probe"] * (key + 8 + bit) +
                rows * (2 * key + 20 + 6 * bit), "flops": 0}
    if kind == "batch":
        return {"bytes": float(batch_shape(case)[0][-1]) * 12 + 44 * result_rows(case), "flops": 0}
    if kind == "window":
        return {"bytes": case["rows"] * 24 + 44 * result_rows(case), "flops": 0}
    if kind == "asof":
        return {"bytes": case["quotes"] * 28 + case["trades"] * (24 + 52 + 1), "flops": 0}
    return {"bytes": case["rows"] * 16 + case["symbols"] * 8, "flops": 0}


# ---- the same answers in 64 bits, without the engine ------------------------------
def grouped(key, vals, valids):
    """Sorted distinct keys and, per value column, (count, sum, mean, min, max)
    over its valid rows in float64 (NaN-free inputs); a group without valid
    rows has zeros, as a fetched NULL has."""
    uniq, inv, rows = torch.unique(key, return_inverse=True, return_counts=True)
    stats = []
    for v, ok in zip(vals, valids):
        iv, x = (inv, v) if ok is None else (inv[ok], v[ok])
        cnt = rows if ok is None else torch.bincount(iv, minlength=uniq.numel())
        x = x.double()
        total = torch.zeros(uniq.numel(), dtype=torch.float64, device="cuda").index_add_(0, iv, x)
        lo = torch.full_like(total, math.inf).scatter_reduce_(0, iv, x, "amin")
        hi = torch.full_like(total, -math.inf).scatter_reduce_(0, iv, x, "amax")
        none = cnt == 0
        stats.append((cnt, total, total / cnt.clamp(min=1), lo.masked_fill_(none, 0), hi.masked_fill_(none, 0)))
    return uniq, rows, stats


def padded(v, room):
    return None if v is None else torch.cat([v, v.new_zeros(max(0, room - v.numel()))])


def exact(case, seed):
    kind = case["kind"]
    if kind == "groupby":
        cols, valid = groupby_columns(case, seed)
        nk = case["keys"]
        key = cols[0].long()
        if nk == 2:
            key = (key << 34) + (cols[1].long() + (1 << 33))
        if valid[0] is not None:  # NULL keys sort first, as one group
            key = torch.where(valid[0], key, torch.full_like(key, -1))
        _, _, stats = grouped(key, cols[nk:], valid[nk:])
        last = stats[-1]
        if case["set"] == "f64":
            vals = [None, last[1], last[2], last[3], last[4]]
        elif case["set"] == "int_f64":
            vals = [None, None, last[1], None, None]
        else:
            vals = [None, None, last[2], last[3], last[4], None]
        vals = [None] * nk + [padded(v, rooms(case)) for v in vals]
        return [None] + ([x for v in vals for x in (v, None)] if case["host"] else vals)
    if kind == "batch":
        offs, key, val = batch_columns(case, seed)
        sizes = torch.from_numpy(np.diff(offs.astype(np.int64))).cuda()
        query = torch.repeat_interleave(torch.arange(case["queries"], device="cuda"), sizes)
        st = grouped((query << 32) + key.long(), [val], [None])[2][0]
        return [None] * 4 + [padded(v, rooms(case)) for v in st[1:]]
    if kind == "window":
        g = generator(seed)
        sym, ts = ticks(case["rows"], case["symbols"], g)
        torch.randint(1, 10001, (case["rows"],), generator=g, device="cuda", dtype=torch.int32)
        width = case["minutes"] * MINUTE_NS
        start = ts.div(width, rounding_mode="trunc") * width
        st = grouped((sym.long() << 48) + (start - T0 + MINUTE_NS * 60), [price(case["rows"], g)], [None])[2][0]
        return [None] * 5 + [padded(st[i], rooms(case)) for i in (3, 4, 2)]
    if kind == "pipeline":
        t = pipeline_columns(case, seed)
        keep = t["price"] > 100
        sector = t["sector"][torch.argsort(t["bmap"])[t["tmap"][t["sym"].long()].long()]].long()[keep]
        st = grouped(sector, [t["price"][keep]], [None])[2][0]
        return [None] * 5 + [padded(st[2], case["sectors"])] + [None] * 3
    return None  # join results are whole numbers and copied columns
