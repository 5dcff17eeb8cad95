"""Performance cases of the priority queue: what programs that use it have it do.

Eight kinds of work, each through the package's public entry points:

* single   -- one insertion / deleteRoot / retrieve call at a time;
* sort     -- the plain heap-sort (reset, insert everything, delete everything);
* queue    -- a queue that is filled in bulk, gives up its smallest keys, is
              filled again, is drained below a threshold and then to the end;
* host     -- the heap-sort between pinned host buffers, copies included;
* fifo     -- the device FIFO buffer, pushed and popped in whole calls;
* sssp     -- single-source shortest paths on an R-MAT graph;
* searches -- many independent A* and knapsack searches in one launch;
* served   -- a burst of SSSP and A* queries through the device request loop.

Sizes are those of the package's tests, of its benchmark and of its autotuners:
batch sizes 128-2048, 2^12 to 2^28 keys, R-MAT scales 12-18, grids up to 512
cells a side.
"""
import math

import numpy as np
import torch

import gpuheap_gb300 as gh
from gpuheap_gb300 import batch as gb
from gpuheap_gb300 import serve as gsv
from gpuheap_gb300 import sssp as gs
from gpuheap_gb300.fifo import Fifo

KEY_BYTES = {"u32": 4, "i32": 4, "u64": 8}
UNREACHABLE = 0xFFFFFFFF
INF = 1 << 60


def listed():
    return [
        # An event queue used call by call: latency of one operation.
        {"name": "single_u32_b256", "kind": "single", "key": "u32", "variant": "bottomup", "batch_size": 256, "ops": 24},
        # A short list: launches and fixed costs.
        {"name": "sort_u32_5k", "kind": "sort", "key": "u32", "variant": "topdown", "partial_buffer": True,
         "batch_size": 256, "n": 5000, "dist": "uniform"},
        # The small configuration of the plain heap-sort.
        {"name": "sort_u32_1m", "kind": "sort", "key": "u32", "variant": "bottomup", "partial_buffer": True,
         "batch_size": 1024, "n": 1 << 20, "dist": "uniform"},
        # Small batches without the partial buffer, signed keys that come in the worst order.
        {"name": "sort_i32_2m_reverse", "kind": "sort", "key": "i32", "variant": "topdown", "partial_buffer": False,
         "batch_size": 256, "n": 1 << 21, "dist": "reverse"},
        # Key and payload packed in 64 bits, few distinct keys, a ragged size.
        {"name": "sort_u64_16m_zipf", "kind": "sort", "key": "u64", "variant": "topdown", "partial_buffer": True,
         "batch_size": 1024, "n": (1 << 24) + 333, "dist": "zipf"},
        # The benchmark's default line.
        {"name": "sort_u32_256m", "kind": "sort", "key": "u32", "variant": "bottomup", "partial_buffer": True,
         "batch_size": 2048, "n": 1 << 28, "dist": "uniform"},
        # A queue that is never simply drained: bulk inserts into a used heap, partial deletes, a threshold.
        {"name": "queue_u64_1m", "kind": "queue", "key": "u64", "variant": "bottomup", "partial_buffer": True,
         "batch_size": 512, "n": (1 << 20) + 77, "dist": "uniform"},
        # The heap-sort as a host program calls it.
        {"name": "host_u32_16m", "kind": "host", "key": "u32", "variant": "bottomup", "partial_buffer": True,
         "batch_size": 2048, "n": (1 << 24) + 777, "dist": "uniform"},
        # The breadth-first frontier of the knapsack models.
        {"name": "fifo_u32_64m", "kind": "fifo", "key": "u32", "n": 1 << 26},
        # Shortest paths with the queue.
        {"name": "sssp_rmat18", "kind": "sssp", "engine": "heap", "scale": 18, "edge_factor": 16},
        # The batched form: uneven grids and knapsacks in one launch.
        {"name": "searches_64", "kind": "searches", "count": 64, "batch_size": 256, "variant": "bottomup",
         "max_side": 512, "max_items": 400},
        # The served form: a burst of queries of different sizes.
        {"name": "served_16", "kind": "served", "count": 16, "batch_size": 1024, "scale": 16, "max_side": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["single", "sort", "queue", "host", "fifo", "sssp", "searches", "served"],
                       [10, 34, 16, 8, 9, 9, 8, 6])[0]
    c = {"kind": kind}
    if kind == "fifo":
        c.update(key=rng.choice(["u32", "i32", "u64"]), n=_log_int(rng, 1 << 12, 1 << 26))
        return c
    if kind == "sssp":
        c.update(engine=rng.choice(["heap", "heap", "retrieve"]), scale=rng.randint(12, 18),
                 edge_factor=rng.choice([8, 16, 24]))
        return c
    if kind == "searches":
        c.update(count=_log_int(rng, 8, 64), batch_size=rng.choice([64, 128, 256, 512]),
                 variant=rng.choice(["bottomup", "topdown"]), max_side=_log_int(rng, 96, 512),
                 max_items=rng.randint(120, 400))
        return c
    if kind == "served":
        c.update(count=rng.randint(4, 24), batch_size=rng.choice([256, 512, 1024]), scale=rng.randint(13, 16),
                 max_side=_log_int(rng, 128, 512))
        return c
    c.update(key=rng.choice(["u32", "u32", "u64", "i32"]), variant=rng.choice(["bottomup", "topdown"]))
    if kind == "single":
        c.update(batch_size=rng.choice([64, 128, 256, 512, 1024, 2048]), ops=rng.randint(12, 40))
        return c
    B = rng.choice([128, 256, 512, 1024, 1024, 2048, 2048])
    top = {"sort": 1 << 26, "queue": 1 << 22, "host": 1 << 24}[kind]
    if B < 512:
        top = min(top, 1 << 22)
    pb = rng.random() < 0.75
    n = _log_int(rng, 1 << 12, top)
    if kind == "host":
        n = max(n, 1 << 16)
    if not pb:  # without the partial buffer only whole batches come back without padding
        n = max(1, n // B) * B
    c.update(partial_buffer=pb, batch_size=B, n=n, dist=rng.choice(["uniform", "uniform", "zipf", "sorted", "reverse"]))
    return c


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _ordered(keys, key):
    """int64 values that order as the keys do (keys: the key's bits)."""
    if key == "u32":
        return keys.to(torch.int64) & 0xFFFFFFFF
    return keys.to(torch.int64) if key == "i32" else keys ^ torch.iinfo(torch.int64).min


def _bits(values, key):
    """The inverse of _ordered()."""
    return values.to(torch.int32) if key != "u64" else values ^ torch.iinfo(torch.int64).min


def _keys(key, dist, n, seed):
    """n keys below the type's maximum, as bits: uniform, sorted, reverse or
    Zipf(1.2) over 2^16 values; u64 keys are (u32 key << 32) | position."""
    g = _gen(seed)
    if dist == "zipf":
        ranks = torch.arange(1, (1 << 16) + 1, device="cuda", dtype=torch.float64)
        cdf = torch.cumsum(ranks.pow(-1.2), 0)
        u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]
        rank = torch.searchsorted(cdf, u).clamp_(max=(1 << 16) - 1)
        v = (rank * 2654435761) & 0x7FFFFFFF
    else:
        v = torch.randint(0, 0xFFFFFFFF, (n,), generator=g, device="cuda", dtype=torch.int64)
        if dist != "uniform":
            v = torch.sort(v, descending=dist == "reverse").values
    if key == "u64":
        return (v << 32) | torch.arange(n, device="cuda")
    return (v if key == "u32" else v - (1 << 31)).to(torch.int32)


def _rmat(scale, edge_factor, seed):
    """R-MAT (a=0.57, b=c=0.19), symmetrised, no self loops, weights 1-1000, as CSR."""
    g = _gen(seed)
    n, m = 1 << scale, edge_factor << scale
    src = torch.zeros(m, dtype=torch.int64, device="cuda")
    dst = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, generator=g, device="cuda")
        src = 2 * src + (r >= 0.76)
        dst = 2 * dst + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    w = torch.randint(1, 1001, (m,), generator=g, device="cuda", dtype=torch.int32)
    keep = src != dst
    s = torch.cat([src[keep], dst[keep]])
    d = torch.cat([dst[keep], src[keep]])
    w = torch.cat([w[keep], w[keep]])
    order = torch.argsort(s * n + d)
    s, d, w = s[order], d[order], w[order]
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(torch.bincount(s, minlength=n), 0)
    return gs.Graph(n, rowptr, d.to(torch.int32).contiguous(), w.contiguous())


def _source(graph, rng):
    """A vertex with edges."""
    deg = (graph.rowptr[1:] - graph.rowptr[:-1]).cpu().numpy()
    return int(rng.choice(np.nonzero(deg)[0]))


def _grid(side, rng):
    """A cost grid: 20 % obstacles (0), costs 1-9, open corners."""
    g = rng.integers(1, 10, (side, side)).astype(np.uint8)
    g[rng.random((side, side)) < 0.2] = 0
    g[0, 0] = g[-1, -1] = 1
    return g


def _instances(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["count"]):
        if i % 2 == 0:
            lo = min(64, case["max_side"])
            side = int(round(lo * (case["max_side"] / lo) ** rng.random()))
            out.append(("astar", _grid(side, rng)))
        else:
            n = int(rng.integers(min(100, case["max_items"]), case["max_items"] + 1))
            w = rng.integers(1, 1001, n).astype(np.int32)
            p = (w + rng.integers(0, 101, n)).astype(np.int32)
            out.append(("knapsack", (w, p, int(w.sum()) // 2)))
    return out


def _served_data(case, seed):
    rng = np.random.default_rng(seed)
    graphs = [_rmat(s, 16, seed + s) for s in (case["scale"] - 2, case["scale"])]
    maps = [_grid(side, rng) for side in (max(64, case["max_side"] // 2), case["max_side"])]
    queries = []
    for i in range(case["count"]):
        big = int(rng.random() < 0.35)
        if i % 2 == 0:
            queries.append((gsv.SSSP, big, _source(graphs[big], rng), 0))
        else:
            cells = np.nonzero(maps[big].reshape(-1))[0]
            a, b = (int(x) for x in rng.choice(cells, 2))
            queries.append((gsv.ASTAR, 2 + big, a, b))
    return graphs, maps, queries


def _ops(case, seed):
    """(operation, size) pairs: inserts first and then a mix of all three, whose
    order the case gives and whose sizes the seed."""
    rng, order = np.random.default_rng(seed), np.random.default_rng(case["ops"])
    B, out = case["batch_size"], []
    for i in range(case["ops"]):
        r = order.random()
        if i < 4 or r < 0.5:
            out.append(("insert", B if rng.random() < 0.5 else int(rng.integers(1, B + 1))))
        elif r < 0.8:
            out.append(("delete", B))
        else:
            out.append(("retrieve", int(rng.integers(1, B + 1))))
    return out


def _batch_num(n, B):
    bn = 1
    while bn * B < 2 * n:
        bn <<= 1
    return bn


def _heap(case, n):
    return gh.Heap(_batch_num(n, case["batch_size"]), case["batch_size"], key=case["key"], variant=case["variant"],
                   partial_buffer=case.get("partial_buffer", True))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sssp":
        g = _rmat(case["scale"], case["edge_factor"], seed)
        src = _source(g, np.random.default_rng(seed))
        s = {"case": case, "graph": g, "source": src, "dist": torch.empty(g.n, dtype=torch.int32, device="cuda")}
        if case["engine"] == "heap":
            s["heap"] = gs.make_heap(g)
        return s
    if kind == "searches":
        b = gb.Batch(_instances(case, seed), batch_size=case["batch_size"], variant=case["variant"],
                     astar_cells_per_block=1 << 16, timeout=20.0)
        return {"case": case, "batch": b}
    if kind == "served":
        graphs, maps, queries = _served_data(case, seed)
        srv = gsv.Server(arena_bytes=2 << 30, max_slots=64, batch_size=case["batch_size"], batches_per_step=32)
        for g in graphs:
            srv.add_graph(g)
        for m in maps:
            srv.add_map(torch.from_numpy(m).cuda())
        return {"case": case, "server": srv, "queries": queries}
    if kind == "single":
        ops = _ops(case, seed)
        n = sum(size for op, size in ops if op == "insert")
        keys = _keys(case["key"], "uniform", n, seed)
        return {"case": case, "ops": ops, "keys": keys, "heap": _heap(case, n), "out": torch.zeros_like(keys),
                "part": torch.zeros_like(keys[:case["batch_size"]]).repeat(len(ops))}
    n = case["n"]
    if kind == "fifo":
        keys = _keys(case["key"], "uniform", n, seed)
        return {"case": case, "keys": keys, "out": torch.zeros_like(keys), "fifo": Fifo(n, case["key"])}
    keys = _keys(case["key"], case["dist"], n, seed)
    if kind == "host":
        host = keys.cpu().pin_memory()
        return {"case": case, "keys": host, "out": torch.zeros_like(host).pin_memory(), "heap": _heap(case, n)}
    return {"case": case, "keys": keys, "out": torch.zeros_like(keys), "heap": _heap(case, n)}


# ---------------------------------------------------------------- one pass
def _queue_plan(case):
    """Of a queue's keys: how many come in the first bulk insert, and the limit of the first bulk delete."""
    B, n = case["batch_size"], case["n"]
    first = max(B, (3 * n // 4) // B * B)
    first = min(first, n)
    return first, first // 3


def _threshold(case):
    """Keys below it leave in the queue's second delete: a bit over a third of the range."""
    v = int(0.4 * 0xFFFFFFFF)
    if case["dist"] == "zipf":
        v >>= 1
    return {"u32": v, "i32": v - (1 << 31), "u64": v << 32}[case["key"]]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sort":
        state["heap"].sort(state["keys"], state["out"])
        return state["out"]
    if kind == "host":
        state["heap"].sort_host(state["keys"], state["out"])
        state["heap"].sync()
        return state["out"]
    if kind == "queue":
        h, keys, out = state["heap"], state["keys"], state["out"]
        first, limit = _queue_plan(case)
        h.reset_async()
        h.insert(keys[:first])
        a = h.delete(out, max_keys=limit)
        if first < keys.numel():
            h.insert(keys[first:])
        b = h.delete_below(out[a:], _threshold(case))
        c = h.delete(out[a + b:])
        return {"out": out, "counts": [a, b, c]}
    if kind == "single":
        h, keys, out, part = state["heap"], state["keys"], state["out"], state["part"]
        B = case["batch_size"]
        h.reset_async()
        counts, pos = [], 0
        for op, size in state["ops"]:
            if op == "insert":
                h.insertion(keys[pos:pos + size], size)
                pos += size
            elif op == "delete":
                counts.append(h.delete_root(part))  # lands at the heap's output cursor
            else:
                counts.append(h.retrieve(out, size))
        return {"deleted": part, "retrieved": out[:B], "counts": np.array(counts, np.int64)}
    if kind == "fifo":
        f = state["fifo"]
        f.push(state["keys"])
        n = f.pop(state["out"])
        return {"out": state["out"], "n": n}
    if kind == "sssp":
        if case["engine"] == "heap":
            return gs.sssp(state["heap"], state["graph"], state["source"], state["dist"])[0]
        return gs.sssp_retrieve(state["graph"], state["source"], dist=state["dist"])[0]
    if kind == "searches":
        b = state["batch"]
        b.run("graph")
        res, status, _ = b.results()
        return {"results": res, "status": status}
    srv = state["server"]
    srv.start(idle_ms=20)
    ids = [srv.submit(*q) for q in state["queries"]]
    left = len(ids)
    while left:
        left -= len(srv.poll()[0])
    srv.stop()
    return np.array([srv.result(q)[:3] for q in ids], np.int64)


def work(case):
    kind = case["kind"]
    if kind == "sssp":
        m = 2 * case["edge_factor"] << case["scale"]
        return {"bytes": 8 * m + (12 << case["scale"]), "flops": 0}  # CSR in, distances out
    if kind == "searches":  # each grid cell and each item read once, on average
        lo, hi = min(64, case["max_side"]), case["max_side"]
        cells = lo * lo if hi == lo else (hi * hi - lo * lo) / (2 * math.log(hi / lo))
        return {"bytes": case["count"] / 2 * (cells + 4 * case["max_items"]), "flops": 0}
    if kind == "served":
        m = 16 * 2 << case["scale"]
        side = case["max_side"]
        return {"bytes": case["count"] / 2 * (8 * (0.35 * m + 0.65 * m / 4) + 0.35 * side * side + 0.65 * side * side / 4),
                "flops": 0}
    if kind == "single":
        return {"bytes": 1.2 * case["ops"] * case["batch_size"] * KEY_BYTES[case["key"]], "flops": 0}
    return {"bytes": 2 * case["n"] * KEY_BYTES[case["key"]], "flops": 0}


# ---------------------------------------------------------------- the same in plain torch and numpy
def _relax(rowptr, col, w, source, n):
    """Shortest distances by repeated relaxation of every edge, int64."""
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), rowptr[1:] - rowptr[:-1])
    dst, w = col.to(torch.int64), w.to(torch.int64)
    dist = torch.full((n,), INF, dtype=torch.int64, device="cuda")
    dist[source] = 0
    while True:
        new = dist.scatter_reduce(0, dst, dist[src] + w, "amin")
        if torch.equal(new, dist):
            return dist
        dist = new


def _grid_cost(cost, a, b):
    """The cheapest 4-connected path from cell a to cell b; a move costs the cell it enters."""
    h, w = cost.shape
    c = torch.from_numpy(cost).cuda().to(torch.int64)
    open_, inf = c > 0, torch.tensor(INF, device="cuda")
    if not cost.reshape(-1)[a] or not cost.reshape(-1)[b]:
        return UNREACHABLE
    d = torch.full((h + 2, w + 2), INF, dtype=torch.int64, device="cuda")
    d[1 + a // w, 1 + a % w] = 0
    for it in range(1, h * w + 2):
        mid = d[1:-1, 1:-1]
        best = torch.minimum(torch.minimum(d[:-2, 1:-1], d[2:, 1:-1]), torch.minimum(d[1:-1, :-2], d[1:-1, 2:]))
        new = torch.minimum(mid, torch.where(open_, best + c, inf))
        if it % 32 == 0 and torch.equal(new, mid):
            break
        d[1:-1, 1:-1] = new
    v = int(d[1 + b // w, 1 + b % w])
    return v if v < INF else UNREACHABLE


def _knapsack_best(w, p, cap):
    dp = torch.zeros(cap + 1, dtype=torch.int64, device="cuda")
    for wi, pi in zip(w.tolist(), p.tolist()):
        if wi <= cap:
            dp[wi:] = torch.maximum(dp[wi:], dp[:cap + 1 - wi] + pi)
    return int(dp.max())


def _exact_queue(case, keys):
    B, key = case["batch_size"], case["key"]
    first, limit = _queue_plan(case)
    v = _ordered(keys, key)
    x = torch.sort(v[:first]).values
    a = x.numel() if limit >= x.numel() else limit // B * B
    if x.numel() < B:  # a partial buffer alone comes out whole or not at all
        a = x.numel() if x.numel() <= limit else 0
    y = torch.sort(torch.cat([x[a:], v[first:]])).values
    t = _threshold(case)
    if key == "u64":
        t -= 1 << 63
    m, b = y.numel(), 0
    while b < m and int(y[b]) < t:
        b += B if m - b >= B else m - b
    return {"out": _bits(torch.cat([x[:a], y]), key), "counts": [a, b, m - b]}


def _exact_single(case, seed):
    ops = _ops(case, seed)
    n = sum(size for op, size in ops if op == "insert")
    key, B = case["key"], case["batch_size"]
    v = _ordered(_keys(key, "uniform", n, seed), key).cpu().numpy()
    held, pos = np.zeros(0, np.int64), 0
    deleted, last, counts = [], np.zeros(0, np.int64), []
    for op, size in ops:
        if op == "insert":
            held = np.sort(np.concatenate([held, v[pos:pos + size]]))
            pos += size
            continue
        got, held = np.split(held, [min(size, B, held.size)])
        counts.append(got.size)
        if op == "delete":
            deleted.append(got)
        else:
            last = np.concatenate([got, last[got.size:]])
    tail = lambda x, m: torch.cat([_bits(torch.from_numpy(x), key), torch.zeros(m - x.size, dtype=torch.int64 if key == "u64" else torch.int32)])  # noqa: E731
    done = np.concatenate(deleted) if deleted else np.zeros(0, np.int64)
    return {"deleted": tail(done, B * len(ops)), "retrieved": tail(last, min(B, n)), "counts": np.array(counts, np.int64)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sort", "host"):
        keys = _keys(case["key"], case["dist"], case["n"], seed)
        return _bits(torch.sort(_ordered(keys, case["key"])).values, case["key"])
    if kind == "queue":
        return _exact_queue(case, _keys(case["key"], case["dist"], case["n"], seed))
    if kind == "single":
        return _exact_single(case, seed)
    if kind == "fifo":
        return {"out": _keys(case["key"], "uniform", case["n"], seed), "n": case["n"]}
    if kind == "sssp":
        g = _rmat(case["scale"], case["edge_factor"], seed)
        d = _relax(g.rowptr, g.col, g.w, _source(g, np.random.default_rng(seed)), g.n)
        return d.clamp(max=UNREACHABLE).to(torch.int32)
    if kind == "searches":
        res = [_grid_cost(d, 0, d.size - 1) if k == "astar" else _knapsack_best(*d) for k, d in _instances(case, seed)]
        return {"results": np.array(res, np.int64), "status": np.zeros(len(res), np.int32)}
    graphs, maps, queries = _served_data(case, seed)
    out = []
    for k, d, a, b in queries:
        if k == gsv.SSSP:
            dist = _relax(graphs[d].rowptr, graphs[d].col, graphs[d].w, a, graphs[d].n)
            fin = dist < INF
            out.append((gsv.FINISHED, int(fin.sum()), int(dist[fin].sum())))
        else:
            out.append((gsv.FINISHED, _grid_cost(maps[d - 2], a, b), 0))
    return np.array(out, np.int64)
