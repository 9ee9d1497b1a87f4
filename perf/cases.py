"""Workloads whose speed is measured: continuous subgraph matching as programs use this package.

A case is one program shape -- plugin calls update by update, batches of a stream, standing queries on one
graph, InitialMatching, Preprocessing -- over a synthetic RMAT graph (a = 0.57, b = c = 0.19) of one of four
label families, with a fixed standing query of that family:

  few    4 vertex labels uniform, 1 edge label     6-vertex induced query
  mid    8 vertex labels Zipf(1.0), 2 edge labels  8- and 12-vertex sparse queries
  many   16 vertex labels Zipf(1.2), 4 edge labels 16-vertex dense query; 5, 13 and 7 vertices beside it
  wide   32 vertex labels Zipf(1.0), 4 edge labels 24-vertex sparse query

The families, average degrees, insertion shares, caps and batch sizes are those of the workload generator's
presets (paracosm_b200/host/workload.cpp) and of bench.py; the queries were drawn once by that generator.

A pass of a stream case is one step of a sliding window: the arriving updates (insertions of held-out edges
and deletions of present ones, in one seeded order), then the same edges leaving again (the reverse order,
every update undone).  Both halves count the same embeddings, and the graph is back where it was.
"""
import numpy as np
import torch

import paracosm_b200 as pc

FAMILIES = {  # vertex labels, Zipf exponent (0: uniform), edge labels, average degree unless the case gives one
    "few": (4, 0.0, 1, 8),
    "mid": (8, 1.0, 2, 16),
    "many": (16, 1.2, 4, 28),
    "wide": (32, 1.0, 4, 32),
}

QUERIES = {  # vertex labels, edges (u, v, label)
    "induced6": ("2 0 3 1 3 0", "0-1:0 0-2:0 1-2:0 2-3:0 2-4:0 2-5:0 3-4:0 4-5:0"),
    "sparse8": ("0 0 3 5 2 0 3 3", "0-1:1 1-2:1 2-3:0 2-5:0 2-7:1 3-4:1 4-5:0 5-6:1 6-7:1"),
    "sparse12": ("5 1 2 1 2 0 6 6 0 3 0 0",
                 "0-1:1 1-2:0 2-3:0 3-4:0 3-10:0 4-5:1 5-6:0 6-7:1 7-8:1 7-9:0 8-9:0 9-10:1 10-11:1"),
    "dense16": ("7 0 2 0 5 1 10 1 0 0 9 0 0 0 8 7",
                "0-1:0 1-2:2 1-4:1 1-7:1 2-3:2 2-6:3 2-13:2 3-4:0 4-5:0 4-6:0 4-7:2 4-8:2 4-13:3 4-14:3 4-15:1 "
                "5-6:0 6-7:1 6-8:0 6-9:0 6-13:2 7-8:0 7-9:1 7-13:2 7-14:0 8-9:3 8-13:1 9-10:3 9-12:1 9-13:1 "
                "10-11:1 10-14:1 11-12:3 12-13:0 13-14:2 14-15:0"),
    "small5": ("3 2 7 3 0", "0-1:0 1-2:0 1-3:0 2-3:2 3-4:3"),
    "dense13": ("3 12 3 0 0 0 2 9 14 4 0 0 1",
                "0-1:0 1-2:2 2-3:0 2-7:0 2-8:1 3-4:3 3-5:2 3-7:1 3-8:2 3-9:3 3-10:1 4-5:1 4-7:1 4-8:0 4-10:3 "
                "5-6:0 5-7:0 5-8:1 5-10:0 5-12:3 6-7:1 6-10:3 7-8:0 7-10:0 7-12:3 8-9:1 8-10:0 8-12:2 9-10:3 "
                "10-11:2 11-12:1"),
    "cycle7": ("0 0 13 1 2 2 0", "0-1:3 1-2:0 2-3:0 2-6:0 3-4:0 4-5:2 5-6:0"),
    "sparse24": ("21 16 10 13 3 4 0 1 17 6 8 9 13 7 2 0 1 3 0 8 10 1 6 1",
                 "0-1:1 1-4:0 1-12:1 1-19:1 1-20:3 2-8:3 2-19:0 3-11:0 3-16:3 4-5:1 4-16:1 4-17:0 6-12:1 7-16:3 "
                 "7-23:3 8-18:1 9-10:1 10-11:0 11-20:0 13-18:1 14-16:3 15-16:3 16-23:3 18-22:0 21-22:3"),
}

STANDING = ("dense16", "small5", "dense13", "cycle7")  # queries of the standing-query cases, in turn


def listed():
    return [
        # a program that calls the plugin update by update, as the reference's driver does: a few edges arrive
        # and leave again (AddEdge, RemoveEdge); latency only
        dict(name="plugin_call", kind="calls", family="few", log2_n=14, query="induced6",
             algorithm="parallel_symbi", updates=12, insert=1.0, cap=0),
        # the same program over a short stream on a larger graph, where most updates match no query edge
        dict(name="plugin_stream", kind="calls", family="mid", log2_n=19, query="sparse8",
             algorithm="parallel_turboflux", updates=125, insert=0.9, cap=100_000),
        # the plain form: one update per launch sequence, many updates queued by one submit
        dict(name="plain_submit", kind="stream", family="many", log2_n=19, query="dense13",
             algorithm="parallel_symbi", updates=1000, insert=0.8, cap=100_000, mode="plain"),
        # a serving loop at a low arrival rate: small batches, replayed as CUDA graphs
        dict(name="serve_batch", kind="stream", family="many", log2_n=20, query="dense13",
             algorithm="parallel_symbi", updates=100, insert=0.85, cap=10_000, graphs=True),
        # the first benchmark configuration: 2,000 insertions in one batch, GraphFlow (no index), no cap
        dict(name="insert_2000", kind="stream", family="few", log2_n=14, query="induced6",
             algorithm="parallel_graphflow", updates=2000, insert=1.0, cap=0),
        # an ordinary batch of a stream that is already on the device, tree index
        dict(name="batch_4097", kind="stream", family="mid", log2_n=19, query="sparse12",
             algorithm="parallel_turboflux", updates=4097, insert=0.9, cap=100_000, resident=True),
        # every embedding's hash (the reference's --print-enum check): the search enumerates instead of
        # counting the tail of an order
        dict(name="hash_3001", kind="stream", family="mid", log2_n=17, query="sparse8",
             algorithm="parallel_symbi", updates=3001, insert=0.8, cap=10_000, hash=True),
        # homomorphisms, lighting filter
        dict(name="homo_1500", kind="stream", family="wide", log2_n=16, query="sparse24",
             algorithm="parallel_calig", updates=1500, insert=0.9, cap=10_000, homo=True),
        # standing queries on one graph: each batch is applied once and searched for every query
        dict(name="standing_4", kind="standing", family="many", log2_n=18, query="dense16",
             algorithm="parallel_symbi", updates=1000, insert=0.85, cap=10_000),
        # InitialMatching on the loaded graph
        dict(name="initial_match", kind="initial", family="few", log2_n=13, query="induced6",
             algorithm="parallel_turboflux"),
        # Preprocessing from host arrays to a built index, with the size of the index read back
        dict(name="preprocess", kind="preprocess", family="mid", log2_n=19, query="sparse8",
             algorithm="parallel_symbi"),
        # the headline configuration: a full batch of 65,536 updates on the 2^22-vertex graph, SymBi
        dict(name="batch_65536", kind="stream", family="many", log2_n=22, query="dense16",
             algorithm="parallel_symbi", updates=65536, insert=0.8, cap=1_000_000),
    ]


def draw(rng):
    def log_uniform(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["calls", "standing", "initial", "preprocess"] + ["stream"] * 5)
    families = {"calls": ["few", "mid"], "standing": ["many"], "initial": ["few"]}.get(kind, ["few", "mid", "many"])
    family = rng.choice(families)
    query = {"few": ["induced6"], "mid": ["sparse8", "sparse12"], "many": ["dense16", "small5"]}[family]
    log2_n = {"few": (11, 15), "mid": (13, 18), "many": (14, 19)}[family]
    if kind == "initial":
        log2_n = (10, 13)
    case = dict(kind=kind, family=family, log2_n=rng.randint(*log2_n), query=rng.choice(query),
                algorithm=rng.choice(["parallel_graphflow", "parallel_turboflux", "parallel_symbi",
                                      "parallel_calig", "parallel_newsp"]))
    if kind in ("initial", "preprocess"):
        return dict(case, degree=rng.randint(4, 10 if kind == "initial" else 32))
    case.update(insert=rng.choice([0.8, 0.85, 0.9, 1.0]), cap=log_uniform(1_000, 100_000))
    fewest = 4 if family == "few" else 48  # most updates of the larger label families match no query edge
    if kind == "calls":
        case.update(updates=log_uniform(fewest, 150))
    elif kind == "standing":
        case.update(updates=log_uniform(fewest, 2000))
    else:
        case.update(updates=log_uniform(fewest, 20_000))
        option = rng.choice(["", "", "plain", "graphs", "hash", "homo", "resident"])
        if option == "plain":
            case.update(mode="plain", updates=min(case["updates"], 1500))
        elif option in ("hash", "homo"):
            case.update({option: True}, cap=min(case["cap"], 10_000))
        elif option:
            case.update({option: True})
    return case


# ---------------------------------------------------------------------------- inputs


def _query(name):
    labels, edges = QUERIES[name]
    trip = [[int(x) for x in e.replace("-", " ").replace(":", " ").split()] for e in edges.split()]
    return np.array([int(x) for x in labels.split()], np.uint32), np.array(trip, np.uint32)


def _graph(case, seed):
    """Vertex labels and edges (v1, v2, label) of a seeded RMAT graph without self loops and repeats, in
    random order, as host arrays (what a loader gives a program)."""
    n_vl, zipf, n_el, degree = FAMILIES[case["family"]]
    dev = torch.device("cuda")
    gen = torch.Generator(dev).manual_seed(seed)
    levels, n = case["log2_n"], 1 << case["log2_n"]
    want = n * case.get("degree", degree) // 2
    keys = torch.empty(0, dtype=torch.int64, device=dev)
    while keys.numel() < want:
        m = int(1.35 * (want - keys.numel())) + 4096
        u = torch.zeros(m, dtype=torch.int64, device=dev)
        v = torch.zeros(m, dtype=torch.int64, device=dev)
        for _ in range(levels):
            r = torch.rand(m, generator=gen, device=dev)
            u = 2 * u + (r >= 0.76)
            v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        k = torch.minimum(u, v) * n + torch.maximum(u, v)
        keys = torch.unique(torch.cat([keys, k[u != v]]))
    keys = keys[torch.randperm(keys.numel(), generator=gen, device=dev)[:want]]
    place = torch.randperm(n, generator=gen, device=dev)  # hubs anywhere in the id range
    edges = torch.stack([place[keys // n], place[keys % n],
                         torch.randint(n_el, (want,), generator=gen, device=dev)], 1)
    weight = torch.arange(1, n_vl + 1, device=dev, dtype=torch.float64) ** -zipf
    cdf = torch.cumsum(weight / weight.sum(), 0)
    vl = torch.searchsorted(cdf, torch.rand(n, generator=gen, device=dev, dtype=torch.float64)).clamp_(max=n_vl - 1)
    return vl.to(torch.int32).cpu().numpy().view(np.uint32), edges.to(torch.int32).cpu().numpy().view(np.uint32)


def _stream(case, seed, edges):
    """(initial edges, arriving updates, the same updates undone)."""
    k = case["updates"]
    n_ins = max(1, int(round(k * case["insert"])))
    held, initial = edges[:n_ins], edges[n_ins:]
    chosen = np.concatenate([held, initial[:k - n_ins]])
    arrive = np.zeros(k, pc.UPDATE_DTYPE)
    arrive["type"] = ord("e")
    arrive["is_add"] = np.arange(k) < n_ins
    arrive["id1"], arrive["id2"], arrive["label"] = chosen[:, 0], chosen[:, 1], chosen[:, 2]
    arrive = arrive[np.random.RandomState(seed % (1 << 31)).permutation(k)]
    leave = arrive[::-1].copy()
    leave["is_add"] ^= 1
    return initial, arrive, leave


def _engine(case):
    return pc.Engine(case["algorithm"], max_results=case.get("cap", 0), homo=case.get("homo", False),
                     mode=case.get("mode", "batched"), want_hash=case.get("hash", False),
                     graphs=case.get("graphs", False))


def prepare(case, seed):
    vl, edges = _graph(case, seed)
    torch.cuda.empty_cache()  # the engine allocates from the device, not from torch's pool
    qv, qe = _query(case["query"])
    s = {"kind": case["kind"], "case": case}
    if case["kind"] in ("initial", "preprocess"):
        s["query"], s["data"] = pc.Graph(qv, qe), pc.Graph(vl, edges)
        if case["kind"] == "initial":
            s["plugin"] = pc.PLUGINS[case["algorithm"]](s["query"], s["data"])
            s["plugin"].Preprocessing()
        return s
    initial, s["arrive"], s["leave"] = _stream(case, seed, edges)
    if case["kind"] == "calls":
        s["plugin"] = pc.PLUGINS[case["algorithm"]](pc.Graph(qv, qe), pc.Graph(vl, initial),
                                                    case["cap"] or 0xFFFFFFFF)
        s["plugin"].Preprocessing()
        s["calls"] = [(int(u["is_add"]), int(u["id1"]), int(u["id2"]), int(u["label"]))
                      for u in np.concatenate([s["arrive"], s["leave"]])]
        return s
    eng = s["engine"] = _engine(case)
    eng.set_query(qv, qe)
    if case["kind"] == "standing":
        eng.reserve_labels(np.arange(FAMILIES[case["family"]][0]), np.arange(FAMILIES[case["family"]][2]))
    eng.load_graph(vl, initial)
    eng.build_index()
    s["engines"] = [eng]
    if case["kind"] == "standing":
        for q, algorithm in zip(STANDING[1:], ("parallel_turboflux", "parallel_symbi", "parallel_graphflow")):
            s["engines"].append(eng.attach(*_query(q), algorithm, max_results=case["cap"]))
    if case.get("resident"):
        s["device"] = [torch.from_numpy(u.view(np.uint8).copy()).cuda() for u in (s["arrive"], s["leave"])]
    return s


# ---------------------------------------------------------------------------- passes


def _fields(r, hashes):
    out = {"pos": r["pos"], "neg": r["neg"], "status": r["status"], "safe": r["safe"]}
    if hashes:
        out["hash"] = r["hash"]
    return out


def _run_calls(s):
    p = s["plugin"]
    pos, neg = [], []
    for is_add, v1, v2, label in s["calls"]:
        a, b = p.GetNumPositiveResults(), p.GetNumNegativeResults()
        if is_add:
            p.AddEdge(v1, v2, label)
        else:
            p.RemoveEdge(v1, v2)
        pos.append(p.GetNumPositiveResults() - a)
        neg.append(p.GetNumNegativeResults() - b)
    return {"pos": np.array(pos, np.int64), "neg": np.array(neg, np.int64)}


def _run_stream(s):
    eng, out = s["engine"], []
    for k, ups in enumerate((s["arrive"], s["leave"])):
        n = len(ups)
        if "device" in s:
            first = eng.submit_device(s["device"][k].data_ptr(), n)
        else:
            first = eng.submit(ups)
        out += [_fields(e.results(first, n), s["case"].get("hash")) for e in s["engines"]]
    return out


def run(state):
    if state["kind"] == "calls":
        return _run_calls(state)
    if state["kind"] == "initial":
        state["plugin"].InitialMatching()
        return state["plugin"].GetNumInitialResults()
    if state["kind"] == "preprocess":
        p = pc.PLUGINS[state["case"]["algorithm"]](state["query"], state["data"])
        p.Preprocessing()
        entries, vertices = p.GetMemoryCost()
        edges = p.engine.stats()["num_edges"]
        p.engine.close()
        return {"edges": edges, "index_entries": entries, "index_vertices": vertices}
    return _run_stream(state)


def work(case):
    """Bytes a pass cannot do without.  Updates: each record in and result out, both directed entries of its
    edge written, and the neighbours of both its endpoints read once (4 B each) -- by every query.  Load and
    InitialMatching: every edge (12 B in, two 4 B entries stored) or every stored entry once, and the labels."""
    degree = case.get("degree", FAMILIES[case["family"]][3])
    n = 1 << case["log2_n"]
    if case["kind"] == "initial":
        return {"bytes": 4.0 * n * degree + 4.0 * n, "flops": 0}
    if case["kind"] == "preprocess":
        return {"bytes": (12.0 + 8.0) * n * degree / 2 + 8.0 * n, "flops": 0}
    queries = len(STANDING) if case["kind"] == "standing" else 1
    per_update = 16.0 + 8.0 + queries * (48.0 + 2 * 4.0 * degree)
    return {"bytes": 2 * case["updates"] * per_update, "flops": 0}


# ---------------------------------------------------------------------------- exact counts


def _count_with_edge(adj, labels, qlab, qadj, v1, v2, label):
    """Embeddings of the query that use edge (v1, v2, label): plain backtracking over sets."""
    total = 0
    for qa in range(len(qlab)):
        for qb, ql in qadj[qa].items():
            if ql != label or qlab[qa] != labels[v1] or qlab[qb] != labels[v2]:
                continue
            m = {qa: v1, qb: v2}
            order = []
            while len(order) + 2 < len(qlab):
                placed = set(m) | set(order)
                order.append(max((q for q in range(len(qlab)) if q not in placed),
                                 key=lambda q: sum(w in placed for w in qadj[q])))

            def extend(i):
                q = order[i]
                cand = None
                for w, l in qadj[q].items():
                    if w in m:
                        near = adj[m[w]].get((qlab[q], l), set())
                        cand = near if cand is None else cand & near
                cand = cand - set(m.values())
                if i + 1 == len(order):
                    return len(cand)
                found = 0
                for x in cand:
                    m[q] = x
                    found += extend(i + 1)
                    del m[q]
                return found

            total += extend(0) if order else 1
    return total


def exact(case, seed):
    """The counts of the smallest plugin cases by plain backtracking; None for the others, whose millions of
    embeddings take minutes that way."""
    if case["kind"] != "calls" or case["family"] != "few" or case["updates"] > 16 or case["log2_n"] > 15:
        return None
    vl, edges = _graph(case, seed)
    initial, arrive, leave = _stream(case, seed, edges)
    qv, qe = _query(case["query"])
    qadj = [{} for _ in qv]
    for a, b, l in qe.tolist():
        qadj[a][b] = qadj[b][a] = l
    labels, adj = vl.tolist(), [{} for _ in range(len(vl))]

    def link(a, b, l, present):
        for x, y in ((a, b), (b, a)):
            near = adj[x].setdefault((labels[y], l), set())
            near.add(y) if present else near.discard(y)

    for a, b, l in initial.tolist():
        link(a, b, l, True)
    pos, neg = [], []
    for u in np.concatenate([arrive, leave]):
        add, a, b, l = int(u["is_add"]), int(u["id1"]), int(u["id2"]), int(u["label"])
        if add:
            link(a, b, l, True)
        c = _count_with_edge(adj, labels, qv.tolist(), qadj, a, b, l)
        if not add:
            link(a, b, l, False)
        c = min(c, case["cap"]) if case["cap"] else c
        pos.append(c if add else 0)
        neg.append(0 if add else c)
    return {"pos": np.array(pos, np.int64), "neg": np.array(neg, np.int64)}
