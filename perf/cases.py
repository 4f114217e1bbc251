"""The work this engine is timed on: one case per thing a user has it do,
each through the calls of emptyheaded_b200 that a program makes.

A case's "kind" names the path:

  count      COUNT of one plan over a resident trie (Trie.count,
             Trie.triangle_annotation): the query a service answers again and
             again once its relation is loaded
  batch      one plan over many resident tries in one launch (Batch.run)
  load       raw edge samples on the device -> encoded relation -> trie ->
             triangle COUNT (preprocess, Trie, count): loading a graph and
             asking the first question
  host_csr   COUNT of a relation that lies as a CSR in host memory
             (count_host_csr): the call of a program whose data is on the host
  rows       the triangles themselves, sorted, on the host (Trie.materialize)
  encode     dictionary of two columns, both columns encoded, the keys decoded
             (Encoding): what the loader does with each attribute
  intersect  set intersections asked pair by pair, with their elements
             (set_intersect): the set operations as a library
  train      minibatch SGD steps of the layout cost model (Model.train), as
             learn.train makes them

Graphs are the seeded synthetic ones of emptyheaded_b200.workloads: Erdos-
Renyi, R-MAT (edge factor 16) and Chung-Lu, relabelled by degree, up-oriented
or symmetric.  Counts, rows, keys and sets are whole numbers; only the cost
model's parameters and losses are floating point.
"""
import numpy as np

import emptyheaded_b200 as E

ABCD = (0.57, 0.19, 0.19)
GAMMA = 2.1  # Chung-Lu degree exponent
DIMS = [6, 32, 32, 1]  # the layout cost model's widths


def listed():
    return [
        # the smallest call: an interactive query on a small relation, where
        # planning, launches and waits are most of the time
        dict(name="triangle_er16k", kind="count", graph="er", nodes=16384, samples=131072, symmetric=False,
             query="triangle"),
        # the headline workload: triangles of a large skewed graph
        dict(name="triangle_rmat22", kind="count", graph="rmat", nodes=1 << 22, samples=16 << 22, symmetric=False,
             query="triangle"),
        # many independent graphs of very uneven sizes answered together
        dict(name="triangle_batch", kind="batch", graphs=96, low=10, high=17, query="triangle"),
        # the deepest join
        dict(name="clique4_rmat20", kind="count", graph="rmat", nodes=1 << 20, samples=16 << 20, symmetric=False,
             query="clique4"),
        # the two-bag plans run on symmetric relations: a power-law graph with
        # hubs far larger than shared memory
        dict(name="lollipop_chunglu21", kind="count", graph="chunglu", nodes=1 << 21, samples=16 << 21,
             symmetric=True, query="lollipop"),
        # and an ordinary one
        dict(name="barbell_chunglu16", kind="count", graph="chunglu", nodes=1 << 16, samples=16 << 16,
             symmetric=True, query="barbell"),
        # loading: sort, dedup, CSR, reverse level, layouts, first query
        dict(name="load_rmat20", kind="load", graph="rmat", nodes=1 << 20, samples=16 << 20, symmetric=False),
        # one question about host data, copies included
        dict(name="host_csr_rmat20", kind="host_csr", graph="rmat", nodes=1 << 20, samples=16 << 20,
             symmetric=False, query="triangle"),
        # a materialised result of some hundred thousand rows
        dict(name="rows_rmat12", kind="rows", graph="rmat", nodes=1 << 12, samples=16 << 12, symmetric=False),
        # user ids: 64-bit, sparse, each seen a few times
        dict(name="encode_int64", kind="encode", value_type="int64", rows=1000000, distinct=300000),
        # uneven sets in every layout
        dict(name="intersect_mixed", kind="intersect", sets=512, longest=16384, span=1 << 20, pairs=4096),
        # a stretch of training on the engine's own logs
        dict(name="train_sgd", kind="train", batch=2048, steps=16),
    ]


def _log_int(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    kind = rng.choice(["count", "count", "count", "batch", "load", "host_csr", "rows", "encode", "intersect", "train"])
    if kind == "count":
        query = rng.choice(["triangle", "triangle", "clique4", "lollipop", "barbell", "annotation"])
        # (an Erdos-Renyi graph has no 4-cliques to speak of)
        graph = rng.choice(["rmat", "chunglu"] if query == "clique4" else ["er", "rmat", "chunglu"])
        symmetric = query in ("lollipop", "barbell", "annotation") or rng.random() < 0.25
        # the 4-clique of a symmetric hub-heavy graph costs far more per row
        top = {"triangle": 1 << 21, "clique4": 1 << 18}.get(query, 1 << 19)
        if symmetric and query in ("triangle", "clique4"):
            top = 1 << 15 if query == "clique4" else 1 << 19
        nodes = _log_int(rng, 1000, top)
        if graph == "rmat":
            nodes = 1 << (nodes.bit_length() - 1)
        return dict(kind=kind, graph=graph, nodes=nodes, samples=int(nodes * rng.uniform(8, 16)),
                    symmetric=symmetric, query=query)
    if kind == "batch":
        low = rng.randint(8, 12)
        return dict(kind=kind, graphs=_log_int(rng, 4, 128), low=low, high=rng.randint(low, 15),
                    query=rng.choice(["triangle", "triangle", "clique4"]))
    if kind in ("load", "host_csr"):
        nodes = _log_int(rng, 1000, 1 << 20)
        graph = rng.choice(["er", "rmat", "chunglu"])
        if graph == "rmat":
            nodes = 1 << (nodes.bit_length() - 1)
        case = dict(kind=kind, graph=graph, nodes=nodes, samples=int(nodes * rng.uniform(4, 16)),
                    symmetric=rng.random() < 0.25)
        if kind == "host_csr":
            case["query"] = "triangle"
        return case
    if kind == "rows":
        nodes = _log_int(rng, 500, 1 << 15)
        graph = rng.choice(["er", "rmat", "chunglu"])
        if graph == "rmat":
            nodes = 1 << (nodes.bit_length() - 1)
        return dict(kind=kind, graph=graph, nodes=nodes, samples=int(nodes * rng.uniform(4, 16)), symmetric=False)
    if kind == "encode":
        rows = _log_int(rng, 1000, 4000000)
        return dict(kind=kind, value_type=rng.choice(["uint32", "int32", "int64", "float32"]), rows=rows,
                    distinct=max(2, int(rows * rng.uniform(0.01, 0.6))))
    if kind == "intersect":
        return dict(kind=kind, sets=_log_int(rng, 2, 1000), longest=_log_int(rng, 100, 30000),
                    span=_log_int(rng, 1 << 16, 1 << 24), pairs=_log_int(rng, 1, 8000))
    return dict(kind=kind, batch=_log_int(rng, 64, 4096), steps=rng.randint(4, 24))


# ------------------------------------------------------------------ inputs
def _samples(case, seed):
    """Device edge samples of the case's graph."""
    if case["graph"] == "er":
        return E.gen_er(seed, case["nodes"], case["samples"])
    if case["graph"] == "rmat":
        return E.gen_rmat(seed, case["nodes"].bit_length() - 1, case["samples"], *ABCD)
    return E.gen_chunglu(seed, case["nodes"], case["samples"], GAMMA)


def _trie(case, seed):
    u, v = _samples(case, seed)
    s, d, _ = E.preprocess(u, v, symmetric=case["symmetric"])
    u.free()
    v.free()
    t = E.Trie(s, d)
    s.free()
    d.free()
    return t


def _gaps(n, rng):
    """A strictly increasing renaming of 0..n-1 that leaves a fifth of the
    ids unused, as a store does after deletions."""
    return np.sort(rng.permutation(n + n // 4)[:n]).astype(np.uint32)


def _rows_trie(case, seed):
    """The case's graph, the same for every seed, with the seed's ids: the
    result has the same number of rows, and others."""
    u, v = _samples(case, 7)
    s, d, nodes = E.preprocess(u, v, symmetric=case["symmetric"])
    ids = _gaps(nodes, np.random.default_rng(seed))
    return E.Trie(ids[s.numpy()], ids[d.numpy()])


def _batch_scales(case):
    # uneven and the same for every seed: spread over the logarithm of the scale
    n, low, high = case["graphs"], case["low"], case["high"]
    return [int(round(low * (high / low) ** ((i + 0.5) / n))) for i in range(n)]


def _columns(case, seed):
    """Two columns over one set of distinct values, each of which occurs."""
    rng = np.random.default_rng(seed)
    dt = E.VALUE_TYPES[case["value_type"]][1]
    n, rows = case["distinct"], case["rows"]
    if dt == np.uint32:  # dense ids
        values = rng.permutation(n + n // 4)[:n].astype(dt)
    else:
        values = np.zeros(0, dt)
        while len(values) < n:
            if dt == np.float32:
                more = rng.normal(0, 1000, n + n // 8 + 64).astype(dt)
            elif dt == np.int32:
                more = rng.integers(-(1 << 31), 1 << 31, n + n // 8 + 64).astype(dt)
            else:
                more = rng.integers(-(1 << 40), 1 << 40, n + n // 8 + 64)
            values = np.unique(np.concatenate([values, more]))
        values = rng.permutation(values)[:n]
    first = np.concatenate([values, values[rng.integers(0, n, rows - n)]])
    return [rng.permutation(first), values[rng.integers(0, n, rows)]]


def _sets(case, seed):
    """Sets that cross in the same places for every seed, over the seed's
    elements and in the seed's layouts."""
    rng = np.random.default_rng(7)
    sizes = np.exp(rng.uniform(np.log(4), np.log(case["longest"]), case["sets"])).astype(int)
    sets = []
    for k, size in enumerate(sizes):
        # from clustered to spread over the whole span
        width = int(min(case["span"], max(size, size * 4 ** (k % 5))))
        start = int(rng.integers(0, case["span"] - width + 1))
        sets.append(np.unique(rng.integers(start, start + width, size)).astype(np.uint32))
    pairs = rng.integers(0, case["sets"], (case["pairs"], 2)).astype(np.uint32)
    rng = np.random.default_rng(seed)
    used = np.unique(np.concatenate(sets))
    ids = used + np.sort(rng.integers(0, case["span"] // 4, len(used))).astype(np.uint32)
    sets = [ids[np.searchsorted(used, s)] for s in sets]
    layouts = np.array([E.UINTEGER, E.RANGE_BITSET, E.BLOCK_BITSET], np.uint8)[rng.integers(0, 3, case["sets"])]
    return sets, layouts, pairs


def _training(case, seed):
    """Initial parameters and one minibatch of standardised rows per step."""
    rng = np.random.default_rng(seed)
    params = []
    for i, o in zip(DIMS[:-1], DIMS[1:]):
        params += [rng.uniform(-1, 1, i * o) * np.sqrt(3.0 / i), np.zeros(o)]
    x = rng.normal(0, 1, (case["steps"], case["batch"], DIMS[0])).astype(np.float32)
    y = (np.tanh(x[..., :1] - x[..., 1:2]) + 0.1 * rng.normal(0, 1, x.shape[:2] + (1,))).astype(np.float32)
    return np.concatenate(params).astype(np.float32), x, y


LR = 0.05


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "count":
        state["trie"] = _trie(case, seed)
    elif kind == "rows":
        state["trie"] = _rows_trie(case, seed)
    elif kind == "batch":
        tries = [_trie(dict(graph="rmat", nodes=1 << s, samples=16 << s, symmetric=False), 1000 * seed + i)
                 for i, s in enumerate(_batch_scales(case))]
        state["batch"] = E.Batch(tries, case["query"])
    elif kind == "load":
        state["u"], state["v"] = _samples(case, seed)
    elif kind == "host_csr":
        t = _trie(case, seed)
        head, off, vals, _ = t.export()
        state["nodes"] = t.info()["n_nodes"]
        t.free()
        state["csr"] = [_pinned(a) for a in (head, off, vals)]
    elif kind == "encode":
        state["cols"] = _columns(case, seed)
    elif kind == "intersect":
        state["sets"], state["layouts"], state["pairs"] = _sets(case, seed)
    elif kind == "train":
        state["params"], state["x"], state["y"] = _training(case, seed)
        state["model"] = E.Model(DIMS)
    return state


def _pinned(a):
    """The array in pinned host memory (uint64 as int64 bits: torch copies
    neither)."""
    import torch
    bits = torch.from_numpy(np.ascontiguousarray(a).view({4: np.int32, 8: np.int64}[a.dtype.itemsize]))
    out = torch.empty(bits.shape, dtype=bits.dtype, pin_memory=True)
    out.copy_(bits)
    return out.numpy().view(a.dtype)


# --------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "count":
        if case["query"] == "annotation":
            return state["trie"].triangle_annotation()
        return state["trie"].count(case["query"])
    if kind == "batch":
        return state["batch"].run()
    if kind == "load":
        s, d, nodes = E.preprocess(state["u"], state["v"], symmetric=case["symmetric"])
        t = E.Trie(s, d)
        s.free()
        d.free()
        info = t.info()
        out = [nodes, t.count("triangle")] + [info[k] for k in (
            "rows", "n_head", "n_nodes", "head_layout", "n_uinteger", "n_range_bitset", "n_block_bitset",
            "bitset_words", "max_set")]
        t.free()
        return out
    if kind == "host_csr":
        head, off, vals = state["csr"]
        return E.count_host_csr(head, off, vals, state["nodes"], case["query"])
    if kind == "rows":
        return state["trie"].materialize()
    if kind == "encode":
        enc = E.Encoding(state["cols"], case["value_type"])
        keys = [enc.encode(c) for c in state["cols"]]
        values = [enc.decode(k) for k in keys]
        out = [enc.values(), keys, values]
        enc.free()
        return out
    if kind == "intersect":
        counts, elems = E.set_intersect(state["sets"], state["layouts"], state["pairs"], materialize=True)
        return counts, np.concatenate(elems)
    model = state["model"]
    model.set_params(state["params"])
    losses = [model.train(x, y, lr=LR, steps=1) for x, y in zip(state["x"], state["y"])]
    return model.params(), losses


def work(case):
    """Bytes and operations of one pass that the path cannot do without."""
    kind = case["kind"]
    if kind in ("count", "load", "host_csr", "rows"):
        rows = case["samples"] * (2 if case["symmetric"] else 1)
        csr = 4 * rows + 8 * case["nodes"]
        if kind == "count":
            return {"bytes": csr + (8 * case["nodes"] if case["query"] == "annotation" else 8), "flops": 0}
        if kind == "load":
            return {"bytes": 8 * case["samples"] + csr, "flops": 0}
        if kind == "host_csr":
            return {"bytes": csr + 8, "flops": 0}
        return {"bytes": csr + 12 * 4 * rows, "flops": 0}
    if kind == "batch":
        edges = sum(16 << s for s in _batch_scales(case))
        return {"bytes": 4 * edges + 8 * case["graphs"], "flops": 0}
    if kind == "encode":
        width = np.dtype(E.VALUE_TYPES[case["value_type"]][1]).itemsize
        return {"bytes": 2 * case["rows"] * (2 * width + 4) + width * case["distinct"], "flops": 0}
    if kind == "intersect":
        mean = (case["longest"] - 4) / max(np.log(case["longest"] / 4.0), 1.0)  # of sizes even in their logarithm
        return {"bytes": float(4 * mean * case["sets"] + 8 * case["pairs"]), "flops": 0}
    params = sum((i + 1) * o for i, o in zip(DIMS[:-1], DIMS[1:]))
    return {"bytes": 4 * case["steps"] * (case["batch"] * (DIMS[0] + DIMS[-1]) + 2 * params),
            "flops": 6 * case["steps"] * case["batch"] * params}


def exact(case, seed):
    """The cost model's parameters and losses in 64 bits; everything else is
    whole numbers."""
    if case["kind"] != "train":
        return None
    p0, xs, ys = _training(case, seed)
    p = p0.astype(np.float64)
    layers, at = [], 0
    for i, o in zip(DIMS[:-1], DIMS[1:]):
        layers.append((p[at:at + i * o].reshape(o, i), p[at + i * o:at + (i + 1) * o]))
        at += (i + 1) * o
    losses = []
    for x, y in zip(xs.astype(np.float64), ys.astype(np.float64)):
        acts = [x]
        for k, (w, b) in enumerate(layers):
            z = acts[-1] @ w.T + b
            acts.append(np.maximum(z, 0.0) if k + 1 < len(layers) else z)
        g = (acts[-1] - y) / len(x)
        losses.append(float(0.5 * np.sum((acts[-1] - y) ** 2) / len(x)))
        for k in range(len(layers) - 1, -1, -1):
            w, b = layers[k]
            gw, gb = g.T @ acts[k], g.sum(0)
            g = (g @ w) * (acts[k] > 0.0)
            w -= LR * gw
            b -= LR * gb
    return p, losses
