"""The work that is measured: static init of a forest and a sliding window of edges over it.

A user of the library builds a graph, computes the betweenness state of K roots (static init) and then follows a
stream of edges: new ones come in, old ones expire, and the BC vector is read after each change.  A case is one of

  init    one static init of K roots on a resident graph, then the BC read (and, for small forests, every root's
          levels, path counts and dependencies: what a program that inspects trees reads)
  window  one step of a sliding window: a batch of new edges is inserted, BC read, the batch that came one step
          before is deleted, BC read.  batch 1 is the caller that follows every edge by itself, as the reference's
          callers do; larger batches are the throughput form.  `via` is the entry point of the insertions: host
          arrays (synchronous, with statistics), async (host arrays, queued) or device (ids already on the GPU)
  group   the same step for many small graphs at once: one group insertion for all, deletions graph by graph

on the graph families that the benchmark and the tests use: Erdos-Renyi, Chung-Lu (connected) and R-MAT.
Graphs, roots and edges are drawn on the GPU from the seed alone.
"""
import numpy as np
import torch

from streamingbc_gb300 import native

DEV = "cuda"


def _init(name, family, size, degree, roots, read="bc"):
    return {"name": name, "op": "init", "family": family, "size": size, "degree": degree, "roots": roots, "read": read}


def _window(name, family, size, degree, roots, batch, via="host", tuned=False):
    return {"name": name, "op": "window", "family": family, "size": size, "degree": degree, "roots": roots,
            "batch": batch, "via": via, "tuned": tuned}


def listed():
    return [
        # the smallest calls: an exact forest of 200 vertices, all of whose state is read back
        _init("init_er200", "er", 200, 8, 200, "state"),
        # exact BC of a small graph (the ER 1024 configuration)
        _init("init_er1024", "er", 1024, 16, 1024),
        # a mid-size power-law graph with sampled roots (the Chung-Lu 40k configuration)
        _init("init_cl40k", "cl", 40000, 8.8, 256),
        # a large skewed graph, an odd number of roots, fewer than two per SM
        _init("init_rmat18", "rmat", 18, 32, 251),
        # the largest: R-MAT 20 with 1024 roots
        _init("init_rmat20", "rmat", 20, 32, 1024),
        # an edge at a time on the smallest graph: latency and launches
        _window("step_er200_b1", "er", 200, 8, 200, 1),
        # the ER 1024 configuration in its batches of 64, launch shape tuned as the benchmark tunes it
        _window("step_er1024_b64", "er", 1024, 16, 1024, 64, "host", True),
        # an edge at a time on the mid-size graph
        _window("step_cl40k_b1", "cl", 40000, 8.8, 256, 1),
        # the Chung-Lu 40k configuration in its batches of 64, ids on the device (replayed from a CUDA graph)
        _window("step_cl40k_b64", "cl", 40000, 8.8, 256, 64, "device"),
        # a large graph, odd batch and root count, queued host batches (what the serving loop issues)
        _window("step_rmat17_b37", "rmat", 17, 32, 301, 37, "async"),
        # the largest: R-MAT 20, 1024 roots, batches of 256
        _window("step_rmat20_b256", "rmat", 20, 32, 1024, 256),
        # many small graphs at once (the 64-graph configuration's kind, a quarter of its members)
        {"name": "group16", "op": "group", "members": 16, "scale_lo": 10, "scale_hi": 14, "degree": 16, "roots": 128,
         "batch": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(("init", "init", "window", "window", "window", "group"))
    if op == "group":
        lo = rng.randint(8, 11)
        return {"op": "group", "members": rng.randint(2, 24), "scale_lo": lo, "scale_hi": rng.randint(lo, 13),
                "degree": 16, "roots": _log_int(rng, 9, 128), "batch": _log_int(rng, 1, 24)}
    family = rng.choice(("er", "cl", "rmat"))
    if family == "er":
        size, degree = _log_int(rng, 90, 20000), round(rng.uniform(4.0, 24.0), 1)
        verts = size
    elif family == "cl":
        size, degree = _log_int(rng, 2000, 100000), round(rng.uniform(6.0, 14.0), 1)
        verts = size // 2
    else:
        size, degree = rng.randint(10, 19), rng.choice((16, 32))
        verts = 1 << size
    roots = _log_int(rng, 12, min(verts // 2, 600))
    case = {"op": op, "family": family, "size": size, "degree": degree, "roots": roots}
    if op == "init":
        case["read"] = "state" if verts * roots <= 50000 else "bc"
    else:
        case.update(batch=_log_int(rng, 1, 150), via=rng.choice(("host", "async", "device")), tuned=False)
    return case


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)
    return g


def _undirected(nv, u, v):
    """Distinct undirected edges as sorted keys lo * nv + hi."""
    keep = u != v
    u, v = u[keep], v[keep]
    return torch.unique(torch.minimum(u, v) * nv + torch.maximum(u, v))


def _rmat_pairs(scale, count, g):
    a, b, c = 0.57, 0.19, 0.19
    u = torch.zeros(count, dtype=torch.int64, device=DEV)
    v = torch.zeros(count, dtype=torch.int64, device=DEV)
    for _ in range(scale):
        r = torch.rand(count, generator=g, device=DEV)
        u = 2 * u + (r >= a + b)
        v = 2 * v + (((r >= a) & (r < a + b)) | (r >= a + b + c))
    return u, v


def _connected(nv, keys, g):
    """The keys with every smaller component tied to the largest one by an edge (the vertex count stays the case's)."""
    u, v = keys // nv, keys % nv
    lab = torch.arange(nv, device=DEV)
    while True:
        m = torch.minimum(lab[u], lab[v])
        new = lab.scatter_reduce(0, u, m, "amin").scatter_reduce(0, v, m, "amin")
        new = new[new]
        if torch.equal(new, lab):
            break
        lab = new
    big = torch.bincount(lab, minlength=nv).argmax()
    inside = torch.nonzero(lab == big).flatten()
    rep = torch.nonzero((lab == torch.arange(nv, device=DEV)) & (lab != big)).flatten()
    to = inside[torch.randint(inside.numel(), (rep.numel(),), generator=g, device=DEV)]
    return torch.sort(torch.cat([keys, torch.minimum(rep, to) * nv + torch.maximum(rep, to)])).values


def _graph(family, size, degree, g):
    """(vertex count, sorted undirected keys)."""
    if family == "rmat":
        nv = 1 << size
        u, v = _rmat_pairs(size, int(nv * degree / 2), g)
        return nv, _undirected(nv, u, v)
    m = int(size * degree / 2)
    if family == "er":
        u = torch.randint(size, (m,), generator=g, device=DEV)
        v = torch.randint(size, (m,), generator=g, device=DEV)
        return size, _undirected(size, u, v)
    # Chung-Lu: power-law expected degrees of exponent 2.4, largest min(300, sqrt(2m))
    i = torch.arange(size, dtype=torch.float64, device=DEV)
    w = torch.clamp(min(300.0, (2.0 * m) ** 0.5) * (1.0 + i / max(1.0, size / 2000.0)) ** (-1.0 / 1.4), min=1.0)
    cdf = torch.cumsum(w / w.sum(), 0)
    u, v = (torch.clamp(torch.searchsorted(cdf, torch.rand(m, generator=g, device=DEV, dtype=torch.float64)),
                        max=size - 1) for _ in range(2))
    return size, _connected(size, _undirected(size, u, v), g)


def _csr(nv, keys):
    """(offsets, neighbours) of the symmetric CSR, neighbours sorted."""
    u, v = keys // nv, keys % nv
    both = torch.sort(torch.cat([keys, v * nv + u])).values
    off = torch.zeros(nv + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(torch.bincount(both // nv, minlength=nv), 0)
    return off, both % nv


def _new_edges(family, size, nv, keys, off, adj, count, g):
    """`count` distinct pairs that are not edges: drawn by the graph's own process (R-MAT), or 70 % between vertices
    two or three steps apart and the rest uniform."""
    out = keys.new_empty(0)
    while out.numel() < count:
        n = 4 * count + 64
        if family == "rmat":
            u, v = _rmat_pairs(size, n, g)
        else:
            u = torch.randint(nv, (n,), generator=g, device=DEV)
            v = torch.randint(nv, (n,), generator=g, device=DEV)
            walk, far = u, torch.rand(n, generator=g, device=DEV)
            for step in range(3):
                d = off[walk + 1] - off[walk]
                at = off[walk] + (torch.rand(n, generator=g, device=DEV) * d).long().clamp(max=(d - 1).clamp(min=0))
                nxt = torch.where(d > 0, adj[at.clamp(max=adj.numel() - 1)], walk)
                walk = nxt if step < 2 else torch.where(far < 0.5, nxt, walk)
            v = torch.where(torch.rand(n, generator=g, device=DEV) < 0.7, walk, v)
        k = torch.minimum(u, v) * nv + torch.maximum(u, v)
        at = torch.searchsorted(keys, k).clamp(max=keys.numel() - 1)
        k = k[(u != v) & (keys[at] != k)]
        k = torch.cat([out, k])
        # distinct, in the order of first appearance
        s, order = torch.sort(k, stable=True)
        first = torch.ones_like(s, dtype=torch.bool)
        first[1:] = s[1:] != s[:-1]
        out = k[torch.sort(order[first]).values]
    return out[:count]


BATCHES = 3  # a state's batches: one is in the graph, the next comes in, and so on round and round


def _inputs(family, size, degree, roots, batch, seed):
    g = _gen(seed)
    nv, keys = _graph(family, size, degree, g)
    off, adj = _csr(nv, keys)
    k = min(roots, nv)
    rt = torch.sort(torch.randperm(nv, generator=g, device=DEV)[:k]).values
    pairs = None
    if batch:
        e = _new_edges(family, size, nv, keys, off, adj, batch * BATCHES, g)
        flip = torch.rand(e.numel(), generator=g, device=DEV) < 0.5
        a, b = e // nv, e % nv
        pairs = torch.stack([torch.where(flip, b, a), torch.where(flip, a, b)], 1).reshape(BATCHES, batch, 2)
    return nv, keys, off, adj, rt, pairs


def _member(case, m):
    """Inputs' arguments of a group's member m: its scale is spread over the range."""
    span = case["scale_hi"] - case["scale_lo"] + 1
    scale = case["scale_lo"] + (m * 7 + 3) % span
    return "rmat", scale, case["degree"], case["roots"], case["batch"]


def _forest(family, size, degree, roots, batch, seed):
    nv, _, off, adj, rt, pairs = _inputs(family, size, degree, roots, batch, seed)
    graph = native.DeviceGraph(nv, off.cpu().numpy(), adj.cpu().numpy())
    forest = native.DeviceForest(graph, rt.cpu().numpy())
    return graph, forest, pairs


# ------------------------------------------------------------------ the interface

def prepare(case, seed):
    if case["op"] == "group":
        members = [_forest(*_member(case, m), seed * 64 + m) for m in range(case["members"])]
        batches = [p.cpu().numpy() for _, _, p in members]
        for _, f, _ in members:
            f.static_init()
        group = native.DeviceGroup([f for _, f, _ in members])
        group.insert([b[0] for b in batches])
        return {"case": case, "graphs": [g for g, _, _ in members], "forests": [f for _, f, _ in members],
                "group": group, "batches": batches, "at": 0}
    graph, forest, pairs = _forest(case["family"], case["size"], case["degree"], case["roots"], case.get("batch", 0), seed)
    state = {"case": case, "graph": graph, "forest": forest, "at": 0}
    if case["op"] == "init":
        return state
    forest.static_init()
    state["batches"] = pairs.cpu().numpy()
    if case["tuned"]:
        forest.autotune(state["batches"][0])
    else:
        forest.insert(state["batches"][0])
    state["ids"] = [(p[:, 0].to(torch.int32).contiguous(), p[:, 1].to(torch.int32).contiguous()) for p in pairs]
    return state


def run(state):
    case = state["case"]
    if case["op"] == "init":
        f = state["forest"]
        f.static_init(sync=False)
        out = {"bc": f.bc()}
        if case["read"] == "state":
            out.update(dist=f.dist(), sigma=f.sigma(), delta=f.delta())
        return out
    old, new = state["at"], (state["at"] + 1) % BATCHES
    state["at"] = new
    if case["op"] == "group":
        group = state["group"]
        group.insert([b[new] for b in state["batches"]])
        grown = group.bc()
        removed = [f.delete(b[old])["inserted"] for f, b in zip(state["forests"], state["batches"])]
        return {"grown": grown, "removed": sum(removed), "shrunk": group.bc()}
    f, batch = state["forest"], state["batches"][new]
    out = {}
    if case["via"] == "host":
        st = f.insert(batch)
        out["insert"] = [st[k] for k in ("inserted", "duplicates", "invalid", "roots_active", "case1", "case2",
                                         "vertices", "edges")]
    elif case["via"] == "async":
        f.insert_async(batch)
    else:
        state["graph"].reserve(batch)
        u, v = state["ids"][new]
        f.insert_device(len(batch), u.data_ptr(), v.data_ptr())
    out["grown"] = f.bc()
    st = f.delete(state["batches"][old])
    out["delete"] = [st[k] for k in ("inserted", "duplicates", "invalid", "case1", "case2")]
    out["shrunk"] = f.bc()
    return out


def _size(case):
    """Vertices, directed adjacency entries."""
    nv = 1 << case["size"] if case["family"] == "rmat" else case["size"]
    return nv, nv * case["degree"]


def work(case):
    """init: the adjacency read once, every (root, vertex) level, path count and dependency written once; one add and
    one multiply-add per (root, adjacency entry).  Steps: two levels per (root, edge) read by each half, BC written by
    each half (what a changed root needs beyond that depends on the edge)."""
    if case["op"] == "group":
        b = f = 0.0
        for m in range(case["members"]):
            _, scale, _, roots, batch = _member(case, m)
            b += 2 * (8.0 * min(roots, 1 << scale) * batch + 8.0 * (1 << scale))
            f += 2.0 * min(roots, 1 << scale) * batch
        return {"bytes": b, "flops": f}
    nv, ne = _size(case)
    k = min(case["roots"], nv)
    if case["op"] == "init":
        return {"bytes": 4.0 * ne + 20.0 * k * nv + 8.0 * nv, "flops": 3.0 * k * ne}
    return {"bytes": 2 * (8.0 * k * case["batch"] + 8.0 * nv), "flops": 2.0 * k * case["batch"]}


def _brandes(nv, keys, roots):
    """(BC, dependencies [K][V]) by level-synchronous sparse products in 64 bits."""
    off, adj = _csr(nv, keys)
    a = torch.sparse_csr_tensor(off, adj, torch.ones(adj.numel(), dtype=torch.float64, device=DEV), size=(nv, nv))
    bc = torch.zeros(nv, dtype=torch.float64, device=DEV)
    small = nv * roots.numel() <= 1 << 24
    rows = []
    width = max(1, min(64, (1 << 27) // nv))
    for at in range(0, roots.numel(), width):
        rt = roots[at:at + width]
        col = torch.arange(rt.numel(), device=DEV)
        sigma = torch.zeros(nv, rt.numel(), dtype=torch.float64, device=DEV)
        sigma[rt, col] = 1.0
        level = torch.full((nv, rt.numel()), -1, dtype=torch.int16, device=DEV)
        level[rt, col] = 0
        front, depth = sigma, 0
        while True:
            front = torch.sparse.mm(a, front) * (level < 0)
            fresh = front > 0
            if not bool(fresh.any()):
                break
            depth += 1
            level[fresh] = depth
            sigma = sigma + front
        delta = torch.zeros_like(sigma)
        for d in range(depth, 0, -1):
            w = torch.where(level == d, (1.0 + delta) / sigma, torch.zeros_like(delta))
            delta = torch.where(level == d - 1, sigma * torch.sparse.mm(a, w), delta)
        if small:
            rows.append(delta.t().contiguous())
        delta[rt, col] = 0.0
        bc += delta.sum(1)
    return bc, torch.cat(rows) if small else None


def _with(nv, keys, pairs):
    p = pairs.reshape(-1, 2)
    return torch.sort(torch.cat([keys, torch.minimum(p[:, 0], p[:, 1]) * nv + torch.maximum(p[:, 0], p[:, 1])])).values


def exact(case, seed):
    if case["op"] == "group":
        grown, shrunk = [], []
        for m in range(case["members"]):
            nv, keys, _, _, rt, p = _inputs(*_member(case, m), seed * 64 + m)
            grown.append(_brandes(nv, _with(nv, keys, p[:2]), rt)[0])
            shrunk.append(_brandes(nv, _with(nv, keys, p[1]), rt)[0])
        return {"grown": grown, "removed": None, "shrunk": shrunk}
    nv, keys, _, _, rt, p = _inputs(case["family"], case["size"], case["degree"], case["roots"], case.get("batch", 0), seed)
    if case["op"] == "init":
        bc, delta = _brandes(nv, keys, rt)
        return {"bc": bc, "dist": None, "sigma": None, "delta": delta if case["read"] == "state" else None}
    out = {"grown": _brandes(nv, _with(nv, keys, p[:2]), rt)[0], "shrunk": _brandes(nv, _with(nv, keys, p[1]), rt)[0]}
    return dict(out, insert=None, delete=None)
