"""What a user of this package has it do, as cases that can be timed and compared.

Each case is one call (or one short sequence of calls) of the public Python API:

  enumerate   all maximal k-biplexes of a graph resident on the GPU, in count
              mode: their number and the two hashes of the set
  limited     the first `limit` results of a graph too large to enumerate
              completely
  load_limited  the same from host memory, as the command line tool does it:
              upload, check, edge hash, enumeration, release
  end_to_end  one request of a service: a graph in host memory is made resident,
              the shipped model predicts its roots' costs, the learned schedule
              enumerates it
  batch       many small graphs, each with its own k, in one run of launches
  records     the sets themselves, delivered to the host
  gradient    forward and backward pass of the subtree-size model over a
              training set

The graphs are seeded Erdos-Renyi and Chung-Lu bipartite graphs and induced
prefixes of the latter, in the sizes of gmkbe_b200.graphgen.WORKLOADS, of the
golden fixtures and of the training families of gmkbe_b200.learned, in the
converter's vertex order.  They are made on the GPU from the seed alone; the
framework takes them from pinned host memory, as it does a file's arrays.
"""
import math

import numpy as np
import torch

import gmkbe_b200 as G
from gmkbe_b200 import learned

DEV = "cuda"


# ----------------------------------------------------------------------------- graphs

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)
    return g


def _weights(n, gamma, mean, cap):
    """Expected degrees w_i ~ i^(-1/(gamma-1)) of the given mean, clipped at cap
    (0: none) and re-normalised."""
    w = torch.arange(1, n + 1, device=DEV, dtype=torch.float64) ** (-1.0 / (gamma - 1.0))
    w *= mean * n / w.sum()
    if cap:
        for _ in range(30):
            over = w >= cap
            if not bool((w > cap).any()):
                break
            w = torch.where(over, torch.full_like(w, cap), w)
            free = w[~over].sum()
            w = torch.where(over, w, w * ((mean * n - cap * over.sum()) / free))
        w = w.clamp(max=cap)
    return w


def _relabel(u, v):
    """Edge list (any ids) -> CSR in the converter's order: isolated vertices and
    parallel edges dropped, each side sorted by (d', id) with d' = degree - 2 on
    the left and degree - 1 on the right in wrapping 32-bit arithmetic (left
    vertices of degree 1 come last)."""
    nv = int(v.max()) + 1
    key = torch.unique(u * nv + v)
    u, v = key // nv, key % nv
    new, count = [], []
    for ids, minus in ((u, 2), (v, 1)):
        deg = torch.bincount(ids)
        wrapped = (deg - minus) & 0xFFFFFFFF
        wrapped[deg == 0] = 1 << 40
        rank = torch.empty_like(deg)
        rank[torch.argsort(wrapped, stable=True)] = torch.arange(deg.numel(), device=DEV)
        new.append(rank)
        count.append(int((deg > 0).sum()))
    nl, n = count[0], count[0] + count[1]
    a, b = new[0][u], new[1][v] + nl
    key = torch.sort(torch.cat([a * n + b, b * n + a])).values
    adj = (key % n).to(torch.int32)
    off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    return off, adj, n, nl


def _edges_er(gen, nu, nv, m):
    """m pairs drawn uniformly (parallel ones collapse)."""
    return (torch.randint(0, nu, (m,), generator=gen, device=DEV),
            torch.randint(0, nv, (m,), generator=gen, device=DEV))


def _edges_cl(gen, nu, nv, m, gamma, cap):
    out = []
    for n in (nu, nv):
        cdf = torch.cumsum(_weights(n, gamma, m / n, cap), 0)
        r = torch.rand(m, generator=gen, device=DEV, dtype=torch.float64) * cdf[-1]
        out.append(torch.searchsorted(cdf, r).clamp(max=n - 1))
    return out


def _graph(case, seed):
    """The case's graph as host CSR (pinned offsets and ids), n, n_left."""
    gen = _generator(seed)
    if case["graph"] == "er":
        u, v = _edges_er(gen, case["nu"], case["nv"], case["edges"])
    else:
        u, v = _edges_cl(gen, case["nu"], case["nv"], case["edges"], case["gamma"], case["max_deg"])
    off, adj, n, nl = _relabel(u, v)
    if case.get("prefix_u"):
        # the subgraph induced by the first ids of each side (the low degrees)
        src = torch.repeat_interleave(torch.arange(nl, device=DEV), off[1:nl + 1] - off[:nl])
        dst = adj[:int(off[nl])].to(torch.int64)
        keep = (src < case["prefix_u"]) & (dst < nl + case["prefix_v"])
        off, adj, n, nl = _relabel(src[keep], dst[keep] - nl)
    return _to_host(off), _to_host(adj), n, nl


def _to_host(x):
    h = torch.empty(x.numel(), dtype=torch.int32, pin_memory=True)
    h.copy_(x.to(torch.int32))
    return h.numpy().view(np.uint32)


def _er(name, kind, nu, nv, edges, k, **more):
    return dict(name=name, kind=kind, graph="er", nu=nu, nv=nv, edges=edges, k=k, **more)


def _cl(name, kind, nu, nv, edges, gamma, max_deg, k, **more):
    return dict(name=name, kind=kind, graph="cl", nu=nu, nv=nv, edges=edges, gamma=gamma,
                max_deg=max_deg, k=k, **more)


# ----------------------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call: a social network of the size of 18 women and 14 events; launches,
        # latency and the spread of one small search over the GPU count
        _er("social_k1", "enumerate", 18, 14, 110, 1),
        # the same network with the largest k in use: a deep tree from a tiny graph
        _er("social_k3", "enumerate", 18, 14, 110, 3),
        # a small sparse graph, complete at k = 2
        _er("er60_k2", "enumerate", 60, 60, 180, 2),
        # a dense-ish random graph, complete at k = 1 (degree 10 on both sides)
        _er("er200_k1", "enumerate", 200, 200, 2050, 1),
        # the low-degree part of a power-law graph, complete: thousands of roots, tiny subtrees
        _cl("cl100k_prefix_k1", "enumerate", 100_000, 300_000, 3_000_000, 2.2, 0, 1,
            prefix_u=20_000, prefix_v=60_000),
        # one request of a service that keeps the model: host CSR in, the learned schedule
        _cl("cl20k_prefix_request_k1", "end_to_end", 20_000, 50_000, 500_000, 2.1, 2000, 1,
            prefix_u=5_000, prefix_v=12_000),
        # the first million of a mid-sized power-law graph that is resident
        _cl("cl20k_first_million_k1", "limited", 20_000, 50_000, 500_000, 2.1, 2000, 1,
            limit=1_000_000),
        # what the command line tool does with its default limit: load, enumerate, release
        _cl("cl100k_load_limit_k2", "load_limited", 100_000, 300_000, 3_000_000, 2.2, 0, 2,
            limit=10_000_000),
        # the largest: 12 M edges, 10^8 results
        _cl("cl500k_limit_k1", "limited", 500_000, 1_000_000, 20_000_000, 2.0, 0, 1,
            limit=100_000_000),
        # many uneven graphs, each with its own k, in one call
        dict(name="batch64", kind="batch", graphs=64, side_lo=6, side_hi=40, deg_lo=1.5, deg_hi=3.0),
        # the sets themselves, sorted, as a program that goes on with them takes them
        _er("er30_records_k1", "records", 30, 30, 155, 1),
        # one gradient of the subtree-size model over a training set of the shipped model's size
        dict(name="model_gradient", kind="gradient", samples=33_738),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["er_k1", "er_k2", "er_k3", "prefix_k1", "prefix_k2", "request", "limited",
                       "limited", "load_limited", "batch", "records", "gradient"])
    if kind in ("er_k1", "er_k2", "er_k3", "records"):
        k = {"er_k1": 1, "er_k2": 2, "er_k3": 3, "records": rng.choice([1, 1, 2])}[kind]
        hi = {"er_k1": 400, "er_k2": 60, "er_k3": 20, "records": 40 if k == 1 else 14}[kind]
        nu, nv = _log_uniform(rng, 8, hi), _log_uniform(rng, 8, hi)
        deg = rng.uniform(2.0, {1: 10.0, 2: 4.0, 3: 4.0}[k] if kind != "records" else 4.0)
        edges = max(4, int(min(deg, 0.5 * min(nu, nv)) * math.sqrt(nu * nv)))
        return _er("", "records" if kind == "records" else "enumerate", nu, nv, edges, k) | {"name": "er"}
    if kind in ("prefix_k1", "request"):
        # 10^3 to 4 10^3 vertices of degree 1 to 2 remain, or a few hundred
        part = rng.uniform(0.06, 0.2)
        return _cl("prefix", "enumerate" if kind == "prefix_k1" else "end_to_end", 100_000, 300_000,
                   3_000_000, 2.2, rng.choice([0, 3000]), 1, prefix_u=int(100_000 * part),
                   prefix_v=int(300_000 * part * rng.uniform(0.8, 1.0)))
    if kind == "prefix_k2":
        part = rng.uniform(0.008, 0.036)
        return _cl("prefix", "enumerate", 500_000, 1_000_000, 20_000_000, 2.0, 0, 2,
                   prefix_u=int(500_000 * part), prefix_v=int(1_000_000 * part))
    if kind in ("limited", "load_limited"):
        nu = _log_uniform(rng, 5_000, 500_000)
        nv = int(nu * rng.uniform(1.5, 3.0))
        return _cl("limited", kind, nu, nv, int(nu * rng.uniform(10, 40)), rng.uniform(2.0, 2.2),
                   rng.choice([0, 2000]), rng.choice([1, 1, 2]),
                   limit=_log_uniform(rng, 100_000, 10_000_000))
    if kind == "batch":
        return dict(name="batch", kind="batch", graphs=_log_uniform(rng, 4, 64), side_lo=6,
                    side_hi=rng.randint(16, 40), deg_lo=1.5, deg_hi=rng.uniform(2.0, 3.0))
    return dict(name="gradient", kind="gradient", samples=_log_uniform(rng, 200, 34_000))


def _batch_graphs(case, seed):
    """The batch's graphs and their k: sides log-uniform, every other one
    Chung-Lu; the larger ones (over 20 vertices on a side) at k = 1 or 2."""
    import random
    rng = random.Random(seed)
    out = []
    for i in range(case["graphs"]):
        nu = _log_uniform(rng, case["side_lo"], case["side_hi"])
        nv = _log_uniform(rng, case["side_lo"], case["side_hi"])
        edges = max(3, int(rng.uniform(case["deg_lo"], case["deg_hi"]) * min(nu, nv)))
        k = rng.randint(1, 3 if max(nu, nv) <= 20 else 2)
        one = dict(graph="er" if i % 2 == 0 else "cl", nu=nu, nv=nv, edges=edges, gamma=2.1, max_deg=0)
        out.append((_graph(one, seed * 1000 + i), k))
    return out


def _samples(case, seed):
    """Features of the scale that root_features gives (log1p of counts) and
    targets of the scale of log1p(search nodes)."""
    gen = _generator(seed)
    n = case["samples"]
    top = torch.tensor([0.7, 0.0, 6.0, 11.0, 11.0, 11.0, 9.0, 7.0, 4.0, 6.0, 11.0, 11.0, 9.0, 9.0, 4.0,
                        2.0], device=DEV)
    x = torch.rand((n, 16), generator=gen, device=DEV) * top
    y = 0.6 * x[:, 2] + 0.5 * x[:, 12] + 0.3 * torch.randn(n, generator=gen, device=DEV) + 1.0
    return x.cpu().numpy(), y.cpu().numpy()


# ----------------------------------------------------------------------------- running them

def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "gradient":
        state["x"], state["y"] = _samples(case, seed)
        state["model"] = learned.load_default()
    elif kind == "batch":
        pairs = _batch_graphs(case, seed)
        state["graphs"] = [G.Graph.from_csr(*csr) for csr, _ in pairs]
        state["ks"] = [k for _, k in pairs]
    elif kind == "end_to_end":
        state["csr"] = _graph(case, seed)
        state["model"] = learned.load_default()
    elif kind == "load_limited":
        state["csr"] = _graph(case, seed)
    else:
        state["g"] = G.Graph.from_csr(*_graph(case, seed))
    return state


def _set(st):
    return {"count": st.count, "hash": np.array([st.hash_sum, st.hash_xor], np.uint64)}


def _identity(g):
    return np.array([g.fingerprint()], np.uint64)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "enumerate":
        return _set(state["g"].enumerate(k=case["k"]))
    if kind == "limited":
        # which results come first depends on the run, so a log holds the graph and the number
        st = state["g"].enumerate(k=case["k"], result_limit=case["limit"])
        return {"count": st.count, "graph": _identity(state["g"])}
    if kind == "load_limited":
        with G.Graph.from_csr(*state["csr"]) as g:
            st = g.enumerate(k=case["k"], result_limit=case["limit"])
            return {"count": st.count, "graph": _identity(g)}
    if kind == "end_to_end":
        with G.Graph.from_csr(*state["csr"]) as g:
            costs = learned.predicted_costs(state["model"], g, case["k"])
            st = g.enumerate(k=case["k"], schedule="ordered", task_cost=costs)
        padded = np.zeros(case["prefix_u"], np.float32)   # one length for all seeds
        padded[:costs.size] = costs
        return {"costs": padded, **_set(st)}
    if kind == "batch":
        got = G.enumerate_batch(state["graphs"], state["ks"])
        return {"counts": np.array([s.count for s in got], np.int64),
                "hashes": np.array([[s.hash_sum, s.hash_xor] for s in got], np.uint64)}
    if kind == "records":
        sets = sorted(state["g"].enumerate(k=case["k"], collect=True).results)
        # flat arrays of one length for all seeds: up to 20 (400) sets a vertex pair at k = 1 (2)
        room = (20 if case["k"] == 1 else 400) * case["nu"] * case["nv"]
        sizes, ids = np.zeros((room, 2), np.int32), np.zeros(16 * room, np.int32)
        sizes[:len(sets)] = [(len(x), len(y)) for x, y in sets]
        flat = [v for x, y in sets for v in x + y]
        ids[:len(flat)] = flat
        return {"sizes": sizes, "ids": ids}
    grad, loss = state["model"].gradient(state["x"], state["y"])
    return {"grad": grad, "loss": loss}


def work(case):
    """The bytes of the inputs (one graph of the case stands for all) read once and
    of the outputs written once; the gradient also has its multiply-adds.  A search has no fixed operation count
    that could be known beforehand."""
    kind = case["kind"]
    if kind == "gradient":
        n = case["samples"]
        return {"bytes": n * 17 * 4 + 2 * 5313 * 4, "flops": 6.0 * n * (16 * 64 + 64 * 64 + 64)}
    graphs = [csr for csr, _ in _batch_graphs(case, 0)] if kind == "batch" else [_graph(case, 0)]
    return {"bytes": sum(4 * (off.size + adj.size) + 24 for off, adj, _, _ in graphs), "flops": 0}


# ----------------------------------------------------------------------------- in 64 bits

def _unpack(params):
    """W1 b1 W2 b2 W3 b3 of the 16-64-64-1 model, rounded to FP16 as it runs."""
    p = torch.from_numpy(params).to(DEV).to(torch.float16).to(torch.float64)
    cut = [1024, 64, 4096, 64, 64, 1]
    w1, b1, w2, b2, w3, b3 = torch.split(p, cut)
    return w1.view(64, 16), b1, w2.view(64, 64), b2, w3, b3


def _forward(w, x):
    w1, b1, w2, b2, w3, b3 = w
    h = torch.relu(x @ w1.T + b1)
    h = torch.relu(h @ w2.T + b2)
    return h @ w3 + b3


def _root_features(csr, k):
    """The 16 features of every root, rounded to FP16 as the model reads them."""
    off, adj, n, nl = csr
    off = torch.from_numpy(off.astype(np.int64)).to(DEV)
    adj = torch.from_numpy(adj.astype(np.int64)).to(DEV)
    deg = off[1:] - off[:-1]
    d = deg[:nl]
    x = torch.repeat_interleave(torch.arange(nl, device=DEV), d)
    y = adj[:int(off[nl])]
    # rank of x in y's row: rows of V are sorted by id
    order = torch.argsort(y * n + x)
    rank = torch.empty_like(x)
    rank[order] = torch.arange(x.numel(), device=DEV) - (off[y[order]] - off[nl])
    dy = deg[y]
    above = dy - rank - 1

    def per_root(v, reduce, start):
        out = torch.full((nl,), start, dtype=torch.int64, device=DEV)
        return out.scatter_reduce(0, x, v, reduce)

    total = per_root(dy, "sum", 0)
    ids = torch.arange(nl, device=DEV)
    bucket = torch.floor(torch.log2(torch.clamp(d, min=1).double())) + 1
    nv = n - nl
    cols = [torch.full_like(d, k), torch.zeros_like(d), d, nv - d, nl - 1 - ids, ids, total,
            per_root(dy, "amax", 0), per_root(dy, "amin", 1 << 40), total / torch.clamp(d, min=1),
            torch.full_like(d, nv), torch.full_like(d, nl), per_root(above, "sum", 0),
            per_root(rank, "sum", 0), per_root((dy <= k + 1).long(), "sum", 0), bucket]
    return torch.stack([torch.log1p(c.double()) for c in cols], 1).half().double()


def exact(case, seed):
    if case["kind"] not in ("gradient", "end_to_end"):
        return None
    params = np.load("gmkbe_b200/models/subtree.npy")
    w = [t.clone().requires_grad_(True) for t in _unpack(params)]
    if case["kind"] == "end_to_end":
        pred = _forward(w, _root_features(_graph(case, seed), case["k"])).detach()
        costs = torch.zeros(case["prefix_u"], dtype=torch.float64, device=DEV)
        costs[:pred.numel()] = torch.expm1(pred.clamp(min=0.0))
        return {"costs": costs, "count": None, "hash": None}
    x, y = _samples(case, seed)
    x = torch.from_numpy(x).to(DEV).half().double()
    loss = torch.mean((_forward(w, x) - torch.from_numpy(y).to(DEV).double()) ** 2)
    loss.backward()
    return {"grad": torch.cat([t.grad.reshape(-1) for t in w]), "loss": loss.detach()}
