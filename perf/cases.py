"""The workloads that the framework is timed on: Leiden runs on resident graphs
from a few hundred to four million nodes, batched runs (many graphs, a
resolution x seed sweep), the Gaussian kNN graph builder, graph construction
with modularity and aggregation, and the learned warm start.

Each workload is a dict; `prepare` makes what a user's program has in hand,
`run` is one pass through the public entry points, `exact` is the same result
from plain 64-bit torch where a result is a computed number.

Inputs are drawn on the GPU from the seed alone. Shapes are those of the
benchmark: Gaussian mixtures of 30 or 50 dimensions, their kNN graphs, and
planted partitions.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "single-clustering_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import sc_gpu  # noqa: E402
from sc_gpu.learned import EdgeMlp  # noqa: E402

DEV = "cuda"


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # a handful of cells or a club-sized network: the latency of one small call
        {"name": "leiden_300", "kind": "leiden", "graph": "planted", "n": 300, "blocks": 6, "intra": 6, "inter": 2,
         "objective": "rb", "resolution": 1.0, "refine": True},
        # plain Leiden on the 20,000-node planted partition of the benchmark
        {"name": "leiden_20k", "kind": "leiden", "graph": "planted", "n": 20_000, "blocks": 40, "intra": 12,
         "inter": 3, "objective": "rb", "resolution": 1.0, "refine": True},
        # CPM on the kNN graph of a single-cell sized data set (200,000 x 50, k = 15)
        {"name": "leiden_cpm_200k", "kind": "leiden", "graph": "knn", "n": 200_000, "d": 50, "k": 15,
         "components": 30, "objective": "cpm", "resolution": 0.05, "refine": True},
        # the headline: RB on the kNN graph of an atlas of four million points
        {"name": "leiden_4m", "kind": "leiden", "graph": "knn", "n": 4_000_000, "d": 30, "k": 10, "components": 100,
         "objective": "rb", "resolution": 1.0, "refine": True},
        # many independent uneven graphs in one batched call
        {"name": "many_graphs", "kind": "many", "count": 96, "n_lo": 100, "n_hi": 50_000},
        # a resolution x seed sweep with warm starts on one graph, concurrent streams
        {"name": "sweep_200k", "kind": "sweep", "n": 200_000, "d": 50, "k": 15, "components": 30, "resolutions": 8,
         "seeds": 2, "streams": 16, "split": 2},
        # the kNN graph of a small data set, the reference's default sigma and emission
        {"name": "knn_5k", "kind": "knn", "n": 5003, "d": 30, "k": 10, "components": 12, "precision": "bf16",
         "sigma": "median", "sym": "lower"},
        # the kNN graph of a single-cell sized data set, built and kept for Leiden
        {"name": "knn_200k", "kind": "knn", "n": 200_000, "d": 50, "k": 15, "components": 30, "precision": "bf16",
         "sigma": "kth", "sym": "union"},
        # the input of the benchmark's 1M-point sweep
        {"name": "knn_1m", "kind": "knn", "n": 1_000_000, "d": 50, "k": 15, "components": 60, "precision": "bf16",
         "sigma": "kth", "sym": "union"},
        # candidates by exact FP32 differences
        {"name": "knn_fp32_30k", "kind": "knn", "n": 30_011, "d": 50, "k": 15, "components": 30, "precision": "fp32",
         "sigma": "kth", "sym": "union"},
        # a graph handed over from the host, the score of labels found elsewhere, and the graph of their groups
        {"name": "handover_500k", "kind": "handover", "n": 500_000, "blocks": 60, "intra": 7, "inter": 1},
        # the learned warm start: a few training epochs on a found partition, then a proposal and the run from it
        {"name": "warm_100k", "kind": "warm", "n": 100_000, "d": 50, "k": 15, "components": 50, "epochs": 4},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["leiden_planted", "leiden_planted", "leiden_knn", "leiden_knn", "many", "sweep", "knn", "knn",
                       "knn_fp32", "handover", "warm"])
    if kind == "leiden_planted":
        n = _log_uniform(rng, 100, 50_000)
        objective = rng.choice(["rb", "rb", "cpm"])
        return {"kind": "leiden", "graph": "planted", "n": n, "blocks": max(2, min(rng.randint(5, 200), n // 5)),
                "intra": rng.randint(4, 12), "inter": rng.randint(1, 3), "objective": objective,
                "resolution": round(rng.uniform(0.5, 2.0), 3) if objective == "rb" else round(rng.uniform(0.02, 0.1), 4),
                "refine": rng.random() < 0.85}
    if kind == "leiden_knn":
        objective = rng.choice(["rb", "rb", "cpm"])
        return {"kind": "leiden", "graph": "knn", "n": _log_uniform(rng, 5_000, 2_000_000), "d": rng.choice([30, 50]),
                "k": rng.choice([10, 15]), "components": rng.randint(10, 100), "objective": objective,
                "resolution": round(rng.uniform(0.3, 2.0), 3) if objective == "rb" else round(rng.uniform(0.01, 0.1), 4),
                "refine": rng.random() < 0.85}
    if kind == "many":
        return {"kind": "many", "count": rng.randint(8, 96), "n_lo": 100, "n_hi": _log_uniform(rng, 2_000, 50_000)}
    if kind == "sweep":
        return {"kind": "sweep", "n": _log_uniform(rng, 10_000, 200_000), "d": rng.choice([30, 50]),
                "k": rng.choice([10, 15]), "components": rng.randint(10, 60), "resolutions": rng.randint(3, 8),
                "seeds": rng.randint(1, 3), "streams": rng.choice([4, 8, 16]), "split": rng.randint(1, 3)}
    if kind == "knn":
        option = rng.choice([("kth", "union"), ("kth", "union"), ("median", "lower")])
        return {"kind": "knn", "n": _log_uniform(rng, 1_000, 1_000_000), "d": rng.choice([7, 30, 50, 62]),
                "k": rng.randint(5, 15), "components": rng.randint(10, 60), "precision": "bf16", "sigma": option[0],
                "sym": option[1]}
    if kind == "knn_fp32":
        return {"kind": "knn", "n": _log_uniform(rng, 1_000, 60_000), "d": rng.choice([7, 30, 50, 62]),
                "k": rng.randint(5, 15), "components": rng.randint(8, 30), "precision": "fp32", "sigma": "kth",
                "sym": "union"}
    if kind == "handover":
        n = _log_uniform(rng, 2_000, 1_000_000)
        return {"kind": "handover", "n": n, "blocks": rng.randint(2, min(200, int(math.sqrt(n / 20)))),
                "intra": rng.randint(4, 10), "inter": rng.randint(1, 3)}
    return {"kind": "warm", "n": _log_uniform(rng, 10_000, 200_000), "d": 50, "k": 15,
            "components": rng.randint(10, 60), "epochs": rng.randint(2, 6)}


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _points(case, seed):
    """An isotropic Gaussian mixture on the device: centres ~ N(0, 4 I), sigma ~ U[0.7, 1.5],
    mixture weights ~ Dirichlet(1). Returns (points f32 (n, d), component of each point)."""
    g = _generator(seed)
    n, d, c = case["n"], case["d"], case["components"]
    centres = 2.0 * torch.randn(c, d, generator=g, device=DEV)
    sigma = 0.7 + 0.8 * torch.rand(c, generator=g, device=DEV)
    share = -torch.log(torch.rand(c, generator=g, device=DEV).clamp_min(1e-12))
    comp = torch.multinomial(share / share.sum(), n, replacement=True, generator=g)
    x = torch.randn(n, d, generator=g, device=DEV)
    x.mul_(sigma[comp][:, None]).add_(centres[comp])
    return x, comp


def _host_points(case, seed):
    x, comp = _points(case, seed)
    return x.cpu().numpy(), comp


def _knn_graph(case, seed):
    x, _ = _host_points(case, seed)
    return x, sc_gpu.knn_gaussian(x, case["k"], sigma=sc_gpu.SIGMA_KTH, sym=sc_gpu.SYM_UNION, build_graph=True).graph


def _planted_pairs(n, blocks, intra, inter, g):
    """Pairs of a planted partition: every node draws `intra` partners in its
    block and `inter` outside it. Returns (from, to, block of each node)."""
    per = max(n // blocks, 2)
    node = torch.arange(n, device=DEV)
    block = torch.clamp(node // per, max=blocks - 1)
    base = block * per
    size = torch.where(block == blocks - 1, n - base, torch.full_like(base, per))
    a = node.repeat_interleave(intra)
    off = 1 + (torch.rand(a.numel(), generator=g, device=DEV, dtype=torch.float64) * (size[a] - 1)).long()
    dst_a = base[a] + (a - base[a] + off) % size[a]
    b = node.repeat_interleave(inter)
    r = (torch.rand(b.numel(), generator=g, device=DEV, dtype=torch.float64) * (n - size[b])).long()
    dst_b = torch.where(r < base[b], r, r + size[b])
    return torch.cat([a, b]), torch.cat([dst_a, dst_b]), block


def _planted(n, blocks, intra, inter, g):
    """Edge arrays of a planted partition with shuffled node ids, weights U[0.5, 1.5]; pairs drawn twice stay in."""
    src, dst, _ = _planted_pairs(n, blocks, intra, inter, g)
    ids = torch.randperm(n, generator=g, device=DEV)
    src, dst = ids[src], ids[dst]
    w = (0.5 + torch.rand(src.numel(), generator=g, device=DEV)).double()
    return src.cpu().numpy().astype(np.uint64), dst.cpu().numpy().astype(np.uint64), w.cpu().numpy()


def _symmetric_csr(case, seed):
    """A planted partition with shuffled node ids as a symmetric CSR (every pair
    once, weights U[0.3, 1.0]) on the device: (ptrs, rows, nbrs, w, block of each node)."""
    g, n = _generator(seed), case["n"]
    src, dst, block = _planted_pairs(n, case["blocks"], case["intra"], case["inter"], g)
    ids = torch.randperm(n, generator=g, device=DEV)
    labels = torch.empty_like(block)
    labels[ids] = block
    src, dst = ids[src], ids[dst]
    pairs = (torch.minimum(src, dst) * n + torch.maximum(src, dst))[src != dst].unique()
    w = 0.3 + 0.7 * torch.rand(pairs.numel(), generator=g, device=DEV)
    lo, hi = pairs // n, pairs % n
    key, at = torch.cat([lo * n + hi, hi * n + lo]).sort()
    rows = key // n
    ptrs = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptrs[1:] = torch.bincount(rows, minlength=n).cumsum(0)
    return ptrs, rows, key % n, torch.cat([w, w])[at], labels


def _config(case, seed):
    objective = sc_gpu.Rb(case["resolution"]) if case["objective"] == "rb" else sc_gpu.Cpm(case["resolution"])
    return sc_gpu.LeidenConfig(objective=objective, seed=int(seed) & 0xFFFF, refine=case["refine"])


def _many_sizes(case):
    """(nodes, blocks, draws a node) of each graph: they belong to the case, the edges to the seed."""
    rng = np.random.Generator(np.random.PCG64(case["count"] + case["n_hi"]))
    n = np.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]), case["count"])).astype(np.int64)
    blocks = rng.integers(5, 201, case["count"])
    degree = rng.uniform(10.0, 30.0, case["count"])
    return [(int(a), int(max(2, min(b, a // 5))), d / 2.0) for a, b, d in zip(n, blocks, degree)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "leiden":
        if case["graph"] == "planted":
            e = _planted(case["n"], case["blocks"], case["intra"], case["inter"], _generator(seed))
            graph = sc_gpu.CSRNetwork.from_edge_arrays(case["n"], *e)
        else:
            graph = _knn_graph(case, seed)[1]
        return {"kind": kind, "graph": graph, "config": _config(case, seed)}
    if kind == "many":
        g = _generator(seed)
        graphs, configs = [], []
        for n, blocks, draws in _many_sizes(case):
            intra = max(1, int(round(0.8 * draws)))
            e = _planted(n, blocks, intra, max(0, int(round(draws)) - intra), g)
            graphs.append(sc_gpu.CSRNetwork.from_edge_arrays(n, *e))
            configs.append(sc_gpu.LeidenConfig(seed=int(seed) & 0xFFFF))
        return {"kind": kind, "graphs": graphs, "configs": configs}
    if kind == "sweep":
        graph = _knn_graph(case, seed)[1]
        return {"kind": kind, "graph": graph, "resolutions": np.geomspace(0.1, 3.0, case["resolutions"]).tolist(),
                "seeds": [(int(seed) + i) & 0xFFFF for i in range(case["seeds"])], "streams": case["streams"],
                "split": case["split"]}
    if kind == "knn":
        x, _ = _host_points(case, seed)
        return {"kind": kind, "x": x, "k": case["k"], **_knn_options(case)}
    if kind == "handover":
        ptrs, _, nbrs, w, labels = _symmetric_csr(case, seed)
        return {"kind": kind, "ptrs": ptrs.cpu().numpy().astype(np.uint64), "nbrs": nbrs.cpu().numpy().astype(np.uint32),
                "w": w.cpu().numpy(), "labels": labels.cpu().numpy().astype(np.uint64)}
    x, graph = _knn_graph(case, seed)
    graph.set_embedding(x)
    # the partitions found at the neighbouring resolutions, which the model reads and learns from
    found = [sc_gpu.leiden(graph, sc_gpu.LeidenConfig(objective=sc_gpu.Rb(g), seed=3)).labels()
             for g in (0.5, 1.0, 2.0)]
    return {"kind": kind, "graph": graph, "found": found, "epochs": case["epochs"], "seed": int(seed) & 0xFFFF}


def _knn_options(case):
    return {"precision": sc_gpu.KNN_FP32 if case["precision"] == "fp32" else sc_gpu.KNN_BF16,
            "sigma": sc_gpu.SIGMA_KTH if case["sigma"] == "kth" else sc_gpu.SIGMA_MEDIAN,
            "sym": sc_gpu.SYM_UNION if case["sym"] == "union" else sc_gpu.SYM_LOWER_ID}


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "leiden":
        c = sc_gpu.leiden(state["graph"], state["config"])
        return {"labels": c.labels(), "n_clusters": c.n_clusters()}
    if kind == "many":
        res = sc_gpu.leiden_batch(state["graphs"], state["configs"], union=True)
        return {"labels": np.concatenate([c.labels() for c in res]),
                "n_clusters": np.array([c.n_clusters() for c in res])}
    if kind == "sweep":
        res = sc_gpu.leiden_sweep(state["graph"], state["resolutions"], state["seeds"], warm_start=True,
                                  n_streams=state["streams"], split=state["split"])
        return {"labels": np.stack([res[key].labels() for key in sorted(res)])}
    if kind == "knn":
        r = sc_gpu.knn_gaussian(state["x"], state["k"], sigma=state["sigma"], sym=state["sym"],
                                precision=state["precision"], build_graph=True)
        # the number of entries differs from one data set to the next: the connectivities come as the row offsets and
        # every node's weight sum, which together with the lists determine them
        return {"index": r.index, "distances": r.distances, "ptrs": r.conn_ptrs, "strengths": r.graph.strengths()}
    if kind == "handover":
        g = sc_gpu.CSRNetwork.from_csr_parts(state["ptrs"], state["nbrs"], state["w"])
        q = sc_gpu.modularity(g, state["labels"], 1.0)
        a = g.aggregate(state["labels"])
        ptrs, nbrs, w = a.to_csr_parts()
        return {"modularity": q, "total": g.total_weight(), "strengths": g.strengths(), "ptrs": ptrs, "nbrs": nbrs,
                "w": w}
    low, mid, high = state["found"]
    model = EdgeMlp(seed=state["seed"])
    loss = model.train(state["graph"], mid, 1.0, epochs=state["epochs"], context=(low, high))
    start, count = model.propose(state["graph"], 0.8, context=(low, mid))
    c = sc_gpu.leiden_from(state["graph"], sc_gpu.LeidenConfig(objective=sc_gpu.Rb(0.8), seed=3, n_iterations=1), start)
    return {"loss": loss, "params": model.params(), "start": start, "count": count, "labels": c.labels()}


# ---------------------------------------------------------------- what a pass cannot do without
def _entries(case):
    """Stored entries of a case's graph: a union-symmetrised kNN list keeps about 1.7 per listed neighbour."""
    if "intra" in case:
        return 2 * case["n"] * (case["intra"] + case["inter"])
    return int(1.7 * case["n"] * case["k"])


def work(case):
    kind = case["kind"]
    if kind == "leiden":  # the graph once (8 bytes an entry), labels out
        return {"bytes": 8 * _entries(case) + 32 * case["n"], "flops": 2 * _entries(case)}
    if kind == "many":
        sizes = _many_sizes(case)
        return {"bytes": sum(8 * 2 * n * draws + 32 * n for n, _, draws in sizes),
                "flops": sum(4 * n * draws for n, _, draws in sizes)}
    if kind == "sweep":
        runs = case["resolutions"] * case["seeds"]
        return {"bytes": runs * (8 * _entries(case) + 32 * case["n"]), "flops": 2 * runs * _entries(case)}
    if kind == "knn":  # every point against its own mixture component (Dirichlet(1): 2 / (C + 1) of the points)
        n, k = case["n"], case["k"]
        return {"bytes": 4 * n * case["d"] + 8 * n * (k + 1) + 8 * n + 8 * int(1.7 * n * k),
                "flops": 2.0 * n * n * case["d"] * 2 / (case["components"] + 1)}
    if kind == "handover":
        return {"bytes": 8 * _entries(case) + 24 * case["n"], "flops": 4 * _entries(case)}
    edges = _entries(case) // 2  # forward, two backward products of a 15 x 128 x 1 network, then one forward
    return {"bytes": (case["epochs"] + 1) * 60 * edges, "flops": (3 * case["epochs"] + 1) * 2.0 * 16 * 128 * edges}


# ---------------------------------------------------------------- the same in 64 bits
def _exact_knn(x, k):
    """The k + 1 nearest points of every point, itself first: (index, distance) from 64-bit differences."""
    n = x.shape[0]
    x64 = x.double()
    nrm = (x64 * x64).sum(1)
    m = min(n, k + 9)
    index = torch.empty(n, k + 1, dtype=torch.int64, device=DEV)
    dist = torch.empty(n, k + 1, dtype=torch.float64, device=DEV)
    step = max(1, min(n, (1 << 28) // n))
    for s in range(0, n, step):
        q = x64[s:s + step]
        score = torch.addmm(nrm[None, :].expand(q.shape[0], n), q, x64.T, alpha=-2.0)
        cand = score.topk(m, dim=1, largest=False).indices
        d2 = (x64[cand] - q[:, None, :]).square().sum(2)
        d2[cand == torch.arange(s, s + q.shape[0], device=DEV)[:, None]] = -1.0  # itself first
        v, at = d2.sort(dim=1)
        index[s:s + step] = cand.gather(1, at)[:, : k + 1]
        dist[s:s + step] = v[:, : k + 1].clamp_min(0.0).sqrt()
    return index, dist


def _exact_strengths(index, dist, kth, union):
    """Every node's sum of connectivity weights."""
    n, k = index.shape[0], index.shape[1] - 1
    if kth:
        sigma = dist[:, -1]
    else:
        pos = (dist > 0).sum(1)
        ordered = torch.where(dist > 0, dist, torch.full_like(dist, math.inf)).sort(dim=1).values
        sigma = torch.where(pos > 0, ordered.gather(1, (pos // 2)[:, None])[:, 0], torch.ones_like(dist[:, 0]))
    i = torch.arange(n, device=DEV).repeat_interleave(k)
    j = index[:, 1:].reshape(-1)
    d = dist[:, 1:].reshape(-1)
    den = sigma[i].square() + sigma[j].square()
    w = (2 * sigma[i] * sigma[j] / den).sqrt() * torch.exp(-d.square() / den)
    keep = (w > 1e-14) & ((i != j) if union else (i <= j))
    i, j, w = i[keep], j[keep], w[keep]
    key, at = torch.cat([i * n + j, j * n + i]).unique(return_inverse=True)
    entry = torch.zeros(key.numel(), dtype=torch.float64, device=DEV)
    entry[at] = torch.cat([w, w])
    return torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, key // n, entry)


def exact(case, seed):
    kind = case["kind"]
    if kind == "knn":
        if case["n"] > 250_000:
            return None
        x, _ = _points(case, seed)
        index, dist = _exact_knn(x, case["k"])
        return {"index": None, "distances": dist, "ptrs": None,
                "strengths": _exact_strengths(index, dist, case["sigma"] == "kth", case["sym"] == "union")}
    if kind == "handover":
        _, row, nbr, w, labels = _symmetric_csr(case, seed)
        n, w = case["n"], w.double()
        strength = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, row, w)
        lab = labels.unique(return_inverse=True)[1]
        groups = int(lab.max()) + 1
        two_m = strength.sum()
        k_c = torch.zeros(groups, dtype=torch.float64, device=DEV).index_add_(0, lab, strength)
        sums = torch.zeros(groups * groups, dtype=torch.float64, device=DEV)
        sums.index_add_(0, lab[row] * groups + lab[nbr], w)
        sums = sums.view(groups, groups)
        q = (sums.diagonal() / two_m - (k_c / two_m).square()).sum()
        sums.diagonal().mul_(0.5)  # an edge inside a group counts once
        return {"modularity": float(q), "total": float(0.5 * two_m), "strengths": strength, "ptrs": None, "nbrs": None,
                "w": sums[sums > 0]}
    return None
