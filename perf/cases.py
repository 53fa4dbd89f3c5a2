"""The calls whose time matters to a user of plato_b200, one pass each.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` builds what a program holds before the call (a graph
resident in HBM, seed sets, a root, a server), ``run(state)`` makes the call
through the package's public entry points, ``work(case)`` counts what the call
cannot do without and ``exact(case, seed)`` gives its results in 64 bits.

Graphs are made on the GPU from the seed alone: RMAT edge lists (a, b, c, d =
.57, .19, .19, .05, self-loops and duplicates removed, ids compacted into a
vertex count that the case alone fixes, odd as often as not, with a few
isolated vertices at its end) and uniform random edge lists of any vertex
count.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import plato_b200 as pb

DAMPING = 0.85


def listed():
    return [
        # A small graph queried often: the call is launches and latency.
        {"name": "pagerank_rmat10", "kind": "pagerank", "graph": "rmat", "scale": 10, "ef": 16,
         "iteration": 20, "eps": 0.0, "device": False},
        # The benchmark's small configuration: RMAT 16, 100 epochs, ranks on the host.
        {"name": "pagerank_rmat16", "kind": "pagerank", "graph": "rmat", "scale": 16, "ef": 16,
         "iteration": 100, "eps": 0.0, "device": False},
        # The default options (100 epochs, eps 0.001) on a graph without hubs.
        {"name": "pagerank_uniform1m", "kind": "pagerank", "graph": "uniform", "vertices": 1000003, "ef": 16,
         "iteration": 100, "eps": 0.001, "device": False},
        # The headline configuration: RMAT 24, 20 epochs, ranks in device memory.
        {"name": "pagerank_rmat24", "kind": "pagerank", "graph": "rmat", "scale": 24, "ef": 16,
         "iteration": 20, "eps": 0.0, "device": True},
        # Weighted edges, the default options.
        {"name": "wpagerank_rmat21", "kind": "wpagerank", "graph": "rmat", "scale": 21, "ef": 16,
         "iteration": 100, "eps": 0.001},
        # One personalized query, push epochs first, to delta < 1e-7.
        {"name": "ppr_rmat22", "kind": "ppr", "graph": "rmat", "scale": 22, "ef": 16,
         "iteration": 100, "eps": 1e-7, "pushpull": True},
        # Seed selection by inverse PageRank in 64 bits, then trust.
        {"name": "trustrank_rmat20", "kind": "trustrank", "graph": "rmat", "scale": 20, "ef": 16,
         "iteration": 100, "eps": 0.001, "seed_num": 100},
        # A batch of queries in one call, Zipf seed sets, top-100 each.
        {"name": "ppr_batch64_rmat21", "kind": "batch", "graph": "rmat", "scale": 21, "ef": 16,
         "queries": 64, "k_tile": 64, "max_seeds": 32, "topk": 100, "eps": 1e-6, "iteration": 300},
        # A server with a small HBM budget: eight slots, two generations of requests.
        {"name": "server8_rmat19", "kind": "server", "graph": "rmat", "scale": 19, "ef": 16,
         "queries": 16, "slots": 8, "max_seeds": 64, "topk": 100, "eps": 1e-6, "iteration": 200},
        # One search over a symmetrised graph, levels on the host.
        {"name": "bfs_rmat22", "kind": "bfs", "graph": "rmat", "scale": 22, "ef": 16},
        # Labels and summary of the components of a symmetrised graph.
        {"name": "cc_rmat21", "kind": "cc", "graph": "rmat", "scale": 21, "ef": 16},
        # Average distance of a symmetrised graph, 64-byte registers.
        {"name": "hyperanf_rmat20", "kind": "hyperanf", "graph": "rmat", "scale": 20, "ef": 16,
         "iteration": 20, "bits": 6},
    ]


def draw(rng):
    kind = rng.choice(["pagerank", "pagerank", "wpagerank", "ppr", "trustrank", "batch", "server", "bfs", "cc",
                       "hyperanf"])
    top = {"pagerank": 23, "wpagerank": 21, "ppr": 22, "trustrank": 20, "batch": 20, "server": 19, "bfs": 22,
           "cc": 21, "hyperanf": 20}[kind]
    case = {"kind": kind, "ef": rng.randint(6, 20)}
    if rng.random() < 0.3:
        case["graph"] = "uniform"
        case["vertices"] = int(2 ** rng.uniform(10, min(top - 1, 20)))
    else:
        case["graph"] = "rmat"
        case["scale"] = rng.randint(10, top)
    if kind == "pagerank":
        if rng.random() < 0.5:
            case.update(iteration=rng.randint(5, 40), eps=0.0)
        else:
            case.update(iteration=100, eps=rng.choice([0.001, 0.0001]))
        case["device"] = rng.random() < 0.5
    elif kind == "wpagerank":
        case.update(iteration=100, eps=rng.choice([0.0, 0.001]))
    elif kind == "ppr":
        case.update(iteration=100, eps=rng.choice([1e-6, 1e-7]), pushpull=rng.random() < 0.5)
    elif kind == "trustrank":
        case.update(iteration=100, eps=0.001, seed_num=rng.randint(10, 200))
    elif kind == "batch":
        case.update(queries=rng.randint(2, 96), k_tile=rng.choice([8, 16, 32, 64]), max_seeds=32,
                    topk=rng.choice([10, 100]), eps=1e-6, iteration=300)
    elif kind == "server":
        case.update(queries=rng.randint(4, 20), slots=rng.randint(2, 8), max_seeds=64, topk=100, eps=1e-6,
                    iteration=200)
    elif kind == "hyperanf":
        case.update(iteration=20, bits=rng.randint(4, 8))
    return case


# -- inputs ------------------------------------------------------------------

def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _edges(case, seed):
    """(V, src, dst) on the GPU, int64, sorted by (src, dst)."""
    gen = _generator(seed, 1)
    if case["graph"] == "uniform":
        n, m = case["vertices"], case["vertices"] * case["ef"]
        src = torch.randint(n, (m,), generator=gen, device="cuda")
        dst = torch.randint(n, (m,), generator=gen, device="cuda")
    else:
        n, m = 1 << case["scale"], case["ef"] << case["scale"]
        src = torch.zeros(m, dtype=torch.int32, device="cuda")
        dst = torch.zeros(m, dtype=torch.int32, device="cuda")
        for _ in range(case["scale"]):
            r = torch.rand(m, generator=gen, device="cuda")
            down = r >= 0.57 + 0.19
            right = ((r >= 0.57) & ~down) | (r >= 0.57 + 0.19 + 0.19)
            src.mul_(2).add_(down)
            dst.mul_(2).add_(right)
        del r, down, right
        src, dst = src.long(), dst.long()
    if _symmetric(case):
        src, dst = torch.minimum(src, dst), torch.maximum(src, dst)
    key = (src * n + dst)[src != dst]
    del src, dst
    key = torch.sort(key).values
    fresh = torch.ones_like(key, dtype=torch.bool)
    fresh[1:] = key[1:] != key[:-1]
    key = key[fresh]
    del fresh
    src, dst = key // n, key % n
    del key
    vertices = _size(case)[0]
    if case["graph"] == "rmat":
        there = torch.zeros(n, dtype=torch.bool, device="cuda")
        there[src] = True
        there[dst] = True
        number = torch.cumsum(there, 0) - 1
        src, dst = number[src], number[dst]
        if int(there.sum()) > vertices:  # as good as never: the ids past the end leave with their edges
            kept = (src < vertices) & (dst < vertices)
            src, dst = src[kept], dst[kept]
    return vertices, src, dst


def _symmetric(case):
    return case["kind"] in ("bfs", "cc", "hyperanf")


def _weights(seed, edges):
    return torch.rand(edges, generator=_generator(seed, 2), device="cuda", dtype=torch.float64) * 9.9 + 0.1


def _picks(case, seed, src, dst):
    """Vertices with out-edges (both ends of a symmetrised list), and the generator that picks among them."""
    ends = torch.unique(torch.cat([src, dst]) if _symmetric(case) else src)
    return ends.cpu().numpy(), np.random.default_rng(seed)


def _seed_sets(case, seed, src, dst):
    """Zipf(1.5) sizes clipped to max_seeds, members uniform among vertices with out-edges."""
    ends, rng = _picks(case, seed, src, dst)
    sizes = np.minimum(rng.zipf(1.5, case["queries"]), min(case["max_seeds"], ends.size))
    return [rng.choice(ends, int(n), replace=False).astype(np.uint32) for n in sizes]


def _root(case, seed, src, dst):
    ends, rng = _picks(case, seed, src, dst)
    return int(rng.choice(ends))


def _host(t):
    return t.to(torch.int32).cpu().numpy().view(np.uint32)


def prepare(case, seed):
    kind = case["kind"]
    vertices, src, dst = _edges(case, seed)
    weights = _weights(seed, src.numel()).cpu().numpy() if kind == "wpagerank" else None
    graph = pb.Graph(vertices, _host(src), _host(dst), is_directed=not _symmetric(case), weights=weights)
    state = {"case": case, "graph": graph}
    if kind == "pagerank" and case["device"]:
        state["ranks"] = torch.empty(vertices, dtype=torch.float32, device="cuda")
    elif kind in ("ppr", "bfs"):
        state["root"] = _root(case, seed, src, dst)
    elif kind in ("batch", "server"):
        state["sets"] = _seed_sets(case, seed, src, dst)
    if kind == "server":
        state["server"] = pb.PPRServer(graph, max_slots=case["slots"], max_iterations=case["iteration"],
                                       eps=case["eps"], topk=case["topk"])
    return state


# -- one pass ------------------------------------------------------------------

def run(state):
    case, graph = state["case"], state["graph"]
    kind = case["kind"]
    if kind == "pagerank":
        if case["device"]:
            stream = torch.cuda.current_stream().cuda_stream
            graph.pagerank_device(state["ranks"].data_ptr(), case["iteration"], DAMPING, case["eps"], stream)
            return state["ranks"]
        return graph.pagerank(case["iteration"], DAMPING, case["eps"])[0]
    if kind == "wpagerank":
        return graph.weighted_pagerank(case["iteration"], DAMPING, case["eps"])[0]
    if kind == "ppr":
        mode = pb.PLATO_PPR_PUSHPULL if case["pushpull"] else pb.PLATO_PPR_PULL
        return graph.personalized_pagerank(state["root"], case["iteration"], DAMPING, case["eps"], mode)[0]
    if kind == "trustrank":
        ranks, seeds, _ = graph.trustrank(None, case["iteration"], DAMPING, case["seed_num"], 0, case["eps"])
        return {"ranks": ranks, "seeds": seeds}
    if kind == "batch":
        out = graph.ppr_batch(state["sets"], case["iteration"], DAMPING, case["eps"], topk=case["topk"],
                              k_tile=case["k_tile"])
        return {k: out[k] for k in ("iterations", "topk_ids", "topk_vals")}
    if kind == "server":
        return _serve(state["server"], state["sets"])
    if kind == "bfs":
        return graph.bfs(state["root"], parents=False)[0]
    if kind == "cc":
        labels, summary, _ = graph.connected_components()
        return {"labels": labels, "summary": summary}
    distance, anfs, _, _ = graph.hyperanf(case["iteration"], case["bits"])
    # the series ends when it stops growing: its last value stands for the epochs that did not run
    return {"distance": distance, "anfs": np.pad(anfs, (0, case["iteration"] + 1 - anfs.size), mode="edge")}


def _serve(server, sets):
    """Every request submitted, the server stepped until all are answered; answers in the order of submission."""
    order = {server.submit(s): i for i, s in enumerate(sets)}
    ids = np.empty((len(sets), server.topk), dtype=np.uint32)
    vals = np.empty((len(sets), server.topk), dtype=np.float32)
    iterations = np.empty(len(sets), dtype=np.uint32)
    left = len(sets)
    while left:
        server.step()
        while (answer := server.poll()) is not None:
            i = order[answer[0]]
            ids[i], vals[i], iterations[i] = answer[1:]
            left -= 1
    return {"iterations": iterations, "topk_ids": ids, "topk_vals": vals}


# -- what a pass cannot do without ---------------------------------------------

def _size(case):
    """Vertices, and stored edges to within a few per cent, without making the graph.  An id of an RMAT list with k
    one bits is an end of an edge with probability 2 * .24^k * .76^(scale - k); two standard deviations and more
    above the expected count of ids that occur, no list needs another vertex."""
    if case["graph"] == "uniform":
        vertices, edges = case["vertices"], case["vertices"] * case["ef"]
    else:
        scale, m = case["scale"], case["ef"] << case["scale"]
        occur = sum(math.comb(scale, k) * -math.expm1(-2 * m * 0.24 ** k * 0.76 ** (scale - k))
                    for k in range(scale + 1))
        vertices = int(occur + 2 * math.sqrt(occur))
        edges = int((1 - 0.35 * 2 ** (-scale / 8)) * m)
    return vertices, edges * (2 if _symmetric(case) else 1)


def work(case):
    """Epochs of an iterative call read the adjacency once and the state once and write the state once;
    a traversal reads its offsets and one in-edge of each vertex and writes its result."""
    kind, (v, e) = case["kind"], _size(case)
    if kind == "bfs":
        return {"bytes": 16 * v, "flops": v}
    if kind == "cc":
        return {"bytes": 2 * (4 * e + 8 * v) + 8 * v, "flops": 2 * e}
    if kind == "hyperanf":
        m = 1 << case["bits"]
        return {"bytes": 3 * (4 * e + 8 * v + 2 * m * v), "flops": 3 * m * e}
    epochs = case["iteration"]
    if case["eps"] > 0:
        mass = v if kind in ("pagerank", "wpagerank") else 1
        epochs = min(epochs, max(3, int(0.6 * math.log(case["eps"] / mass) / math.log(DAMPING))))
    columns = case.get("queries", 1)
    if kind == "trustrank":  # the selection's 64-bit epochs before the trust epochs
        chosen = min(100, max(3, int(0.6 * math.log(0.001 / v) / math.log(DAMPING))))
        return {"bytes": chosen * (4 * e + 28 * v) + epochs * (4 * e + 20 * v), "flops": (chosen + epochs) * (e + 3 * v)}
    edge = 8 if kind == "wpagerank" else 4
    return {"bytes": epochs * (edge * e + 12 * v + 8 * v * columns), "flops": epochs * (e + 3 * v) * columns}


# -- the same in 64 bits ---------------------------------------------------------

class _Pull:
    """y[dst] = sum over in-edges of value * x[src], in 64 bits."""

    def __init__(self, vertices, src, dst, values=None):
        order = torch.argsort(dst, stable=True)
        heads = torch.zeros(vertices + 1, dtype=torch.int64, device="cuda")
        heads[1:] = torch.cumsum(torch.bincount(dst, minlength=vertices), 0)
        if values is None:
            values = torch.ones(src.numel(), dtype=torch.float64, device="cuda")
        else:
            values = values[order]
        self.matrix = torch.sparse_csr_tensor(heads, src[order], values, size=(vertices, vertices))

    def __call__(self, x):
        return self.matrix @ x


def _epochs(pull, degree, x, teleport, iteration, eps):
    """Columns x (V x K) of rank / out-degree through the epochs; each column leaves with its own final epoch."""
    safe = degree.clamp(min=1)[:, None]
    live = torch.ones(x.shape[1], dtype=torch.bool, device="cuda")
    last = torch.full((x.shape[1],), iteration == 1, device="cuda")
    ranks = torch.zeros_like(x)
    for epoch in range(iteration):
        r = teleport + DAMPING * pull(x)
        ranks = torch.where((live & last)[None, :], r, ranks)
        live = live & ~last
        if not bool(live.any()):
            break
        y = r / safe
        delta = ((y - x).abs() * safe).sum(0)
        x = y
        last = (delta < eps) | (epoch + 1 >= iteration - 1)
    return ranks


def _seeded(pull, degree, vertices, sets, iteration, eps):
    x = torch.zeros(vertices, len(sets), dtype=torch.float64, device="cuda")
    teleport = torch.zeros_like(x)
    for q, s in enumerate(sets):
        at = torch.as_tensor(np.asarray(s, dtype=np.int64), device="cuda")
        x[at, q] = 1.0 / len(s) / degree[at].clamp(min=1)
        teleport[at, q] = (1 - DAMPING) / len(s)
    return _epochs(pull, degree, x, teleport, iteration, eps)


def _pagerank(pull, degree, vertices, iteration, eps):
    """Ranks that sum to about 1; eps counts in the units where they sum to the vertex count."""
    x = (1.0 / vertices / degree.clamp(min=1))[:, None]
    return _epochs(pull, degree, x, (1 - DAMPING) / vertices, iteration, eps / vertices)[:, 0]


def _weighted(pull, wsum, vertices, iteration, eps):
    r = torch.ones(vertices, dtype=torch.float64, device="cuda")
    x = 1.0 / wsum
    last = iteration == 1
    for epoch in range(iteration):
        new = (1 - DAMPING) + DAMPING * pull(x[:, None])[:, 0]
        if last:
            return new
        delta = float((new - r).abs().sum())
        r, x = new, new / wsum
        last = delta < eps or epoch + 2 == iteration
    return r


def exact(case, seed):
    kind = case["kind"]
    if kind in ("bfs", "cc", "hyperanf"):  # whole numbers, or sketches of them
        return None
    vertices, src, dst = _edges(case, seed)
    degree = torch.bincount(src, minlength=vertices).double()
    if kind == "wpagerank":
        w = _weights(seed, src.numel())
        wsum = torch.zeros(vertices, dtype=torch.float64, device="cuda").index_add_(0, src, w)
        return _weighted(_Pull(vertices, src, dst, w), wsum, vertices, case["iteration"], case["eps"]).cpu().numpy()
    if kind == "trustrank":
        inverse = _pagerank(_Pull(vertices, dst, src), torch.bincount(dst, minlength=vertices).double(), vertices,
                            100, 0.001)
        n = case["seed_num"]
        seeds = torch.argsort(inverse, descending=True, stable=True)[:n] if vertices > n else torch.arange(vertices)
        ranks = _seeded(_Pull(vertices, src, dst), degree, vertices, [seeds.cpu().numpy()], case["iteration"],
                        case["eps"])
        return {"ranks": ranks[:, 0].cpu().numpy(), "seeds": None}
    pull = _Pull(vertices, src, dst)
    if kind == "pagerank":
        ranks = _pagerank(pull, degree, vertices, case["iteration"], case["eps"])
        return ranks if case["device"] else ranks.cpu().numpy()
    if kind == "ppr":
        root = _root(case, seed, src, dst)
        return _seeded(pull, degree, vertices, [[root]], case["iteration"], case["eps"])[:, 0].cpu().numpy()
    sets = _seed_sets(case, seed, src, dst)
    ranks = _seeded(pull, degree, vertices, sets, case["iteration"], case["eps"])
    k = min(case["topk"], vertices)
    vals = torch.zeros(len(sets), case["topk"], dtype=torch.float64, device="cuda")
    vals[:, :k] = torch.topk(ranks, k, dim=0).values.T
    return {"iterations": None, "topk_ids": None, "topk_vals": vals.cpu().numpy()}
