"""Timed cases of the framework: what a user's program calls, over the range of graphs it is used on.

A case is one call of an app (or of the graph builder) on a seeded graph.  Graphs are R-MAT
(a = 0.57, b = c = 0.19, the skew of the benchmark's graphs) or uniform random, generated on the GPU
with ids shuffled, from a few thousand edges (a unit test, an interactive query) to 2^28 edges (the
benchmark's graph); vertex counts are mostly not powers of two.  Results go to page-locked host
buffers, as in a program that keeps its result buffers.

Keys of a case:
  app       bfs | pagerank | bc | radii | pagerank_delta | triangles | bfs_multi | bc_multi | build
  n, edges  vertices, generated edges (before both directions, repeats and self loops are dealt with)
  graph     rmat | uniform
  directed  out-lists and in-lists instead of one symmetric list
  sorted    degree-sorted (the RADAR variant's default) or in original order (push, push-pull)
  variant   the reference variant that is asked for
  schedule  "default": the library's own options; "tuned": the schedule that the autotuner picks on
            graphs of this kind, kept by the program with set_tuning
  k         sources (bc, bfs_multi, bc_multi); iters: PageRank iterations
"""

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "radar-graph_gb300"))
import radar_graph as rg  # noqa: E402

RMAT = (0.57, 0.19, 0.19)

# The autotuner's choices on degree-sorted skewed graphs: dense iterations pull (PageRank with 16
# edges per lane and cached hubs), BC pushes with 4 KiB of hub counters in its backward phase.
TUNED = {
    "pagerank": (0.0, {"direction": 1, "hub_smem_kb": 48, "sweep_shape": 161, "dense_div": 20}),
    "bfs": (0.0, {"direction": 1, "dense_div": 20}),
    "bc": (0.0, {"direction": 0, "hub_smem_kb": 4, "bc_fwd_hubs": 0, "dense_div": 20}),
    "radii": (0.0, {"direction": 1, "dense_div": 20}),
}


def _case(app, n, edges, **more):
    c = {"app": app, "n": n, "edges": edges, "graph": "rmat", "directed": False, "sorted": True, "variant": "radar",
         "schedule": "tuned"}
    c.update(more)
    return c


def listed():
    return [
        # an interactive query on a small graph, library defaults: launches and latency
        _case("bfs", 1 << 10, 16 << 10, schedule="default", name="bfs-1k"),
        # the benchmark's BFS: a social-network-sized graph, autotuned
        _case("bfs", 1 << 24, 1 << 28, name="bfs-16m"),
        # ranking a small graph (a site, a citation set) to the reference's 20 iterations
        _case("pagerank", 9001, 131072, iters=20, name="pagerank-9k"),
        # the benchmark's PageRank
        _case("pagerank", 1 << 24, 1 << 28, iters=20, name="pagerank-16m"),
        # betweenness from a few sampled sources on a directed graph (a web crawl), library defaults
        _case("bc", 60001, 900000, directed=True, schedule="default", k=4, name="bc-60k-directed"),
        # the benchmark's BC: one source, autotuned
        _case("bc", 8000009, 1 << 27, k=1, name="bc-8m"),
        # eccentricity estimate (64 samples) on a mid-sized graph, autotuned
        _case("radii", 1000003, 16000000, name="radii-1m"),
        # PageRankDelta to convergence on an unsorted graph, the push-pull variant
        _case("pagerank_delta", 1 << 21, 1 << 25, sorted=False, variant="push-pull", schedule="default",
              name="prdelta-2m-unsorted"),
        # triangle counts per vertex
        _case("triangles", 200003, 4000000, name="triangles-200k"),
        # 64 BFS roots at once (the serving layer's coalesced batch)
        _case("bfs_multi", 1000003, 16000000, k=64, name="bfs_multi-1m-64"),
        # 16 independent BC queries at once
        _case("bc_multi", 500009, 8000000, k=16, name="bc_multi-500k-16"),
        # loading: a host edge list to the cleaned, degree-sorted CSR, and that CSR back for saving
        _case("build", 1 << 21, 1 << 25, name="build-2m"),
    ]


#: Largest drawn vertex count and edge count by app (edges over vertices: 4 to 32).
LIMITS = {"bfs": (1 << 24, 1 << 28), "pagerank": (1 << 24, 1 << 28), "bc": (1 << 23, 1 << 27), "radii": (1 << 22, 1 << 26),
          "pagerank_delta": (1 << 21, 1 << 25), "triangles": (200003, 4000000), "bfs_multi": (1000003, 16000000),
          "bc_multi": (500009, 8000000), "build": (1 << 21, 1 << 25)}


def draw(rng):
    app = rng.choice(list(LIMITS))
    top_n, top_e = LIMITS[app]
    n = int(math.exp(rng.uniform(math.log(1000), math.log(top_n))))
    edges = min(int(n * math.exp(rng.uniform(math.log(4), math.log(32)))), top_e)
    c = _case(app, n, edges, graph=rng.choice(["rmat", "rmat", "uniform"]))
    if app in ("build", "triangles"):
        if app == "build":
            c["directed"] = rng.random() < 0.3
        return c
    c["directed"] = rng.random() < 0.25
    c["variant"] = rng.choice(["radar", "radar", "push-pull"])
    c["sorted"] = c["variant"] == "radar"
    c["schedule"] = rng.choice(["default", "tuned"])
    if app == "pagerank":
        c["iters"] = rng.choice([5, 20])
    elif app == "bc":
        c["k"] = rng.choice([1, 4])
    elif app == "bfs_multi":
        c["k"] = rng.randint(2, 64)
    elif app == "bc_multi":
        c["k"] = rng.randint(2, 16)
    return c


def _edges(case, seed):
    """(src, dst) int32 on the GPU: R-MAT or uniform ids below n, shuffled."""
    n, ne = case["n"], case["edges"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + n)
    if case["graph"] == "uniform":
        return tuple(torch.randint(0, n, (ne,), generator=g, device="cuda", dtype=torch.int32) for _ in range(2))
    a, b, c = RMAT
    src = torch.zeros(ne, dtype=torch.int32, device="cuda")
    dst = torch.zeros(ne, dtype=torch.int32, device="cuda")
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(ne, generator=g, device="cuda")
        down = r >= a + b
        src.mul_(2).add_(down)
        dst.mul_(2).add_(torch.where(down, r >= a + b + c, r >= a))
    perm = torch.randperm(n, generator=g, device="cuda", dtype=torch.int32)
    for x in (src, dst):
        x.sub_((x >= n).to(torch.int32) * n)  # ids are below the next power of two, so below 2 n
        x.copy_(perm[x])
    return src, dst


def _check(status):
    if status:
        raise RuntimeError(rg.lib().rg_last_error().decode())


def _sources(src, k, seed):
    """k vertices with edges, drawn from the seed (degree-proportional, as queries hit busy vertices)."""
    g = torch.Generator()
    g.manual_seed(seed)
    at = torch.randint(0, src.numel(), (k,), generator=g)
    return src[at.to(src.device)].cpu().numpy().astype(np.uint32)


def prepare(case, seed):
    app, n = case["app"], case["n"]
    src, dst = _edges(case, seed)
    if app == "build":
        h_src, h_dst = (rg.pinned_empty(case["edges"], np.uint32) for _ in range(2))
        torch.from_numpy(np.asarray(h_src).view(np.int32)).copy_(src)
        torch.from_numpy(np.asarray(h_dst).view(np.int32)).copy_(dst)
        adj = rg.pinned_empty(case["edges"] * (1 if case["directed"] else 2), np.uint32)  # room for every entry
        adj[:] = 0
        return {"case": case, "src": h_src, "dst": h_dst, "off": rg.pinned_empty(n + 1, np.uint32),
                "ids": rg.pinned_empty(n, np.uint32), "adj": adj}
    k = case.get("k", 1)
    roots = _sources(src, k, seed)
    torch.cuda.synchronize()  # the edges are made on torch's stream
    L = rg.lib()
    h = C.c_void_p()
    make = L.rg_graph_create_directed_from_edges if case["directed"] else L.rg_graph_create_from_edges
    _check(make(n, case["edges"], src.data_ptr(), dst.data_ptr(), 1, C.byref(h)))
    g = rg.Graph(h)
    if case["sorted"]:
        plain, g = g, g.degree_sort()
        plain.free()
    if case["schedule"] == "tuned":
        g.set_tuning(TUNED)
    s = {"case": case, "g": g, "roots": roots}
    if app in ("pagerank", "bc", "pagerank_delta"):
        s["out"] = rg.pinned_empty(n, np.float64)
    elif app in ("bfs", "radii"):
        s["out"] = rg.pinned_empty(n, np.int32)
    elif app == "triangles":
        s["out"] = rg.pinned_empty(n, np.uint64)
    else:
        s["out"] = rg.pinned_empty((k, n), np.int32 if app == "bfs_multi" else np.float64)
    if app == "radii":
        s["seeds"] = rg.radii_query_seeds(seed, n)
    return s


def run(state):
    case = state["case"]
    app, variant = case["app"], case["variant"]
    if app == "build":
        with rg.Graph.from_edges(case["n"], state["src"], state["dst"], directed=case["directed"]) as g0, \
                g0.degree_sort() as g:
            m = g.m
            p = [state[x].ctypes.data_as(C.POINTER(C.c_uint32)) for x in ("off", "adj", "ids")]
            _check(rg.lib().rg_graph_download(g.handle, *p))
        return {"off": state["off"].view(np.int32), "adj": state["adj"].view(np.int32),
                "ids": state["ids"].view(np.int32), "m": m}
    g, out = state["g"], state["out"]
    if app == "bfs":
        _, depth, rounds, reached = g.bfs(variant, int(state["roots"][0]), depth_out=out, parents=False)
        return {"depth": depth, "rounds": rounds, "reached": reached}
    if app == "pagerank":
        ranks, it, l1 = g.pagerank(variant, case["iters"], out=out)
        return {"ranks": ranks, "iterations": it, "l1": l1}
    if app == "bc":
        deps, levels = g.bc_sources(state["roots"], variant, out=out)
        return {"deps": deps, "levels": levels}
    if app == "radii":
        r, rounds = g.radii_seeds(state["seeds"], variant, out=out)
        return {"radii": r, "rounds": rounds}
    # the calls below allocate their results in the Python mirror; the C ABI takes the program's buffers
    L = rg.lib()
    count, l1, total = C.c_int64(), C.c_double(), C.c_uint64()
    if app == "pagerank_delta":
        _check(L.rg_pagerank_delta(g.handle, rg.VARIANTS[variant], 100, out.ctypes.data_as(C.POINTER(C.c_double)),
                                   C.byref(count), C.byref(l1)))
        return {"ranks": out, "iterations": count.value, "l1": l1.value}
    if app == "triangles":
        _check(L.rg_triangle_count(g.handle, out.ctypes.data_as(C.POINTER(C.c_uint64)), C.byref(total)))
        return {"triangles": out.view(np.int64), "total": total.value}
    roots = state["roots"]
    p = roots.ctypes.data_as(C.POINTER(C.c_uint32))
    if app == "bfs_multi":
        _check(L.rg_bfs_multi(g.handle, p, len(roots), out.ctypes.data_as(C.POINTER(C.c_int32)), C.byref(count)))
        return {"depths": out, "rounds": count.value}
    if app == "bc_multi":
        _check(L.rg_bc_multi(g.handle, p, len(roots), out.ctypes.data_as(C.POINTER(C.c_double)), C.byref(count)))
        return {"deps": out, "levels": count.value}
    raise ValueError(app)


def work(case):
    """Bytes of the CSR's entries and offsets read once per traversal (per PageRank iteration), plus the
    per-vertex values read and written; operations per edge.  Repeats in the edge list are counted as edges."""
    app, n = case["app"], case["n"]
    m = case["edges"] * (1 if case["directed"] else 2)
    csr, k = 4 * m + 4 * (n + 1), case.get("k", 1)
    if app == "bfs":
        return {"bytes": csr + 4 * n, "flops": m}
    if app == "pagerank":
        return {"bytes": case["iters"] * (csr + 16 * n), "flops": 2 * m * case["iters"]}
    if app == "bc":
        return {"bytes": k * (2 * csr + 32 * n), "flops": 2 * m * k}
    if app == "radii":
        return {"bytes": 2 * csr + 20 * n, "flops": 2 * m}
    if app == "pagerank_delta":
        return {"bytes": 5 * (csr + 40 * n), "flops": 10 * m}
    if app == "triangles":
        return {"bytes": csr + 8 * n, "flops": 20 * m}
    if app == "bfs_multi":
        return {"bytes": 2 * csr + 24 * n + 4 * n * k, "flops": 2 * m}
    if app == "bc_multi":
        return {"bytes": 4 * csr + 40 * n * k, "flops": 2 * m * k}
    return {"bytes": 8 * case["edges"] + 2 * csr + 4 * n, "flops": m}


# ---------------------------------------------------------------------------
# the same results in 64 bits by plain torch
# ---------------------------------------------------------------------------
def _entries(case, seed):
    """The cleaned graph's directed entries (a, b), each once, no self loops."""
    src, dst = _edges(case, seed)
    a, b = src.long(), dst.long()
    key = a * case["n"] + b
    if not case["directed"]:
        key = torch.cat([key, b * case["n"] + a])
    del a, b, src, dst
    key = torch.unique_consecutive(torch.sort(key).values)
    a = torch.div(key, case["n"], rounding_mode="floor")
    b = key - a * case["n"]
    keep = a != b
    return a[keep], b[keep]


def _pagerank(case, a, b):
    n, damp = case["n"], 0.85
    deg = torch.bincount(a, minlength=n).double()
    p = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    l1, it = 0.0, 0
    for it in range(1, case["iters"] + 1):
        c = torch.where(deg > 0, p / deg.clamp(min=1), torch.zeros_like(p))
        q = damp * torch.zeros_like(p).index_add_(0, b, c[a]) + (1 - damp) / n
        l1 = float((p - q).abs().sum())
        p = q
        if l1 < 1e-7:
            break
    else:
        it += 1
    return {"ranks": p.cpu(), "iterations": None, "l1": l1}


def _pagerank_delta(case, a, b):
    n, damp = case["n"], 0.85
    deg = torch.bincount(a, minlength=n).double()
    p = torch.zeros(n, dtype=torch.float64, device="cuda")
    delta = torch.full_like(p, 1.0 / n)
    active = torch.ones(n, dtype=torch.bool, device="cuda")
    added, l1 = (1 - damp) / n, 0.0
    for r in range(100):
        c = torch.where(active & (deg > 0), delta / deg.clamp(min=1), torch.zeros_like(p))
        s = damp * torch.zeros_like(p).index_add_(0, b, c[a])
        if r == 0:
            delta = s + added
            p = p + delta
            delta = delta - 1.0 / n
            active = delta.abs() > 0.01 * p
        else:
            delta = s
            active = delta.abs() > 0.01 * p
            p = torch.where(active, p + delta, p)
        l1 = float(delta.abs().sum())
        if l1 < 1e-7:
            break
    return {"ranks": p.cpu(), "iterations": None, "l1": l1}


def _bc_pass(n, fwd, bwd, root, deps):
    """One source: path counts along `fwd`, dependencies pushed along `bwd`, added to `deps` in place of
    a fresh array (the reference chains its sources)."""
    a, b = fwd
    level = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    sigma = torch.zeros(n, dtype=torch.float64, device="cuda")
    level[root], sigma[root] = 0, 1.0
    r = 0
    while True:
        e = (level[a] == r) & (level[b] < 0)
        if not bool(e.any()):
            break
        eb = b[e]
        sigma.index_add_(0, eb, sigma[a[e]])
        r += 1
        level[eb] = r
    inv = 1.0 / sigma
    c, d = bwd
    visited = torch.zeros(n, dtype=torch.bool, device="cuda")
    for x in range(r, -1, -1):
        at = level == x
        visited |= at
        deps = torch.where(at, deps + inv, deps)
        if x:
            e = (level[c] == x) & ~visited[d]
            deps.index_add_(0, d[e], deps[c[e]])
    return (deps - inv) * sigma


def exact(case, seed):
    app = case["app"]
    if app not in ("pagerank", "pagerank_delta", "bc", "bc_multi"):
        return None  # whole numbers
    a, b = _entries(case, seed)
    if app == "pagerank":
        return _pagerank(case, a, b)
    if app == "pagerank_delta":
        return _pagerank_delta(case, a, b)
    n = case["n"]
    roots = _sources(_edges(case, seed)[0], case["k"], seed)
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    if app == "bc_multi":
        return {"deps": torch.stack([_bc_pass(n, (a, b), (b, a), int(r), zero.clone()).cpu() for r in roots]),
                "levels": None}
    deps = zero
    for i, r in enumerate(roots):  # a directed graph is transposed after every source
        turn = case["directed"] and i % 2 == 1
        deps = _bc_pass(n, (b, a) if turn else (a, b), (a, b) if turn else (b, a), int(r), deps)
    return {"deps": deps.cpu(), "levels": None}
