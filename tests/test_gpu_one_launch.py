"""The one-launch traversals (BFS, BC, Radii, PageRank) at the sizes where their
queues, pieces, steps and shares can go wrong: against the level-by-level run of
the same call (which rg_set_trace asks for) and against the oracle.  Depths,
radii and exact-sum ranks are equal; BC is 1e-9 relative."""

import numpy as np
import pytest

import oracle as orc
import radar_graph as rg
from conftest import assert_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build as b
    b.build()


def star(leaves, extra=0):
    """Vertex 0 joined to `leaves` others, then a path of `extra` vertices."""
    s = np.concatenate([np.zeros(leaves, np.int64), leaves + np.arange(extra)])
    d = np.concatenate([1 + np.arange(leaves), leaves + 1 + np.arange(extra)])
    return leaves + 1 + extra, s, d


def path(n):
    return n, np.arange(n - 1), np.arange(1, n)


def random_graph(n, edges, seed, hub=0):
    r = np.random.default_rng(seed)
    s, d = r.integers(0, n, edges), r.integers(0, n, edges)
    return n, np.concatenate([s, np.zeros(hub, np.int64)]), np.concatenate([d, r.integers(0, n, hub)])


GRAPHS = {
    "one": (1, np.zeros(0, np.int64), np.zeros(0, np.int64)),
    "pair": path(2),
    "path300": path(300),
    # degrees at the small/large line (32) and at one, two and many pieces (128 edges)
    "star32": star(32), "star33": star(33), "star127": star(127), "star128": star(128, 3), "star129": star(129),
    "star5000": star(5000, 40),
    # more rows than one CTA takes, isolated vertices, a hub over many steps
    "ragged": random_graph(1033, 700, 1), "sparse": random_graph(70001, 60000, 2),
    "hub": random_graph(20011, 150000, 3, hub=12000), "dense": random_graph(257, 30000, 4),
    # over the largest share of the one-launch PageRank: it must answer all the same
    "star_wide": star(300000),
}


@pytest.mark.parametrize("directed", [False, True], ids=["sym", "dir"])
@pytest.mark.parametrize("name", GRAPHS)
def test_one_launch_equals_levels(name, directed):
    n, s, d = GRAPHS[name]
    g0 = rg.Graph.from_edges(n, s.astype(np.uint32), d.astype(np.uint32), directed=directed)
    off, adj, _ = g0.download()
    r = np.random.default_rng(7)
    roots = [0, n - 1] + [int(x) for x in r.integers(0, n, 2)]
    seeds = np.concatenate([r.integers(0, n, 40), [0, 0, n - 1]]).astype(np.uint32)
    for g in (g0, g0.degree_sort()):
        for v in ("push", "push-pull"):
            one = [g.bfs(v, root) for root in roots], g.radii_seeds(seeds, v), g.bc_sources(roots[:3], v)
            rg.set_trace(True)
            many = [g.bfs(v, root) for root in roots], g.radii_seeds(seeds, v), g.bc_sources(roots[:3], v)
            rg.set_trace(False)
            for a, b in zip(one[0], many[0]):
                assert np.array_equal(a[1], b[1]) and a[2:] == b[2:]
            for a, root in zip(one[0], roots):
                if not directed:
                    assert np.array_equal(a[1], orc.bfs_depths(off, adj, root))
                if not g.sorted:
                    par, depth = a[0].astype(np.int64), a[1]
                    assert np.array_equal(par == 0xFFFFFFFF, depth < 0)
                    at = np.nonzero(depth > 0)[0]
                    assert np.array_equal(depth[par[at]] + 1, depth[at])
                    e = set(zip(np.repeat(np.arange(n), np.diff(off.astype(np.int64))).tolist(), adj.tolist()))
                    assert all((p, c) in e for p, c in zip(par[at].tolist(), at.tolist()))
            assert np.array_equal(one[1][0], many[1][0]) and one[1][1] == many[1][1]
            assert_close(one[2][0], many[2][0], what="bc")
            assert one[2][1] == many[2][1]
        one = g.pagerank("push-pull", 25)
        rg.set_trace(True)
        many = g.pagerank("push-pull", 25)
        rg.set_trace(False)
        assert np.array_equal(one[0], many[0]) and one[1:] == many[1:]


@pytest.mark.parametrize("directed", [False, True], ids=["sym", "dir"])
@pytest.mark.parametrize("k", [1, 2, 31, 33, 64])
@pytest.mark.parametrize("name", ["one", "path300", "star129", "star5000", "ragged", "hub", "dense"])
def test_batched_one_launch(name, k, directed):
    """Sources on one vertex, more sources than groups, rows deeper than the depth
    planes (63), source counts around a word."""
    n, s, d = GRAPHS[name]
    g0 = rg.Graph.from_edges(n, s.astype(np.uint32), d.astype(np.uint32), directed=directed)
    src = np.random.default_rng(k).integers(0, n, k).astype(np.uint32)
    src[-1] = src[0]
    for g in (g0, g0.degree_sort()):
        one = g.bfs_multi(src), g.bc_multi(src)
        rg.set_trace(True)
        many = g.bfs_multi(src), g.bc_multi(src)
        rg.set_trace(False)
        assert np.array_equal(one[0][0], many[0][0]) and one[0][1] == many[0][1]
        assert_close(one[1][0], many[1][0], what="bc rows")
        assert one[1][1] == many[1][1]


@pytest.mark.parametrize("directed", [False, True], ids=["sym", "dir"])
@pytest.mark.parametrize("name", ["one", "path300", "star129", "star5000", "ragged", "sparse", "hub", "dense"])
def test_pagerank_delta_one_launch(name, directed):
    n, s, d = GRAPHS[name]
    g0 = rg.Graph.from_edges(n, s.astype(np.uint32), d.astype(np.uint32), directed=directed)
    for g in (g0, g0.degree_sort()):
        for iters in (0, 1, 2, 100):
            one = g.pagerank_delta("push-pull", iters)
            rg.set_trace(True)
            many = g.pagerank_delta("push-pull", iters)
            rg.set_trace(False)
            assert_close(one[0], many[0], what="ranks")
            assert one[1] == many[1]
            assert_close([one[2]], [many[2]], what="l1")


def test_pagerank_delta_handed_over():
    """Above the one-launch size: dense rounds swept, the sparse ones handed over."""
    off, adj = rg.rmat_csr(20, 16, seed=5)
    with rg.Graph.from_csr(off, adj) as g:
        one = g.pagerank_delta("push-pull", 100)
        rg.set_trace(True)
        many = g.pagerank_delta("push-pull", 100)
        rg.set_trace(False)
        want, rounds, _ = orc.pagerank_delta(off, adj, "push", 100, 0)
    assert one[1] == many[1] == rounds
    assert_close(one[0], many[0], what="levels")
    assert_close(one[0], want, what="oracle")


@pytest.mark.parametrize("sorted_handle", [False, True])
@pytest.mark.parametrize("length", [62, 63, 64, 65, 127, 128, 1025, 5000])
def test_deep_batched_bfs(length, sorted_handle):
    """Depths around the planes that the kernel holds in registers (63) and powers of
    two above, in one launch."""
    n = length + 1 + 40
    off, adj = rg.csr_from_edges(n, np.arange(length, dtype=np.uint32), 1 + np.arange(length, dtype=np.uint32))
    src = np.array([0, length, length // 2, 3, n - 1, 0], np.uint32)  # n - 1: isolated
    with rg.Graph.from_csr(off, adj) as g, g.degree_sort() as s:
        rows, rounds = (s if sorted_handle else g).bfs_multi(src)
        assert rg.last_timing()["kernel_launches"] == 1
    assert rounds == length + 1
    for q, root in enumerate(src):
        assert np.array_equal(rows[q], orc.bfs_depths(off, adj, int(root)))
