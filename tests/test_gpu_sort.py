"""The one-sweep sort behind the device CSR builder, the in-lists, the degree sort
and the triangle lists, at the sizes where its tiles (6144 keys) and the CSR tail's
(2048 entries) end: the built graph equals the host clean-up, the permutation the
oracle's, and triangle counts the oracle's."""

import numpy as np
import pytest

import oracle as orc
import radar_graph as rg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build as b
    b.build()


@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned"])
@pytest.mark.parametrize("edges", [1, 2, 1023, 1024, 1025, 3071, 3072, 3073, 6145, 50001])
@pytest.mark.parametrize("n", [2, 255, 257, 65537, 1 << 20])
def test_builders(n, edges, pinned):
    r = np.random.default_rng(n + edges)
    src = r.integers(0, n, edges).astype(np.uint32)
    dst = np.minimum(r.integers(0, n, edges), r.integers(0, n, edges)).astype(np.uint32)
    if pinned:  # an odd start: the edge arrays need no alignment
        ps, pd = rg.pinned_empty(edges + 1, np.uint32), rg.pinned_empty(edges + 1, np.uint32)
        ps[1:], pd[1:] = src, dst
        src, dst = ps[1:], pd[1:]
    off, adj = orc.csr_from_edges(n, np.asarray(src), np.asarray(dst))
    with rg.Graph.from_edges(n, src, dst) as g:
        o, a, _ = g.download()
        assert np.array_equal(o, off) and np.array_equal(a, adj)
        ids, soff, sadj = orc.degree_sort(off, adj)
        with g.degree_sort() as gs:
            o, a, i = gs.download()
            assert np.array_equal(i, ids) and np.array_equal(o, soff) and np.array_equal(a, sadj)
            if len(adj):
                want, total = orc.triangles(off, adj, 0)
                for h in (g, gs):
                    counts, t = h.triangles()
                    assert t == total and np.array_equal(counts, want)
    key = np.unique(np.asarray(src, np.int64) * n + np.asarray(dst, np.int64))
    key = key[key // n != key % n]
    with rg.Graph.from_edges(n, src, dst, directed=True) as g:
        o, a, _ = g.download()
        assert np.array_equal(o, np.searchsorted(key // n, np.arange(n + 1))) and np.array_equal(a, key % n)


@pytest.mark.parametrize("n,edges", [(1, 12 << 20), (300, 12 << 20), (1 << 16, (12 << 20) + 1), ((1 << 20) + 1, 13000000)])
def test_builder_halves(n, edges):
    """Enough edges to be sorted once each: none kept, nearly all dropped, ragged."""
    r = np.random.default_rng(n)
    src = r.integers(0, n, edges).astype(np.uint32)
    dst = np.minimum(r.integers(0, n, edges), r.integers(0, n, edges)).astype(np.uint32)
    lo, hi = np.minimum(src, dst).astype(np.int64), np.maximum(src, dst).astype(np.int64)
    half = np.unique((lo * n + hi)[lo != hi])
    key = np.sort(np.concatenate([half, half % n * n + half // n]))
    with rg.Graph.from_edges(n, src, dst) as g:
        o, a, _ = g.download()
    assert np.array_equal(o, np.searchsorted(key // n, np.arange(n + 1))) and np.array_equal(a, key % n)


def test_endpoint_out_of_range():
    for bad in ([0, 5], [5, 0]):
        with pytest.raises(rg.RgError, match="edge endpoint 5 >= n"):
            rg.Graph.from_edges(5, np.array(bad[:1], np.uint32), np.array(bad[1:], np.uint32))


@pytest.mark.parametrize("hub", [200, 5000])
def test_triangles_streamed(hub):
    """Lists long enough to be streamed against a marked one, ids past the marked and
    counted ranges, and rows that share a group."""
    r = np.random.default_rng(hub)
    n = 40000
    s = np.concatenate([r.integers(0, hub, 60000), r.integers(0, n, 120000)])
    d = np.concatenate([r.integers(0, hub, 60000), r.integers(0, hub, 120000)])
    off, adj = orc.csr_from_edges(n, s.astype(np.uint32), d.astype(np.uint32))
    want, total = orc.triangles(off, adj, 0)
    with rg.Graph.from_csr(off, adj) as g:
        counts, t = g.triangles()
    assert t == total and np.array_equal(counts, want)
