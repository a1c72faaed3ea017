"""Pulls beside long lists and empty rows that the search has not reached: hubs whose
only reached neighbour is the last of their list, at the lengths where a pull's reading
changes hands, and calls whose time must not follow what they do not reach."""

import ctypes as C

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


def core(n, base):
    """Every pair of n vertices from id `base` on."""
    i, j = np.triu_indices(n, 1)
    return base + i, base + j


def graph(n, parts, directed=False):
    s, d = (np.concatenate([np.asarray(p[k], np.int64) for p in parts]).astype(np.uint32) for k in (0, 1))
    return rg.Graph.from_edges(n, s, d, directed=directed)


# 16 edges by a lane, 32 and 256 by its warp, pieces of 512 after that
LENGTHS = [16, 17, 48, 49, 304, 305, 304 + 512, 304 + 513, 304 + 2 * 512, 9001]


@pytest.mark.parametrize("directed", [False, True], ids=["sym", "dir"])
@pytest.mark.parametrize("many", [False, True], ids=["last", "every"])
def test_hubs_found_by_their_last_edges(directed, many):
    """Hub after hub of the lengths above: ids of its leaves, then of the hubs, then of a
    dense core (whose frontier is pulled); the core is next to a hub's last entry, or
    (every) to every 97th as well, so that several pieces find it."""
    leaves, hubs = sum(LENGTHS), len(LENGTHS)
    base = leaves + hubs
    rng = np.random.default_rng(1)
    parts, at = [core(300, base)], 0
    for h, length in enumerate(LENGTHS):
        mine = np.arange(at, at + length - 1)
        if many:
            mine[::97] = base + rng.choice(300, len(mine[::97]), replace=False) if len(mine[::97]) < 300 else mine[::97]
        parts.append((mine, np.full(len(mine), leaves + h)))
        parts.append(([base + 299], [leaves + h]))
        at += length
    with graph(base + 300, parts, directed) as g:
        off, adj, _ = g.download()
        for root in (base, base + 299):
            par, depth, rounds, reached = g.bfs("push", root)
            assert rg.last_timing()["kernel_launches"] == 1
            if directed:
                rg.set_trace(True)
                _, want, r2, n2 = g.bfs("push", root)
                rg.set_trace(False)
                assert (rounds, reached) == (r2, n2)
            else:
                want = orc.bfs_depths(off, adj, root)
            assert np.array_equal(depth, want)
            assert reached == int((want >= 0).sum())
            v = np.nonzero(depth > 0)[0]
            assert np.array_equal(depth[par[v]] + 1, depth[v])
        with g.degree_sort() as s:
            assert np.array_equal(s.bfs("push", base)[1], g.bfs("push", base)[1])


def device_ms(call, reps=5):
    call()
    best = 1e9
    for _ in range(reps):
        call()
        best = min(best, rg.last_timing()["total_ms"])
    return best


def one_launch_against_levels(call):
    one = device_ms(call)
    assert rg.last_timing()["kernel_launches"] <= 2
    rg.set_trace(True)
    levels = device_ms(call)
    rg.set_trace(False)
    return one, levels


@pytest.mark.parametrize("directed", [False, True], ids=["sym", "dir"])
def test_bfs_time_beside_an_unreached_hub(directed):
    """A star of 2e6 that the root does not reach (read by one warp it took 60 times the
    level-by-level run; the bound leaves room for a busy machine)."""
    src, dst = rg.generate_edges(18, 16, seed=2)
    n = 1 << 18
    hub = (n + 1 + np.arange(2000000), np.full(2000000, n))
    with graph(n + 2000001, [(src, dst), hub], directed) as g:
        one, levels = one_launch_against_levels(lambda: g.bfs("push", int(src[0]), parents=False))
        assert one < 3 * levels, (one, levels)


def test_radii_and_batched_bfs_beside_empty_rows():
    """4e6 ids without edges between two halves of the others (a lane that walked over
    their rows one by one took 0.8 s): results as level by level, and the time of the
    graph without the gap but for the passes over its vertices."""
    src, dst = rg.generate_edges(18, 16, seed=3)
    n, gap = 1 << 18, 4000000

    def shift(x):
        return np.where(x >= n // 2, x + gap, x)

    seeds = rg.radii_query_seeds(5, n)
    times = []
    for f, size in ((lambda x: x, n), (shift, n + gap)):
        with graph(size, [(f(src.astype(np.int64)), f(dst.astype(np.int64)))]) as g:
            s = f(seeds.astype(np.int64)).astype(np.uint32)
            for variant in ("push", "push-pull"):
                call = lambda: g.radii_seeds(s, variant)
                ms = device_ms(call)
                one = call()
                assert rg.last_timing()["kernel_launches"] == 1
                rg.set_trace(True)
                levels = call()
                rg.set_trace(False)
                assert np.array_equal(one[0], levels[0]) and one[1] == levels[1]
                times.append(ms)
            ms = device_ms(lambda: g.bfs_multi(s))
            one = g.bfs_multi(s)
            assert rg.last_timing()["kernel_launches"] == 1
            rg.set_trace(True)
            levels = g.bfs_multi(s)
            rg.set_trace(False)
            assert np.array_equal(one[0], levels[0]) and one[1] == levels[1]
            times.append(ms)
    for plain, gapped in zip(times[:3], times[3:]):
        assert gapped < 10 * plain, times


def test_pagerank_delta_beside_empty_rows():
    """The same for PageRankDelta's swept rounds, on a graph above the one-launch size."""
    src, dst = rg.generate_edges(18, 24, seed=3)
    n, gap = 1 << 18, 4000000

    def shift(x):
        return np.where(x >= n // 2, x + gap, x).astype(np.int64)

    with graph(n + gap, [(shift(src), shift(dst))]) as g:
        assert g.m > 6 << 20
        ms = device_ms(lambda: g.pagerank_delta("push-pull", 100), reps=2)
        pushed = device_ms(lambda: g.pagerank_delta("push", 100), reps=2)
        assert ms < 5 * pushed, (ms, pushed)
        one, levels = g.pagerank_delta("push-pull", 100), g.pagerank_delta("push", 100)
        assert one[1] == levels[1]
        assert_close(one[0], levels[0], what="ranks")


@pytest.mark.parametrize("variant", ["push", "push-pull"])
def test_pagerank_delta_time_of_a_star(variant):
    """Few edges a vertex: no slower than the swept rounds that rg_set_trace asks for (in
    one launch 2.9 times as slow)."""
    n = 2500001
    with graph(n, [(np.zeros(n - 1), 1 + np.arange(n - 1))]) as g:
        ms = device_ms(lambda: g.pagerank_delta(variant, 100), reps=3)
        rg.set_trace(True)
        swept = device_ms(lambda: g.pagerank_delta("push-pull", 100), reps=3)
        rg.set_trace(False)
    assert ms < 1.6 * swept, (ms, swept)


@pytest.mark.parametrize("k,pinned,one", [(3, False, True), (16, False, False), (16, True, True)])
def test_batched_calls_on_many_vertices_without_edges(k, pinned, one):
    """Fewer edges than vertices: which calls are one launch, and their results."""
    n, rng = 1 << 20, np.random.default_rng(8)
    src = rng.integers(0, n, k).astype(np.uint32)
    ends = rng.integers(0, n, (2, 1000))
    ends[0, 0] = src[0]
    with graph(n, [tuple(ends)]) as g:
        rg.set_trace(True)
        want, levels = g.bc_multi(src)
        rg.set_trace(False)
        if pinned:
            got = rg.pinned_empty((k, n), np.float64)
            count = C.c_int64()
            rg._check(rg.lib().rg_bc_multi(g.handle, src.ctypes.data_as(C.POINTER(C.c_uint32)), k,
                                           got.ctypes.data_as(C.POINTER(C.c_double)), C.byref(count)))
            assert count.value == levels
        else:
            got, count = g.bc_multi(src)
            assert count == levels
        assert (rg.last_timing()["kernel_launches"] == 1) == one
        assert_close(got, want, what="bc rows")


@pytest.mark.parametrize("n,one", [(6 << 20, True), (7 << 20, False)])
def test_batched_bfs_on_many_vertices_without_edges(n, one):
    src = np.array([5, 9], np.uint32)
    with graph(n, [(np.arange(5, 50), np.arange(6, 51))]) as g:
        rows, rounds = g.bfs_multi(src)
        assert (rg.last_timing()["kernel_launches"] == 1) == one
        assert rounds == 46
        for row, s in zip(rows, src):
            assert np.array_equal(row[5:51], np.abs(np.arange(5, 51) - int(s)))
            assert (row[:5] == -1).all() and (row[51:] == -1).all()


def pagerank_is_swept(G, variant):
    got = G.pagerank(variant, 20)
    launches = rg.last_timing()["kernel_launches"]
    rg.set_trace(True)
    want = G.pagerank(variant, 20)
    rg.set_trace(False)
    assert launches > 2
    assert_close(got[0], want[0], what=variant)
    assert got[1] == want[1]
    return np.array_equal(got[0], want[0])


def test_pagerank_of_many_vertices():
    """1.4e6 vertices, one edge each, pulled: in one launch 1.3 times as slow as swept."""
    n, rng = 1400000, np.random.default_rng(2)
    with graph(n, [tuple((n * rng.random((2, n)) ** 6).astype(np.int64))]) as g:
        assert pagerank_is_swept(g, "push-pull")


def test_pagerank_of_skewed_rows():
    """Rows that a CTA of the one launch can hold only by counting for many edges each
    (up to 12 times as slow as the pushes)."""
    n, m, rng = 1700000, 4200000, np.random.default_rng(2)
    ends = (n * rng.random((2, m)) ** [[4], [3]]).astype(np.int64)
    with graph(n, [tuple(ends)]) as g, g.degree_sort() as s:
        pagerank_is_swept(s, "radar")
        pagerank_is_swept(g, "push")


def test_pagerank_beside_a_long_row():
    """Rows of up to 2.5 CTA shares in 2.9e6 edges, pulled (1.7 times as slow in one
    launch)."""
    n, m, rng = 450000, 1450000, np.random.default_rng(3)
    ends = (n * rng.random((2, m)) ** [[1], [4]]).astype(np.int64)
    with graph(n, [tuple(ends)]) as g:
        assert g.m > 1 << 20
        assert pagerank_is_swept(g, "push-pull")
