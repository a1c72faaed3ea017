"""Waits inside a launch that run out (rg_set_wait_polls makes them short): whatever
barrier the CTAs give up at, the last one included, the call's results are those of
an undisturbed one, and so are the next call's.  Integers and exact sums are equal,
BC and PageRankDelta 1e-9 relative.  A sort that gives up is an error of its call."""

import numpy as np
import pytest

import radar_graph as rg
from conftest import assert_close

pytestmark = pytest.mark.gpu

# a barrier takes a few polls: these let some of the CTAs pass
POLLS = [0, 1, 2, 4]


@pytest.fixture(scope="module", autouse=True)
def built():
    import build as b
    b.build()


@pytest.fixture(scope="module")
def graphs():
    off, adj = rg.rmat_csr(15, 16, seed=9)
    with rg.Graph.from_csr(off, adj) as g, g.degree_sort() as s:
        yield {"plain": g, "sorted": s}


@pytest.fixture
def polls():
    yield rg.set_wait_polls
    rg.set_wait_polls(-1)


SRC = np.arange(3, 43, 5, dtype=np.uint32)


def calls(g):
    n = g.n
    depth, deps, radii = rg.pinned_empty(n, np.int32), rg.pinned_empty(n, np.float64), rg.pinned_empty(n, np.int32)
    seeds = rg.radii_query_seeds(1, n)
    return {
        "bfs": lambda: g.bfs("push", int(SRC[0]), depth_out=depth, parents=False)[1:],
        "bc": lambda: g.bc_sources(SRC[:1], "push", out=deps),  # (one group: another would wait its second out)
        "radii": lambda: g.radii_seeds(seeds, "push", out=radii),
        "pagerank": lambda: g.pagerank("push-pull", 10)[:2],
        "delta": lambda: g.pagerank_delta("push-pull", 100)[:2],
        "bfs_multi": lambda: g.bfs_multi(SRC),
        "bc_multi": lambda: g.bc_multi(SRC),
    }


def check(name, got, want):
    if name in ("bc", "delta", "bc_multi"):
        assert_close(got[0], want[0], what=name)
    else:
        assert np.array_equal(got[0], want[0]), name
    assert got[1:] == want[1:], name


@pytest.mark.parametrize("app", ["bfs", "bc", "radii", "pagerank", "delta", "bfs_multi", "bc_multi"])
@pytest.mark.parametrize("kind", ["plain", "sorted"])
def test_a_launch_that_gives_up(graphs, polls, kind, app):
    call = calls(graphs[kind])[app]
    want = tuple(np.array(x) if isinstance(x, np.ndarray) else x for x in call())
    assert rg.last_timing()["kernel_launches"] <= 3
    for first in range(200):  # more barriers than any of these runs has
        gave_up = 0
        for limit in POLLS:
            polls(limit, first)
            for _ in range(3):
                got = call()
                gave_up += rg.last_timing()["kernel_launches"] > 3
                check(app, got, want)
        if not gave_up:
            break
    assert 1 < first < 200
    polls(-1)
    check(app, call(), want)
    assert rg.last_timing()["kernel_launches"] <= 3


def built_lists(g):
    return [x for x in g.download() if x is not None]


@pytest.mark.parametrize("build", ["edges", "edges-halves", "edges-directed", "sort", "sort-directed", "triangles"])
def test_a_sort_that_gives_up(polls, build):
    """The call fails, or is right where no wait was needed; nothing is indexed with
    what the sort left behind, and the next call is right."""
    r = np.random.default_rng(4)
    n, ne = (300000, 13 << 20) if build == "edges-halves" else (90001, 400000)
    s, d = (r.integers(0, n, ne).astype(np.uint32) for _ in range(2))
    directed = build.endswith("directed")
    if build.startswith("edges"):
        call, lists = lambda: rg.Graph.from_edges(n, s, d, directed=directed), built_lists
    else:
        g = rg.Graph.from_edges(n, s, d, directed=directed)
        if build == "triangles":
            g = g.degree_sort()
            call, lists = g.triangles, lambda x: [x[0]]
        else:
            call, lists = g.degree_sort, built_lists
    want = lists(call())
    failed = 0
    for limit in [0, 0, 1, 2, 4, 8, 16]:
        polls(limit)
        try:
            got = call()
        except rg.RgError as e:
            failed += 1
            assert "did not finish" in str(e)
            got = None
        polls(-1)
        if got is not None:
            assert all(np.array_equal(a, b) for a, b in zip(lists(got), want))
    assert failed
    assert all(np.array_equal(a, b) for a, b in zip(lists(call()), want))
