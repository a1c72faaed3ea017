"""Every schedule of the level-by-level runs, which answer large graphs, traced calls and
those whose one launch gives up: variants, directions, dense thresholds and hub
budgets against the oracle (integers bit-exact, doubles 1e-9), with rg_set_trace on so
that no call of these graphs is one launch; and PageRank's cached hubs, which only
graphs of more than 6.3e6 vertices have."""

import contextlib

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


@contextlib.contextmanager
def traced(**kw):
    old = {k: rg.get_option(k) for k in kw}
    try:
        for k, v in kw.items():
            rg.set_option(k, v)
        rg.set_trace(True)
        yield
    finally:
        rg.set_trace(False)
        for k, v in old.items():
            rg.set_option(k, v)


class G:
    def __init__(self, uniform):
        self.off, self.adj = rg.rmat_csr(15, 16, seed=3, uniform=uniform)
        self.g = rg.Graph.from_csr(self.off, self.adj)
        self.gs = self.g.degree_sort()
        deg = np.diff(self.off.astype(np.int64)).astype(np.uint32)
        self.pr = orc.pagerank(self.off, self.adj, "push", 20, 0)
        self.prd = orc.pagerank_delta(self.off, self.adj, "push", 30, 0)
        self.src = orc.bc_sources(deg, 2)
        self.root = int(self.src[0])
        self.depth = orc.bfs_depths(self.off, self.adj, self.root)
        self.bc = orc.bc(self.off, self.adj, self.src, "push", 0)[0]
        self.radii = orc.radii(self.off, self.adj, orc.radii_seeds(len(deg)), "push", 1)[0]

    def of(self, variant):
        return self.gs if variant in ("radar", "degree-sorting") else self.g


@pytest.fixture(scope="module", params=[False, True], ids=["rmat", "er"])
def graph(request):
    return G(request.param)


VARIANTS = ["push", "push-pull", "degree-sorting", "hubdup", "radar"]


def hub_modes():
    """The hub copies of the pushes traced since the last call."""
    return {r["hub_mode"] for r in rg.take_trace() if r["mode"] != "pull"}


@pytest.mark.parametrize("kb", [0, 4, 48])
@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("variant", VARIANTS)
def test_bfs_radii_and_bc(graph, variant, direction, kb):
    S = graph.of(variant)
    hubs = {"radar": 1, "hubdup": 2}.get(variant, 0) if kb else 0
    for div in (2, 20):
        with traced(dense_div=div, direction=direction, hub_smem_kb=kb):
            par, depth, _, _ = S.bfs(variant, graph.root)
            assert hub_modes() <= {0, hubs}
            radii, _ = S.radii(variant)
            assert hub_modes() <= {0, hubs}
        assert np.array_equal(depth, graph.depth)
        assert np.array_equal(radii, graph.radii)
        if not S.sorted:
            at = np.nonzero(depth > 0)[0]
            assert np.array_equal(depth[par[at]] + 1, depth[at])
        for fwd in (0, 1):
            with traced(dense_div=div, direction=direction, hub_smem_kb=kb, bc_fwd_hubs=fwd):
                deps, _ = S.bc_sources(graph.src, variant)
                modes = hub_modes()
            assert modes <= {0, hubs}
            assert hubs in modes or direction or not hubs
            assert_close(deps, graph.bc, what=f"bc {variant} fwd {fwd}")


@pytest.mark.parametrize("shape", [40, 41, 42, 80, 81, 82, 160, 161, 162])
@pytest.mark.parametrize("direction,kb", [(0, 0), (0, 16), (1, 0), (1, 48)])
@pytest.mark.parametrize("variant", ["radar", "hubdup", "push-pull"])
def test_pagerank(graph, shape, direction, kb, variant):
    with traced(sweep_shape=shape, direction=direction, hub_smem_kb=kb):
        r, it, _ = graph.of(variant).pagerank(variant, 20)
        assert rg.last_timing()["kernel_launches"] > 40
    assert it == graph.pr[1]
    assert_close(r, graph.pr[0], what=f"pr {variant} {shape} {direction} {kb}")


@pytest.mark.parametrize("direction,kb", [(0, 0), (0, 16), (1, 0)])
@pytest.mark.parametrize("variant", VARIANTS)
def test_pagerank_delta(graph, variant, direction, kb):
    for div in (2, 20):
        with traced(dense_div=div, direction=direction, hub_smem_kb=kb):
            r, it, _ = graph.of(variant).pagerank_delta(variant, 30)
        assert it == graph.prd[1]
        assert_close(r, graph.prd[0], what=f"delta {variant}")


@pytest.mark.parametrize("shape", [81, 161])
@pytest.mark.parametrize("k", [2, 33, 64])
def test_batched(graph, shape, k):
    src = np.random.default_rng(k).integers(0, graph.g.n, k).astype(np.uint32)
    for S in (graph.g, graph.gs):
        with traced(sweep_shape=shape):
            depths, _ = S.bfs_multi(src)
            rows, _ = S.bc_multi(src)
        for q in {0, 1, k - 1}:
            s = int(src[q])
            assert np.array_equal(depths[q], orc.bfs_depths(graph.off, graph.adj, s))
            assert_close(rows[q], orc.bc(graph.off, graph.adj, src[q:q + 1], "push", 0)[0], what=f"row {q}")


@pytest.mark.parametrize("layers,past", [(10, False), (18, True)])
def test_batched_bc_path_counts(layers, past):
    """16^(layers - 1) shortest paths reach the last layer; past 2^64 the shared
    traversal's integers are dropped for single-source passes."""
    assert (16 ** (layers - 1) >= 2 ** 64) == past
    ids = 1 + np.arange(16 * layers, dtype=np.uint32).reshape(layers, 16)
    src = [np.zeros(16, np.uint32)] + [np.repeat(ids[i], 16) for i in range(layers - 1)]
    dst = [ids[0]] + [np.tile(ids[i + 1], 16) for i in range(layers - 1)]
    off, adj = rg.csr_from_edges(1 + ids.size, np.concatenate(src), np.concatenate(dst))
    roots = np.array([0, 3, 100], np.uint32)
    with rg.Graph.from_csr(off, adj) as g:
        with traced():
            rows, _ = g.bc_multi(roots)
    for row, s in zip(rows, roots):
        assert_close(row, orc.bc(off, adj, np.array([s], np.uint32), "push", 0)[0], what=f"source {s}")


def test_pagerank_with_cached_hubs_is_bit_identical():
    """Contributions of the first ids from shared memory, for every sweep shape."""
    n, rng = (6 << 20) + 12345, np.random.default_rng(6)
    dst = (n * rng.random(9 << 20) ** 4).astype(np.uint32)
    with rg.Graph.from_edges(n, rng.integers(0, n, len(dst)).astype(np.uint32), dst) as g, g.degree_sort() as s:
        old = {k: rg.get_option(k) for k in ("direction", "hub_smem_kb", "sweep_shape")}
        try:
            rg.set_option("direction", 1)
            rg.set_option("hub_smem_kb", 0)
            want = s.pagerank("radar", 6)
            for shape in (40, 41, 42, 80, 81, 82, 160, 161, 162):
                for kb in (1, 48, 200):
                    rg.set_option("sweep_shape", shape)
                    rg.set_option("hub_smem_kb", kb)
                    got = s.pagerank("radar", 6)
                    assert np.array_equal(got[0], want[0]) and got[1:] == want[1:], (shape, kb)
        finally:
            for k, v in old.items():
                rg.set_option(k, v)
