"""Results by original id that the launches write into page-locked buffers themselves:
the same as in pageable ones, at buffers that begin on an odd element or an odd byte
(copied to instead), and nothing beyond the n results."""

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


@pytest.mark.parametrize("shift", ["aligned", "element", "byte"])
@pytest.mark.parametrize("n", [1, 31, 1025, 300001])
def test_pinned_equals_pageable(n, shift):
    r = np.random.default_rng(n)
    m = 4 * n
    src, dst = r.integers(0, n, m).astype(np.uint32), r.integers(0, max(n - n // 8, 1), m).astype(np.uint32)
    off, adj = orc.csr_from_edges(n, src, dst)
    k = min(3, n)
    seeds = np.arange(k, dtype=np.uint32)
    p = seeds.ctypes.data_as(C.POINTER(C.c_uint32))
    L, V = rg.lib(), rg.VARIANTS["radar"]
    num = C.c_int64()
    calls = {
        "bfs": (np.int32, 1, lambda g, o: L.rg_bfs(g, V, 0, None, C.cast(o, C.POINTER(C.c_int32)), None, None)),
        "bc": (np.float64, 1,
               lambda g, o: L.rg_bc_sources(g, V, p, k, C.cast(o, C.POINTER(C.c_double)), C.byref(num))),
        "radii": (np.int32, 1,
                  lambda g, o: L.rg_radii_seeds(g, V, p, k, C.cast(o, C.POINTER(C.c_int32)), C.byref(num))),
        "bc_multi": (np.float64, k,
                     lambda g, o: L.rg_bc_multi(g, p, k, C.cast(o, C.POINTER(C.c_double)), C.byref(num))),
    }
    with rg.Graph.from_csr(off, adj) as g0, g0.degree_sort() as g:
        for name, (dtype, rows, call) in calls.items():
            size = np.dtype(dtype).itemsize
            want = np.empty(rows * n, dtype)
            assert call(g.handle, want.ctypes.data) == 0, name
            start = {"aligned": 0, "element": size, "byte": 1}[shift]
            buf = rg.pinned_empty((rows * n + 4) * size, np.uint8)
            buf[:] = 0xA5
            assert call(g.handle, buf.ctypes.data + start) == 0, name
            got = np.asarray(buf[start:start + rows * n * size]).copy().view(dtype)
            assert np.all(buf[:start] == 0xA5) and np.all(buf[start + rows * n * size:] == 0xA5), name
            if dtype == np.int32:
                assert np.array_equal(got, want), name
            else:  # FP64 additions in any order
                assert np.array_equal(np.isnan(got), np.isnan(want)), name
                assert_close(np.nan_to_num(got), np.nan_to_num(want), what=name)


@pytest.mark.parametrize("k", [2, 5, 64, 65])
@pytest.mark.parametrize("directed", [False, True], ids=["sym", "dir"])
def test_bc_sources_side_by_side(k, directed):
    """Sources whose forward phases run together add up as one after another (the
    level-by-level run of the same call)."""
    r = np.random.default_rng(k)
    n = 3001
    src, dst = r.integers(0, n, 9000).astype(np.uint32), r.integers(0, n, 9000).astype(np.uint32)
    s = r.integers(0, n, k).astype(np.uint32)
    with rg.Graph.from_edges(n, src, dst, directed=directed) as g:
        one, levels = g.bc_sources(s, "push")
        rg.set_trace(True)
        many, want = g.bc_sources(s, "push")
        rg.set_trace(False)
    assert levels == want and np.array_equal(np.isnan(one), np.isnan(many))
    assert_close(np.nan_to_num(one), np.nan_to_num(many), what="deps")
