"""GPU: a radix sort whose bounded wait runs out.  With a bound of no looks every
part of the sort but the first gives up at once: the call that sorted must
report it and nothing may be made of the unfinished keys."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")

DEVICE_ERROR = -5
DEFAULT_LOOKS = 1 << 22


def set_sort_wait(g, looks):
    assert vx.capi().vx_graph_set_sort_wait(C.c_void_p(g.handle), C.c_uint32(looks)) == 0


def load(g, e):
    e = np.ascontiguousarray(e, np.uint32)
    return vx.capi().vx_graph_bulk_load(C.c_void_p(g.handle), e.ctypes.data_as(C.POINTER(C.c_uint32)),
                                        C.c_size_t(len(e)))


def arcs(e, directed):
    a = e[e[:, 0] != e[:, 1]].astype(np.uint64)
    k = a[:, 0] << np.uint64(32) | a[:, 1]
    if not directed:
        k = np.r_[k, a[:, 1] << np.uint64(32) | a[:, 0]]
    return np.unique(k)


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("n", [20_000, 1_000_000])
def test_a_load_reports_it_and_can_be_repeated(n, directed):
    e = np.random.default_rng(n).integers(0, 30_000, (n, 2), dtype=np.uint32)
    g = vx.Graph(30_000, directed)
    set_sort_wait(g, 0)
    for _ in range(3):
        assert load(g, e) == DEVICE_ERROR
        assert "sort" in vx.last_error()
    assert load(g, e[:100]) == 0  # sorted by one block: nothing waits
    set_sort_wait(g, DEFAULT_LOOKS)
    assert load(g, e) == 0
    want = arcs(e, directed)
    assert g.edge_count_directed() == want.size
    for u in (0, 17, 29_999):
        lo, hi = np.searchsorted(want, [u << 32, u + 1 << 32])
        assert g.neighbors(u) == (want[lo:hi] & np.uint64(0xFFFFFFFF)).tolist()


def big_batch(ops=60_000, V=30_000, seed=2):
    rng = np.random.default_rng(seed)
    return (rng.integers(0, V, ops, dtype=np.uint32), rng.integers(0, V, ops, dtype=np.uint32),
            (rng.random(ops) < 0.7).astype(np.uint8))


def small_graph(directed, V=30_000):
    g = vx.Graph(V, directed)
    g.bulk_load_edges(np.random.default_rng(1).integers(0, V, (2 * V, 2), dtype=np.uint32))
    return g


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("fused", [True, False])
def test_a_batch_reports_it_and_holds_no_arcs(fused, directed):
    g = small_graph(directed)
    b = vx.IncrementalBFS(g, 5)
    b.set_fused(fused)
    before = [g.neighbors(u) for u in range(40)]
    set_sort_wait(g, 0)
    b.apply_arrays(*big_batch(100_000))
    for call in (b.stats, b.distances_array, g.edge_count_directed):
        with pytest.raises(RuntimeError):
            call()
    assert [g.neighbors(u) for u in range(40)] == before
    set_sort_wait(g, DEFAULT_LOOKS)  # the error stays
    b.apply_arrays(*big_batch(10))
    with pytest.raises(RuntimeError):
        b.stats()


@pytest.mark.parametrize("directed", [False, True])
def test_a_graph_batch_reports_it(directed):
    g = small_graph(directed)
    set_sort_wait(g, 0)
    g.apply_arrays(*big_batch(100_000))
    with pytest.raises(RuntimeError):
        g.edge_count_directed()


@pytest.mark.parametrize("stats", [False, True])
def test_a_stream_reports_it(stats):
    g = small_graph(False)
    b = vx.IncrementalBFS(g, 5)
    set_sort_wait(g, 0)
    s, d, a = big_batch()
    with pytest.raises(RuntimeError):
        b.apply_stream(s, d, a, np.arange(0, 60_001, 6000, dtype=np.uint64), digests=True, stats=stats)


def test_components_report_it():
    g = small_graph(False)
    c = vx.IncrementalComponents(g)
    set_sort_wait(g, 0)
    c.apply_arrays(*big_batch())
    with pytest.raises(RuntimeError):
        c.labels_array()
    with pytest.raises(RuntimeError):
        c.last_repaired_vertices


@pytest.mark.parametrize("directed", [False, True])
def test_batches_after_an_error_stay_within_the_lists(directed):
    # each of them would append its arcs behind the lengths the one before left
    g = small_graph(directed)
    b = vx.IncrementalBFS(g, 5)
    set_sort_wait(g, 0)
    b.apply_arrays(*big_batch(100_000))
    for t in range(60):
        b.apply_arrays(*big_batch(16_384, seed=t))
    with pytest.raises(RuntimeError):
        b.stats()
    set_sort_wait(g, DEFAULT_LOOKS)  # the memory around the lists is sound
    h = small_graph(directed)
    c = vx.IncrementalBFS(h, 5)
    c.apply_arrays(*big_batch(16_384))
    assert np.array_equal(c.distances_array(), vx.IncrementalBFS(h, 5).distances_array())
