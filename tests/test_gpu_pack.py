"""GPU: host batches are the caller's once the call has returned, whatever is
done with the stream in between: many small batches without a wait, and batches
captured from the graph's stream and run after later calls."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_capture import GLOBAL_MODE, runtime

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")

V = 50_000


def batch(seed, n):
    rng = np.random.default_rng(seed)
    return (rng.integers(0, V, n, dtype=np.uint32), rng.integers(0, V, n, dtype=np.uint32),
            (rng.random(n) < 0.8).astype(np.uint8))


def make():
    g = vx.Graph(V, False)
    b = vx.IncrementalBFS(g, 0)
    b.apply_arrays(*batch(0, 20_000))
    b.stats()
    return g, b


def stream_of(g):
    p = C.c_void_p()
    assert vx.capi().vx_graph_stream(C.c_void_p(g.handle), C.byref(p)) == 0
    return p


@pytest.mark.parametrize("n", [1, 64, 8192, 8193])
def test_a_captured_host_batch_keeps_its_ops(n):
    rt = runtime()
    first, later = batch(1, n), batch(2, n)
    g, b = make()
    stream, graph, ex = stream_of(g), C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamBeginCapture(stream, C.c_int(GLOBAL_MODE)) == 0
    try:
        b.apply_arrays(*first)
    finally:
        ended = rt.cudaStreamEndCapture(stream, C.byref(graph))
    assert ended == 0
    assert rt.cudaGraphInstantiate(C.byref(ex), graph, C.c_ulonglong(0)) == 0
    b.apply_arrays(*later)
    assert rt.cudaGraphLaunch(ex, stream) == 0
    got = b.distances_array()
    rt.cudaGraphExecDestroy(ex)
    rt.cudaGraphDestroy(graph)
    g1, b1 = make()
    b1.apply_arrays(*later)
    b1.apply_arrays(*first)
    assert g.edge_count_directed() == g1.edge_count_directed()
    assert np.array_equal(got, b1.distances_array())


@pytest.mark.parametrize("sizes", [(1,), (64, 1, 700), (8192, 8191, 3, 5000), (8192, 8193, 1)])
def test_batches_without_a_wait(sizes):
    g, b = make()
    have = {}
    s, d, a = batch(0, 20_000)
    todo = [(s, d, a)]
    for t in range(120):
        s, d, a = batch(100 + t, sizes[t % len(sizes)])
        todo.append((s.copy(), d.copy(), a.copy()))
        b.apply_arrays(s, d, a)
        s[:], d[:], a[:] = 0, 1, 0  # the caller's arrays are its own again
    for s, d, a in todo:
        for u, v, x in zip(s.tolist(), d.tolist(), a.tolist()):
            if u != v:
                have[(min(u, v), max(u, v))] = x
    assert g.edge_count_directed() == 2 * sum(have.values())
    assert np.array_equal(b.distances_array(), vx.IncrementalBFS(g, 0).distances_array())
