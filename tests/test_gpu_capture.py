"""GPU: an update batch on device arrays captured from the graph's stream, with
a readback of the arena's top still to be looked at.  The captured launch, run
once, gives what the same batch gives without a capture."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")
torch = pytest.importorskip("torch")

GLOBAL_MODE = 0


def runtime():
    torch.cuda.init()
    for name in ("libcudart.so.12", "libcudart.so"):
        try:
            return C.CDLL(name)
        except OSError:
            continue
    pytest.skip("no shared CUDA runtime")


def make(V, fill):
    g = vx.Graph(V, False)
    b = vx.IncrementalBFS(g, 0)
    rng = np.random.default_rng(8)
    ops = 16_000  # 256,008 entries of the bound a batch, of 4,194,304
    for _ in range(fill):
        b.apply_arrays(rng.integers(0, V, ops, dtype=np.uint32), rng.integers(0, V, ops, dtype=np.uint32),
                       np.ones(ops, np.uint8))
    return g, b


@pytest.mark.parametrize("fill", [1, 6, 7, 8, 9, 10, 11, 12])
def test_a_captured_batch(fill):
    rt = runtime()
    V, n = 200_000, 300
    rng = np.random.default_rng(9)
    batch = (rng.integers(0, V, n, dtype=np.uint32), rng.integers(0, V, n, dtype=np.uint32),
             (rng.random(n) < 0.7).astype(np.uint8))
    dev = [torch.from_numpy(x.view(np.int32) if x.dtype == np.uint32 else x).cuda() for x in batch]
    torch.cuda.synchronize()
    g, b = make(V, fill)
    stream = C.c_void_p()
    assert vx.capi().vx_graph_stream(C.c_void_p(g.handle), C.byref(stream)) == 0
    graph, ex = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamBeginCapture(stream, C.c_int(GLOBAL_MODE)) == 0
    try:
        b.apply_device(*(x.data_ptr() for x in dev), n, V)
    finally:
        ended = rt.cudaStreamEndCapture(stream, C.byref(graph))
    assert ended == 0
    assert rt.cudaGraphInstantiate(C.byref(ex), graph, C.c_ulonglong(0)) == 0
    assert rt.cudaGraphLaunch(ex, stream) == 0
    got = b.distances_array()
    rt.cudaGraphExecDestroy(ex)
    rt.cudaGraphDestroy(graph)
    g1, b1 = make(V, fill)
    b1.apply_arrays(*batch)
    assert np.array_equal(got, b1.distances_array())
    assert g.edge_count_directed() == g1.edge_count_directed()
    b.apply_arrays(*batch)  # and goes on as before
    b1.apply_arrays(*batch)
    assert np.array_equal(b.distances_array(), b1.distances_array())
