"""GPU: version windows over rows of the lengths at which a pulled row changes
hands -- the group, a warp (256 to 2,047 arcs) or the whole grid -- with arcs
of those rows added and removed inside the window.  Every batch's digest
against the same batches applied one at a time, by the distances."""
import numpy as np
import pytest

from tests.helpers import splitmix_digest as digest

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")

LENGTHS = (1, 8, 9, 128, 255, 256, 257, 511, 2047, 2048, 2049, 5000)


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("window,batches", [(1, 3), (32, 32), (64, 70), (128, 128), (256, 256)])
def test_row_lengths(window, batches, directed):
    rng = np.random.default_rng(batches)
    n, leaves = len(LENGTHS), 6000
    V = n + leaves + 5
    e = [(n + int(x), h) for h, k in enumerate(LENGTHS) for x in rng.choice(leaves, k, replace=False)]
    e += [(h, n + h) for h in range(n)]
    e = np.unique(np.array(e, dtype=np.uint32), axis=0)
    if directed:
        e = np.concatenate([e, e[rng.random(len(e)) < 0.5][:, ::-1]])
    k = 60
    src = np.empty((batches, k), np.uint32)
    dst = np.empty((batches, k), np.uint32)
    for t in range(batches):  # half of the ops on arcs that are there, into hubs
        old = e[rng.integers(0, len(e), size=k // 2)]
        src[t, : k // 2], dst[t, : k // 2] = old[:, 0], old[:, 1]
        src[t, k // 2 :] = rng.integers(0, V, size=k - k // 2)
        dst[t, k // 2 :] = rng.integers(0, n + 50, size=k - k // 2)
    add = (rng.random((batches, k)) < 0.5).astype(np.uint8)
    off = np.arange(batches + 1, dtype=np.uint64) * k
    root = V - 9  # a leaf: the hubs' rows are pulled and pushed

    g = vx.Graph(V, directed)
    g.bulk_load_edges(e)
    b = vx.IncrementalBFS(g, root)
    b.set_stream_window(window)
    digs, _ = b.apply_stream(src.ravel(), dst.ravel(), add.ravel(), off, digests=True)

    g1 = vx.Graph(V, directed)
    g1.bulk_load_edges(e)
    b1 = vx.IncrementalBFS(g1, root)
    for t in range(batches):
        b1.apply_arrays(src[t], dst[t], add[t])
        assert int(digs[t]) == int(digest(b1.distances_array())), f"batch {t}"
    assert np.array_equal(b.distances_array(), b1.distances_array())
