"""GPU: version windows over rows on both sides of the lengths from which a warp (256
arcs) and the whole grid (2,048) read them, part of each row in its delta list before
the window begins, some of its base arcs removed.  Digests and distances equal those of
the batches applied one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")


@pytest.mark.parametrize("length", [255, 256, 257, 2047, 2048, 2049])
def test_long_rows_with_delta_arcs(length):
    rng = np.random.default_rng(length)
    V, hubs = 6000, np.arange(4, dtype=np.uint32)
    rows = [rng.choice(np.arange(10, V, dtype=np.uint32), length, replace=False) for _ in hubs]
    path = np.stack((np.arange(4, 9), np.arange(5, 10)), 1).astype(np.uint32)  # the source is 4
    base = np.concatenate([np.stack((np.full(length - 9, h), r[9:]), 1) for h, r in zip(hubs, rows)] + [path])
    late = np.concatenate([np.stack((np.full(9, h), r[:9]), 1) for h, r in zip(hubs, rows)])
    gone = np.concatenate([np.stack((np.full(2, h), r[20:22]), 1) for h, r in zip(hubs, rows)])
    first = np.concatenate((late, gone, [[9, rows[0][0]]])).astype(np.uint32)
    n = 8 * 12
    s = np.where(rng.random(n) < 0.5, rng.choice(hubs, n), rng.integers(4, V, n)).astype(np.uint32)
    d = rng.integers(4, V, n).astype(np.uint32)
    back = rng.random(n) < 0.3  # arcs of the rows go and come
    pick = base[rng.integers(0, len(base), n)]
    s, d = np.where(back, pick[:, 0], s).astype(np.uint32), np.where(back, pick[:, 1], d).astype(np.uint32)
    a = (rng.random(n) < 0.5).astype(np.uint8)
    off = (np.arange(9) * 12).astype(np.uint64)
    out = []
    for window in (256, 0):
        g = vx.Graph(V, False)
        g.bulk_load_edges(base.astype(np.uint32))
        b = vx.IncrementalBFS(g, 4)
        b.apply_arrays(first[:, 0].copy(), first[:, 1].copy(), np.r_[np.ones(36), np.zeros(8), 1].astype(np.uint8))
        b.set_stream_window(window)
        b.set_window_pull_fraction(1e-9)
        digests, _ = b.apply_stream(s, d, a, off, digests=True, stats=False)
        out.append((digests.copy(), b.distances_array()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
