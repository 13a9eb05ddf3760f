"""GPU: the delta arena's room.  The host's bound passes the arena's first
4,194,304 entries many times over while the rows themselves stay small, so the
bound is read back from the device (no growth: storage_bytes stands); rows
that keep outgrowing their blocks do make it grow; either way the graph equals
a mirrored edge set and no batch overflows the arena."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("read", [False, True])
def test_steady_rows_do_not_grow_the_arena(directed, read):
    rng = np.random.default_rng(5)
    V, ops = 60_000, 50_000
    g = vx.Graph(V, directed)
    g.bulk_load_edges(rng.integers(0, V, (2 * V, 2), dtype=np.uint32))
    b = vx.IncrementalBFS(g, 0)
    s = rng.integers(0, V, ops, dtype=np.uint32)
    d = rng.integers(0, V, ops, dtype=np.uint32)
    on, off = np.ones(ops, np.uint8), np.zeros(ops, np.uint8)
    b.apply_arrays(s, d, on)
    size = g.storage_bytes()
    for t in range(40):  # 40 x 2 x 50,000 ops: a bound of 32M (64M) entries
        b.apply_arrays(s, d, off)
        b.apply_arrays(s, d, on)
        if read:
            b.stats()
            g.edge_count_directed()
    assert g.storage_bytes() == size
    fresh = vx.IncrementalBFS(g, 0)
    assert np.array_equal(b.distances_array(), fresh.distances_array())


@pytest.mark.parametrize("read", [False, True])
def test_doubling_rows_stay_within_the_arena(read):
    # 2,000 hubs whose delta rows double over and over (their blocks, old ones
    # included, take several times their entries)
    V, hubs, step = 40_000, 2000, 30
    g = vx.Graph(V, True)
    b = vx.IncrementalBFS(g, 0)
    rng = np.random.default_rng(6)
    have = [set() for _ in range(hubs)]
    for t in range(25):
        s = np.repeat(np.arange(hubs, dtype=np.uint32), step)
        d = rng.integers(hubs, V, s.size, dtype=np.uint32)
        b.apply_arrays(s, d, np.ones(s.size, np.uint8))
        for u, v in zip(s.tolist(), d.tolist()):
            have[u].add(v)
        if read:
            g.edge_count_directed()
    for u in (0, 1, 777, hubs - 1):
        assert g.neighbors(u) == sorted(have[u])
    assert g.edge_count_directed() == sum(len(x) for x in have)
    fresh = vx.IncrementalBFS(g, 0)
    assert np.array_equal(b.distances_array(), fresh.distances_array())
