"""GPU: the full BFS's level kinds at the sizes where they can go wrong -- the
stretches one block runs by itself (in and out of them, back after a wide
level), the grid's top-down levels on either side of the staged frontier's
1,024 vertices, rows expanded by the whole grid, and the first and later
bottom-up levels (forced by the tuning) with isolated vertices, ragged vertex
counts, delta rows, tombstones and directed rows.  Distances against scipy's
unweighted shortest paths."""
import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import dijkstra

import workloads as w

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")

UNREACHED = 0xFFFFFFFF


def expect(edges, V, root, directed):
    e = edges[edges[:, 0] != edges[:, 1]].astype(np.int64)
    m = coo_matrix((np.ones(len(e)), (e[:, 0], e[:, 1])), shape=(V, V)).tocsr()
    m.data[:] = 1
    d = dijkstra(m, directed=directed, indices=root, unweighted=True)
    return np.where(np.isinf(d), UNREACHED, d).astype(np.uint32)


def shape(kind, rng):
    if kind == "path":  # one-block stretches past their 4,096 levels
        V = 9001
        return np.stack((np.arange(V - 1), np.arange(1, V)), 1).astype(np.uint32), V, 0
    if kind == "star":  # one level of 1, one of V - 1; the hub's row goes to one block or the grid
        V = 5000
        return np.stack((np.full(V - 1, 7), np.delete(np.arange(V), 7)), 1).astype(np.uint32), V, 3
    if kind == "hourglass":  # thin, wide (two hubs' rows over the grid), thin again
        a = np.arange(100, 3100)
        e = np.concatenate((np.stack((np.arange(50), np.arange(1, 51)), 1),
                            np.stack((np.full(3000, 50), a), 1), np.stack((a, np.full(3000, 3100)), 1),
                            np.stack((np.arange(3100, 3150), np.arange(3101, 3151)), 1)))
        return e.astype(np.uint32), 3160, 0
    if kind == "fans":  # 1,500 frontier vertices with rows of 1,100 arcs: rows listed for the grid
        hubs = np.arange(1, 1501)
        e = np.concatenate((np.stack((np.zeros(1500, int), hubs), 1),
                            np.stack((np.repeat(hubs, 1100), rng.integers(1501, 20000, 1500 * 1100)), 1)))
        return e.astype(np.uint32), 20011, 0
    if kind == "lattice":
        return w.grid_edges(150, 170, 0.001, seed=5), 150 * 170, 0
    V = 3001 if kind == "rmat-small" else 40003
    e = w.rmat_edges(12 if kind == "rmat-small" else 16, 8, seed=9) % np.uint32(V)
    return e, V, int(e[0, 0])


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("kind", ["path", "star", "hourglass", "fans", "lattice", "rmat-small", "rmat"])
def test_levels(kind, directed):
    rng = np.random.default_rng(4)
    e, V, root = shape(kind, rng)
    g = vx.Graph(V, directed)
    g.bulk_load_edges(e)
    b = vx.IncrementalBFS(g, root)
    want = expect(e, V, root, directed)

    def check(want):
        # the default switch; bottom-up from level 1 on and for as long as it
        # can; bottom-up for one level; top-down only
        for alpha, beta, large in ((14.0, 24.0, 1024), (1e12, 1e12, 64), (1e12, 0.5, 1024), (1e-9, 24.0, 1 << 30)):
            b.set_tuning(alpha, beta, large)
            b.recompute()
            assert np.array_equal(b.distances_array(), want), (kind, directed, alpha, beta, large)
            assert b.reachable_count == int((want != UNREACHED).sum())

    check(want)
    # an overlay: a quarter of a sample of the edges deleted (tombstones), new ones inserted (delta rows)
    k = min(2000, len(e))
    dele = e[rng.choice(len(e), k // 4, replace=False)]
    new = rng.integers(0, V, size=(k, 2), dtype=np.uint32)
    ops = np.concatenate((dele, new))
    g.apply_arrays(ops[:, 0].copy(), ops[:, 1].copy(), np.r_[np.zeros(len(dele), np.uint8), np.ones(k, np.uint8)])
    code = lambda x: (x.astype(np.uint64)[:, 0] << np.uint64(32)) | x[:, 1]  # noqa: E731
    gone = np.isin(code(e), code(dele))
    if not directed:
        gone |= np.isin(code(e[:, ::-1]), code(dele))
    check(expect(np.concatenate((e[~gone], new)), V, root, directed))
