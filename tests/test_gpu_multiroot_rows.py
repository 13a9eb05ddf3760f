"""GPU: the multi-root BFS's ways through a row at the lengths where they
change -- the roots' rows that a warp or the whole grid pushes, and the pulled
rows that a group, a warp or the whole grid reads (255 to 257 and 2,047 to
2,049 arcs) -- for one to eight words of roots, with rows in the base, in the
delta rows and across both, reached by every root at once, by half of them and
by one.  Distances against scipy's unweighted shortest paths."""
import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import dijkstra

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")

UNREACHED = 0xFFFFFFFF
LENGTHS = (1, 8, 9, 94, 95, 96, 97, 128, 129, 255, 256, 257, 511, 2047, 2048, 2049, 5000)


def expect(edges, V, roots, directed):
    m = coo_matrix((np.ones(len(edges)), (edges[:, 0], edges[:, 1])), shape=(V, V)).tocsr()
    m.data[:] = 1
    inside = sorted({int(r) for r in roots if r < V})
    d = dijkstra(m, directed=directed, indices=inside, unweighted=True)
    rows = {r: np.where(np.isinf(x), UNREACHED, x).astype(np.uint32) for r, x in zip(inside, d)}
    return np.stack([rows.get(int(r), np.full(V, UNREACHED, np.uint32)) for r in roots])


def hubs(rng, directed):
    """A hub of each length over shared leaves, a ring through the hubs, and
    tails behind some leaves; with reversed arcs as well when directed, half of
    them left out."""
    n = len(LENGTHS)
    leaves, tails = 6000, 40
    V = n + leaves + tails + 3  # the last 3 stay isolated
    e = [(n + int(x), h) for h, k in enumerate(LENGTHS) for x in rng.choice(leaves, k, replace=False)]
    e += [(h, (h + 1) % n) for h in range(n)]
    e += [(n + leaves + t, n + int(rng.integers(leaves))) for t in range(tails)]
    e = np.array(e, dtype=np.uint32)
    if directed:
        back = e[rng.random(len(e)) < 0.5][:, ::-1]
        e = np.concatenate([e, back])
    return np.unique(e, axis=0), V


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("k", [1, 32, 33, 64, 100, 256])
def test_row_lengths(k, directed):
    rng = np.random.default_rng(k)
    e, V = hubs(rng, directed)
    first = rng.random(len(e)) < 0.9
    g = vx.Graph(V, directed)
    g.bulk_load_edges(e[first])
    late = e[~first]  # into the delta rows
    g.apply_arrays(late[:, 0], late[:, 1], np.ones(len(late), np.uint8))
    roots = rng.integers(0, V, size=k).astype(np.uint32)
    roots[: min(k, len(LENGTHS)) // 2] = np.arange(min(k, len(LENGTHS)) // 2)  # hubs
    if k > 3:
        roots[-1] = V + 7
        roots[-2] = roots[-3]
    m = vx.MultiRootBFS(g, roots)
    exp = expect(e, V, roots, directed)
    for run in range(2):
        m.run()
        assert np.array_equal(m.distances_array(), exp), f"run {run}"
