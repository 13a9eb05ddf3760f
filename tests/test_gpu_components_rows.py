"""GPU: the component repair's hook / link / sample / rows passes at the sizes
where they can go wrong -- fewer vertices than samples, ragged bitmap words, no
giant component, a giant that is cut, delta rows and tombstones in front of a
row, and a batch that grows the label array while it cuts components.  Labels
are compared with a union of the mirrored edge set (scipy) after every batch."""
import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import connected_components

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")


def smallest_ids(edges, n):
    e = np.array(sorted(edges), np.int64).reshape(-1, 2)
    _, lab = connected_components(coo_matrix((np.ones(len(e), np.int8), (e[:, 0], e[:, 1])), shape=(n, n)), False)
    first = np.full(lab.max() + 1, n, np.int64)
    np.minimum.at(first, lab, np.arange(n))
    return first[lab]


def shapes(kind, V, rng):
    if kind == "star":  # one hub that every deletion cuts
        hub = V // 2
        return np.array([(hub, v) for v in range(V) if v != hub], np.uint32).reshape(-1, 2)
    if kind == "path":  # long hook chains
        return np.stack((np.arange(V - 1), np.arange(1, V)), 1).astype(np.uint32)
    if kind == "pairs":  # no giant
        v = np.arange(0, V - 1, 2)
        return np.stack((v, v + 1), 1).astype(np.uint32)
    return rng.integers(0, V, size=(2 * V, 2), dtype=np.uint32)  # random


@pytest.mark.parametrize("kind", ["star", "path", "pairs", "random"])
@pytest.mark.parametrize("V", [2, 31, 33, 511, 513, 1020, 5000])
def test_labels_after_every_batch(kind, V):
    rng = np.random.default_rng(V)
    e = shapes(kind, V, rng)
    g = vx.Graph(V, False)
    g.bulk_load_edges(e)
    have = {(min(a, b), max(a, b)) for a, b in e.tolist() if a != b}
    cc = vx.IncrementalComponents(g)
    n = V
    assert np.array_equal(cc.labels_array(), smallest_ids(have, n))
    for t in range(8):
        ops = int(rng.integers(1, 40))
        grown = n + (40 if t == 5 else 0)  # V = 1020: past the labels' first 1,024 slots
        s = rng.integers(0, grown, ops, dtype=np.uint32)
        d = rng.integers(0, grown, ops, dtype=np.uint32)
        a = (rng.random(ops) < 0.5).astype(np.uint8)
        pool = sorted(have)
        for i in np.flatnonzero(a == 0):
            if pool:
                s[i], d[i] = pool[int(rng.integers(len(pool)))]
        before = smallest_ids(have, n)
        pre = set(have)
        final = {}
        for u, v, x in zip(s.tolist(), d.tolist(), a.tolist()):
            if u != v:
                final[(min(u, v), max(u, v))] = x
                n = max(n, u + 1, v + 1)
        have = (have | {k for k, x in final.items() if x}) - {k for k, x in final.items() if not x}
        cut = {int(before[v]) for k, x in final.items() if not x and k in pre for v in k}
        cc.apply_arrays(s, d, a)
        assert np.array_equal(cc.labels_array(), smallest_ids(have, n)), (kind, V, t)
        assert cc.last_repaired_vertices == int(np.isin(before, list(cut)).sum()), (kind, V, t)
