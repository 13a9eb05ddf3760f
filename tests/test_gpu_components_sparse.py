"""GPU: components of sparse and of evenly random graphs -- no vertex order that
helps, no arc that the first two of a row make redundant, rows on both sides of the
lengths at which a lane and a warp take them, in base and delta rows and behind
tombstones.  And the time of a cut in a uniform graph, whose sets meet at one root."""
import time

import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import connected_components

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")


def smallest_ids(e, n):
    _, lab = connected_components(coo_matrix((np.ones(len(e), np.int8), (e[:, 0], e[:, 1])), shape=(n, n)), False)
    first = np.full(lab.max() + 1, n, np.int64)
    np.minimum.at(first, lab, np.arange(n))
    return first[lab]


def bushes(V, arms, rng):
    """A random recursive tree of hubs with `arms` leaves each, over random ids."""
    hubs = np.arange(0, V, arms + 1)
    up = (hubs[1:] // (arms + 1) * rng.random(len(hubs) - 1)).astype(np.int64) * (arms + 1)
    v = np.arange(V)
    leaf = v[v % (arms + 1) != 0]
    e = np.concatenate((np.stack((hubs[1:], up), 1), np.stack((leaf, leaf - leaf % (arms + 1)), 1)))
    return rng.permutation(V)[e].astype(np.uint32)


@pytest.mark.parametrize("arms", [1, 2, 6, 7, 8, 9, 31, 33])
@pytest.mark.parametrize("V", [257, 3001, 40000])
def test_trees_of_rows_of_every_length(arms, V):
    rng = np.random.default_rng(1000 * arms + V)
    e = bushes(V, arms, rng)
    e.sort(axis=1)
    g = vx.Graph(V, False)
    inside = rng.random(len(e)) < 0.7  # the others come as delta rows
    g.bulk_load_edges(e[inside])
    cc = vx.IncrementalComponents(g)
    assert np.array_equal(cc.labels_array(), smallest_ids(e[inside], V))
    cc.apply_arrays(e[~inside, 0], e[~inside, 1], np.ones((~inside).sum(), np.uint8))
    assert np.array_equal(cc.labels_array(), smallest_ids(e, V))
    there = np.ones(len(e), bool)
    for share in (0.01, 0.3, 0.9):  # each deletion cuts; all come back with the next batch
        cut = rng.random(len(e)) < share
        cut[rng.integers(len(e))] = True
        flip = cut | ~there
        cc.apply_arrays(e[flip, 0], e[flip, 1], (~cut[flip]).astype(np.uint8))
        there = ~cut
        assert np.array_equal(cc.labels_array(), smallest_ids(e[there], V)), share


def test_a_cut_in_a_uniform_graph():
    V, rng = 1 << 20, np.random.default_rng(3)
    e = rng.integers(0, V, (8 * V, 2), dtype=np.uint32)
    g = vx.Graph(V, False)
    g.bulk_load_edges(e)
    cc = vx.IncrementalComponents(g)
    us = []
    for k in range(20):
        t = time.perf_counter()
        cc.apply_arrays(e[100:101, 0], e[100:101, 1], np.full(1, k & 1, np.uint8))
        g.synchronize()
        us.append(1e6 * (time.perf_counter() - t))
    assert np.array_equal(cc.labels_array(), smallest_ids(e, V))
    # 16M arcs once are 30 us; with every thread at one root's word a cut took 1,000
    assert sorted(us[0::2])[3] < 600, us
