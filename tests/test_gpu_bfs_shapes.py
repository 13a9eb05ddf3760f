"""GPU: the full BFS on graphs of one shape: stars, wide trees, lattices of a
frontier's width.  Which direction their levels take (the level trace), and how
their times compare with a graph of the same or of more work."""
import numpy as np
import pytest

import workloads as w

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")

V = 1 << 18


def star(hub):
    leaves = np.setdiff1d(np.arange(V, dtype=np.uint32), [hub]).astype(np.uint32)
    return np.stack((np.full(V - 1, hub, np.uint32), leaves), 1)


def tree(arity, vertices=V):
    v = np.arange(1, vertices, dtype=np.uint32)
    return np.stack(((v - 1) // arity, v), 1).astype(np.uint32)


def lattice(width, rows):
    idx = np.arange(width * rows, dtype=np.uint32).reshape(rows, width)
    return np.concatenate((np.stack((idx[:, :-1].ravel(), idx[:, 1:].ravel()), 1),
                           np.stack((idx[:-1].ravel(), idx[1:].ravel()), 1)))


def search(vertices, e, root):
    g = vx.Graph(vertices, False)
    g.bulk_load_edges(e)
    return g, vx.IncrementalBFS(g, root)


def tree_depth(arity):
    d = np.zeros(V, np.uint32)
    for v in range(1, V):  # parents come first
        d[v] = d[(v - 1) // arity] + 1
    return d


@pytest.mark.parametrize("arity", [8, 64, 1000])
def test_the_last_wide_level_of_a_tree_goes_bottom_up(arity):
    g, b = search(V, tree(arity), 0)
    depth = tree_depth(arity)
    assert np.array_equal(b.distances_array(), depth)
    levels = b.level_trace()  # (us, frontier, bottom-up)
    sizes = np.bincount(depth)
    assert [n for _, n, _ in levels] == sizes.tolist()
    left = V - np.cumsum(sizes)
    wide = (left <= 4 * sizes) & (V <= 16 * sizes) & (sizes > 1024)
    assert wide.any()
    assert all(up for (_, _, up), x in zip(levels, wide) if x), levels


@pytest.mark.parametrize("root", [0, 77])
def test_a_star_is_swept_not_pushed(root):
    hub = 77
    g, b = search(V, star(hub), root)
    want = np.full(V, 1 if root == hub else 2, np.uint32)
    want[hub], want[root] = (0, 0) if root == hub else (1, 0)
    assert np.array_equal(b.distances_array(), want)
    levels = b.level_trace()
    assert levels[-1][2], levels          # the leaves
    if root != hub:
        assert levels[1][2], levels       # the hub, whose row holds nearly as many arcs as there are vertices


def test_a_lattice_is_pushed():
    g, b = search(1000 * 1000, lattice(1000, 1000), 0)
    r, c = np.divmod(np.arange(10**6, dtype=np.uint32), 1000)
    assert np.array_equal(b.distances_array(), r + c)
    assert not any(up for _, _, up in b.level_trace())


def test_a_hub_of_a_million_leaves_is_pushed_at_the_rate_of_the_memory():
    vertices = 1 << 20
    hub = np.stack((np.full(vertices - 1, vertices - 1), np.arange(vertices - 1)), 1).astype(np.uint32)
    g, b = search(vertices, hub, vertices - 1)
    us = []
    for _ in range(20):
        b.recompute()
        us.append(b.level_trace()[0][0])
    # 2^20 claims: some 45 us are their atomics; with too few arcs in flight 118
    assert min(us) < 80, us


def test_a_level_of_a_thousand_vertices_takes_no_longer_than_one_of_two_thousand():
    # a root with an arc to every vertex of a lattice's first row: each level is a row
    rows, level = 200, []
    for width in (1024, 2048):
        e = np.concatenate((lattice(width, rows) + np.uint32(1),
                            np.stack((np.zeros(width), np.arange(1, width + 1)), 1).astype(np.uint32)))
        g, b = search(1 + width * rows, e, 0)
        want = np.r_[0, np.repeat(np.arange(1, rows + 1), width)].astype(np.uint32)
        assert np.array_equal(b.distances_array(), want)
        best = np.full(rows + 1, np.inf)
        for _ in range(6):
            b.recompute()
            best = np.minimum(best, [us for us, _, _ in b.level_trace()])
        level.append(np.median(best[20:-20]))
    # half of the arcs: by one block alone such a level took twice as long as the wider one
    assert level[0] < 1.05 * level[1], level
