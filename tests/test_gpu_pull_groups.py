"""GPU: how the warps share out the vertex groups of a pull level -- fewer groups than
warps, as many, and more, with little and with much to do in each -- for multi-root
BFS and for version windows.  And the time of a level that reaches nothing new."""
import numpy as np
import pytest

import workloads as w

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")

WARPS = 2 * 148 * 16  # of the launch: two blocks of 16 warps per SM
SIZES = [33, 32 * WARPS - 1, 32 * WARPS + 1, 32 * (WARPS + 1) + 1, 32 * (3 * WARPS + 2) - 5]


def graph(kind, V, rng):
    if kind == "pairs":
        v = rng.permutation(V)[: V // 2 * 2].astype(np.uint32)
        return v.reshape(-1, 2)
    if kind == "star":
        return np.stack((np.full(V - 1, V - 1), np.arange(V - 1)), 1).astype(np.uint32)
    # uniform, and dense at the smallest ids: heavy groups side by side
    e = rng.integers(0, V, (2 * V, 2))
    e[: V // 2] //= 64
    return e.astype(np.uint32)


@pytest.mark.parametrize("kind", ["pairs", "star", "skewed"])
@pytest.mark.parametrize("V", SIZES)
def test_multi_root_levels_all_pulled(kind, V):
    rng = np.random.default_rng(V)
    e = graph(kind, V, rng)
    g = vx.Graph(V, False)
    g.bulk_load_edges(e)
    roots = e[rng.integers(0, len(e), 3), 0]
    mr = vx.MultiRootBFS(g, roots)
    mr.set_pull_fraction(1e-9)
    mr.run()
    assert all(pull for _, _, pull in mr.level_trace())
    got = mr.distances_array().reshape(3, V)
    for k, r in enumerate(roots):
        assert np.array_equal(got[k], w.bfs_levels(e, V, int(r))), k


@pytest.mark.parametrize("kind", ["pairs", "star", "skewed"])
@pytest.mark.parametrize("V", SIZES)
def test_window_levels_all_pulled(kind, V):
    rng = np.random.default_rng(V + 1)
    e = graph(kind, V, rng)
    st = w.mixed_stream(e, V, [5, 40, 1, 17, 30, 9], 0.6, seed=V)
    off = np.asarray(st.offsets, np.uint64)
    out = []
    for window in (256, 0):
        g = vx.Graph(V, False)
        g.bulk_load_edges(e)
        b = vx.IncrementalBFS(g, int(e[0, 0]))
        b.set_stream_window(window)
        b.set_window_pull_fraction(1e-9)
        digests, _ = b.apply_stream(st.src, st.dst, st.add, off, digests=True, stats=False)
        out.append((digests.copy(), b.distances_array()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


def test_a_level_that_reaches_nothing_new_is_a_sweep():
    V = 1 << 20
    g = vx.Graph(V, False)
    g.bulk_load_edges(graph("star", V, None))
    mr = vx.MultiRootBFS(g, np.array([V - 1], np.uint32))
    us = []
    for _ in range(20):
        mr.run()
        last = mr.level_trace()[-1]
        assert last[1] == V - 1 and last[2]
        us.append(last[0])
    # 2^20 visited words are read: 17 to 22 us; a claim of the counter per group made it 33
    assert min(us) < 27, us
