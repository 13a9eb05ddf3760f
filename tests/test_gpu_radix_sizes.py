"""GPU: the radix sort behind bulk loads and large batches at tile edges (4,096
keys) and past the one-block sort (8,192), with keys that are all equal, all
different, and skewed: loaded graphs against numpy's sorted unique arcs, and a
batch's last op per arc past one cluster's canonicalisation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")


@pytest.mark.parametrize("n", [8191, 8192, 8193, 12287, 12288, 12289, 40961, 1 << 20, (1 << 20) + 7])
@pytest.mark.parametrize("kind", ["equal", "wide", "skewed"])
def test_directed_load_is_the_sorted_unique_arcs(n, kind):
    rng = np.random.default_rng(n)
    V = 70_001
    if kind == "equal":
        e = np.tile(np.array([[5, 9]], np.uint32), (n, 1))
    elif kind == "wide":
        e = rng.integers(0, V, (n, 2), dtype=np.uint32)
    else:
        e = (V * rng.random((n, 2)) ** 6).astype(np.uint32)
    g = vx.Graph(V, True)
    g.bulk_load_edges(e)
    a = e[e[:, 0] != e[:, 1]].astype(np.uint64)
    want = np.unique(a[:, 0] << np.uint64(32) | a[:, 1])
    assert g.edge_count_directed() == want.size
    for u in np.unique(np.r_[rng.choice(e[:, 0], 12), [0, 1, 5]]):
        lo, hi = np.searchsorted(want, [int(u) << 32, int(u) + 1 << 32])
        assert g.neighbors(int(u)) == (want[lo:hi] & np.uint64(0xFFFFFFFF)).tolist(), u


def test_last_op_wins_in_a_large_batch():
    rng = np.random.default_rng(3)
    V, ops = 5000, 60_000  # 120,000 arcs, repeats among them
    g = vx.Graph(V, False)
    s = rng.integers(0, 300, ops, dtype=np.uint32)
    d = rng.integers(0, 300, ops, dtype=np.uint32)
    a = (rng.random(ops) < 0.6).astype(np.uint8)
    g.apply_arrays(s, d, a)
    last = {}
    for u, v, x in zip(s.tolist(), d.tolist(), a.tolist()):
        if u != v:
            last[(min(u, v), max(u, v))] = x
    rows = {}
    for (u, v), x in last.items():
        if x:
            rows.setdefault(u, set()).add(v)
            rows.setdefault(v, set()).add(u)
    for u in range(0, 300, 7):
        assert g.neighbors(u) == sorted(rows.get(u, ()))
