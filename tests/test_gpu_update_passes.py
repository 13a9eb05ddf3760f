"""GPU: the update launch's passes against the per-phase path, directed and
undirected, at the batch sizes where they change: one op, the most ops the
launch canonicalises itself (16,384) and one more, past one cluster's
canonicalisation; with hub rows (runs of several arcs, blocks with more arcs
than they process or sort at once, one arc repeated more often than that, delta rows of more than 8 and 32 arcs), repeated ops on one
arc, self-loops, growth, and batches that undo the one before.  After every
batch: distances, counters, edge and delta counts, dirty rows, and the rows
of touched vertices in both directions; at the end the mirrored edge set."""
import numpy as np
import pytest

import workloads as w

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")


def star_batches(rng, V, e, ops):
    """Most ops on one row; then half of a batch on one arc."""
    out = []
    for t in range(2):
        s = np.full(ops, 3, np.uint32)
        d = rng.integers(0, V, ops, dtype=np.uint32)
        s[: ops // 8] = rng.integers(0, V, ops // 8, dtype=np.uint32)
        a = (rng.random(ops) < 0.8).astype(np.uint8)
        p = rng.permutation(ops)
        out += [(s[p], d[p], a[p]), (s[p], d[p], (1 - a[p]).astype(np.uint8))]
        d = d.copy()
        d[ops // 8: ops // 8 + ops // 2] = 17
        out += [(s, d, a), (s[::-1].copy(), d[::-1].copy(), a[::-1].copy())]
    return out


def batches(rng, V, e, ops):
    hubs = np.array([1, 2, 5], np.uint32)
    out = []
    for t in range(3):
        s = rng.integers(0, V, ops, dtype=np.uint32)
        d = rng.integers(0, V, ops, dtype=np.uint32)
        a = (rng.random(ops) < 0.7).astype(np.uint8)
        h = rng.random(ops)
        s[h < 0.2] = rng.choice(hubs, int((h < 0.2).sum()))   # runs in out-rows
        d[h > 0.8] = rng.choice(hubs, int((h > 0.8).sum()))   # and in in-rows
        pick = rng.integers(0, len(e), ops)
        dele = (a == 0) & (rng.random(ops) < 0.7)
        s[dele], d[dele] = e[pick[dele], 0], e[pick[dele], 1]
        rep = rng.random(ops) < 0.1                           # several ops on one arc
        s[rep], d[rep] = s[0], d[0]
        if ops > 4:
            d[3] = s[3]
        if t == 1:
            s[-1] = V + 7  # growth
        out += [(s, d, a), (s, d, (1 - a).astype(np.uint8)), (s[::-1].copy(), d[::-1].copy(), a[::-1].copy())]
    return out


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("star,ops", [(False, n) for n in (1, 33, 512, 1024, 2368, 4800, 16384, 16385, 46000)] +
                         [(True, n) for n in (600, 2100, 2500, 9000, 16384)])
def test_passes_match_the_per_phase_path(star, ops, directed):
    rng = np.random.default_rng(ops + directed)
    V = 20_011
    e = w.rmat_edges(14, 8, seed=3)
    have = {(u, v) for u, v in e.tolist() if u != v}
    if not directed:
        have |= {(v, u) for u, v in have}
    pair = []
    for fused in (True, False):
        g = vx.Graph(V, directed)
        g.bulk_load_edges(e)
        b = vx.IncrementalBFS(g, int(e[0, 0]))
        b.set_fused(fused)
        pair.append((g, b))
    for t, (s, d, a) in enumerate((star_batches if star else batches)(rng, V, e, ops)):
        for u, v, x in zip(s.tolist(), d.tolist(), a.tolist()):
            if u == v:
                continue
            for arc in ((u, v),) if directed else ((u, v), (v, u)):
                have.add(arc) if x else have.discard(arc)
        rows = np.unique(np.concatenate((s[:20], d[:20], [1, 2, 5])))
        seen = []
        for g, b in pair:
            b.apply_arrays(s, d, a)
            st = b.stats()
            if st["last_used_full_recompute"]:
                st.pop("last_affected_vertices")
            st.pop("levels")
            seen.append((b.distances_array().tobytes(), st, g.edge_count_directed(), g.delta_edge_count(),
                         g.dirty_out_segment_count(), g.dirty_in_segment_count(), g.version, g.vertex_count,
                         [g.neighbors(int(r)) for r in rows], [g.in_neighbors(int(r)) for r in rows]))
        assert seen[0] == seen[1], (ops, directed, t)
    g, b = pair[0]
    assert g.edge_count_directed() == len(have)
    out = {}
    for u, v in have:
        out.setdefault(u, []).append(v)
    for r in list(range(0, 60)) + sorted(out)[-20:]:
        assert g.neighbors(r) == sorted(out.get(r, [])), r
    fresh = vx.IncrementalBFS(g, int(e[0, 0]))
    assert np.array_equal(b.distances_array(), fresh.distances_array())
