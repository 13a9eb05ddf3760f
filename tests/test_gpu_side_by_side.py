"""GPU: update launches of several graphs running side by side (each graph has
its own stream, so blocks of one launch start, wait and read the phase words at
very different times): every batch's counters and digest equal those of the same
batch applied alone, and no wait of any launch expires."""
import numpy as np
import pytest

import workloads as w

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")


@pytest.mark.parametrize("ops", [300, 3000])
def test_interleaved_graphs_match_one_at_a_time(ops):
    torch = pytest.importorskip("torch")
    V = 1 << 16
    sets = []
    for seed in range(3):
        e = w.rmat_edges(16, 8, seed=seed)
        st = w.mixed_stream(e, V, [ops] * 40, 0.6, seed=seed + 9)
        sets.append((e, st, w.max_degree_root(e, V)))

    def make(e, root):
        g = vx.Graph(V, False)
        g.bulk_load_edges(e)
        g.reserve(ops, 40 * ops)
        return g, vx.IncrementalBFS(g, root)

    alone = []
    for e, st, root in sets:
        g, b = make(e, root)
        rec = []
        for t in range(st.batches):
            b.apply_arrays(*st.batch(t))
            s = b.stats()
            rec.append((s["reachable_count"], s["last_deletion_candidates"], s["last_affected_vertices"]))
        alone.append((rec, b.digest()))
    objs = [make(e, root) for e, _, root in sets]
    dev = []
    for _, st, _ in sets:
        dev.append(tuple(torch.from_numpy(x.view(np.int32) if x.dtype == np.uint32 else x).cuda()
                         for x in (st.src, st.dst, st.add)))
    torch.cuda.synchronize()
    for t in range(40):
        for (g, b), (_, st, _), (s, d, a) in zip(objs, sets, dev):
            o = int(st.offsets[t])
            b.apply_device(s.data_ptr() + 4 * o, d.data_ptr() + 4 * o, a.data_ptr() + o, ops, V)
        if t % 8 == 7:  # the counters of this batch, the batches between only queued
            for k, (g, b) in enumerate(objs):
                c = b.stats()
                assert (c["reachable_count"], c["last_deletion_candidates"],
                        c["last_affected_vertices"]) == alone[k][0][t], (k, t)
    for k, (g, b) in enumerate(objs):
        assert b.digest() == alone[k][1], k
