"""GPU: room reserved for a stream holds for it.  A readback of what is really
taken allows every entry's row its next blocks, 12 entries for an arc in a row of
its own where the reservation counts 8: it may lower the bound, not raise it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")


@pytest.mark.parametrize("read", [False, True])
def test_a_reserved_stream_of_new_rows_allocates_nothing(read):
    V, ops, batches = 1 << 22, 16_000, 65
    total = ops * batches  # 16.6M entries, a little below the 16.8M the arena grows to
    g = vx.Graph(V, False)
    g.reserve(ops, total)
    b = vx.IncrementalBFS(g, 0)
    size = g.storage_bytes()
    rng = np.random.default_rng(4)
    on = np.ones(ops, np.uint8)
    for t in range(batches):
        b.apply_arrays(rng.integers(0, V, ops, dtype=np.uint32), rng.integers(0, V, ops, dtype=np.uint32), on)
        if read:
            g.edge_count_directed()
        assert g.storage_bytes() == size, t
    assert np.array_equal(b.distances_array(), vx.IncrementalBFS(g, 0).distances_array())
