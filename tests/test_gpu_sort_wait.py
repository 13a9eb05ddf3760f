"""GPU: a radix sort whose bounded wait runs out.  With a bound of no looks every
part of the sort but the first gives up at once: the call that sorted must
report it and nothing may be made of the unfinished keys."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("velographx_b200")

DEVICE_ERROR = -5
DEFAULT_LOOKS = 1 << 22


def set_sort_wait(g, looks):
    assert vx.capi().vx_graph_set_sort_wait(C.c_void_p(g.handle), C.c_uint32(looks)) == 0


def load(g, e):
    e = np.ascontiguousarray(e, np.uint32)
    return vx.capi().vx_graph_bulk_load(C.c_void_p(g.handle), e.ctypes.data_as(C.POINTER(C.c_uint32)),
                                        C.c_size_t(len(e)))


def arcs(e, directed):
    a = e[e[:, 0] != e[:, 1]].astype(np.uint64)
    k = a[:, 0] << np.uint64(32) | a[:, 1]
    if not directed:
        k = np.r_[k, a[:, 1] << np.uint64(32) | a[:, 0]]
    return np.unique(k)


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("n", [20_000, 1_000_000])
def test_a_load_reports_it_and_can_be_repeated(n, directed):
    e = np.random.default_rng(n).integers(0, 30_000, (n, 2), dtype=np.uint32)
    g = vx.Graph(30_000, directed)
    set_sort_wait(g, 0)
    for _ in range(3):
        assert load(g, e) == DEVICE_ERROR
        assert "sort" in vx.last_error()
    assert load(g, e[:100]) == 0  # sorted by one block: nothing waits
    set_sort_wait(g, DEFAULT_LOOKS)
    assert load(g, e) == 0
    want = arcs(e, directed)
    assert g.edge_count_directed() == want.size
    for u in (0, 17, 29_999):
        lo, hi = np.searchsorted(want, [u << 32, u + 1 << 32])
        assert g.neighbors(u) == (want[lo:hi] & np.uint64(0xFFFFFFFF)).tolist()
