"""The calls this library is timed on, through its public entry points.

A case is one workload of the dynamic-BFS path with its sizes:

  update      ``IncrementalBFS`` update batches, the library's main use.  One
              pass applies two batches: the one that takes back what the
              state's last batch did (its ops with insertion and deletion
              swapped) and that batch again.  A pass therefore starts and ends
              in the same graph, and both directions are timed: a 70%-insertion
              batch and its 70%-deletion counterpart.
  bfs         a full BFS (``recompute``) of a loaded graph.
  multiroot   one bit-parallel traversal from many roots.
  stream      ``apply_stream`` over a whole stream of lognormal-sized batches
              with a digest per batch; its second half takes the first back.
  components  ``IncrementalComponents`` update batches and the label read.
  load        an edge array on the host to a graph, its first BFS and the
              distances back on the host: a program's first answer.

Graphs are R-MAT (a, b, c = 0.57, 0.19, 0.19, edge factor 16 unless said, ids
folded to ``vertices``) or the 4-neighbour lattice with 0.1% random long-range
edges, as in the benchmark's configurations.  Lattice batches delete edges
drawn from the 1/64 nearest the root, so their repairs cascade; R-MAT batches
delete uniformly drawn loaded edges.  Every output is a whole number.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import velographx_b200 as vx

EDGE_FACTOR = 16


def listed():
    return [
        # a small service graph fed by trickling insertions (64 per batch): pure latency
        {"name": "update-16k-64-inserts", "kind": "update", "graph": "rmat", "vertices": 1 << 14, "ops": 64,
         "insert": 1.0, "directed": False, "arrays": "host"},
        # the median batch of the lognormal stream, one call at a time with its counters read
        {"name": "update-1m-475", "kind": "update", "graph": "rmat", "vertices": 1 << 20, "ops": 475,
         "insert": 0.7, "directed": False, "arrays": "host"},
        # the headline: 10,000-op batches that are already in device memory
        {"name": "update-4m-10k", "kind": "update", "graph": "rmat", "vertices": 1 << 22, "ops": 10_000,
         "insert": 0.7, "directed": False, "arrays": "device"},
        # a bulk refresh: batches past one cluster's canonicalisation
        {"name": "update-1m-100k", "kind": "update", "graph": "rmat", "vertices": 1 << 20, "ops": 100_000,
         "insert": 0.7, "directed": False, "arrays": "host"},
        # a directed graph (two adjacencies) with a ragged vertex count
        {"name": "update-directed-300k-1000", "kind": "update", "graph": "rmat", "vertices": 300_007, "ops": 1000,
         "insert": 0.7, "directed": True, "arrays": "host"},
        # a road-like graph with near-root deletions: long cascades and relaxations
        {"name": "update-lattice-2048-1000", "kind": "update", "graph": "lattice", "vertices": 2048 * 2048,
         "ops": 1000, "insert": 0.5, "directed": False, "arrays": "host"},
        # full recompute of a skewed, shallow graph and of a deep one
        {"name": "bfs-4m", "kind": "bfs", "graph": "rmat", "vertices": 1 << 22, "directed": False},
        {"name": "bfs-lattice-4096", "kind": "bfs", "graph": "lattice", "vertices": 4096 * 4096, "directed": False},
        # distances from 64 sources at once (landmarks, centrality samples)
        {"name": "multiroot-4m-64", "kind": "multiroot", "graph": "rmat", "vertices": 1 << 22, "roots": 64},
        # replay of a recorded stream: 512 batches of lognormal size (median 500, sigma 2)
        {"name": "stream-1m-512", "kind": "stream", "graph": "rmat", "vertices": 1 << 20, "batches": 512,
         "median": 500, "counters": False},
        # component labels kept up to date beside the graph
        {"name": "components-1m-1000", "kind": "components", "graph": "rmat", "vertices": 1 << 20, "ops": 1000,
         "insert": 0.7},
        # a program's start: 16.8M edges from a numpy array to the first distances
        {"name": "load-1m", "kind": "load", "graph": "rmat", "vertices": 1 << 20, "directed": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("update", "update", "update", "bfs", "multiroot", "stream", "components", "load"))
    if kind == "update":
        directed = rng.random() < 0.25
        lattice = not directed and rng.random() < 0.25
        v = _log(rng, 64, 2048) ** 2 if lattice else _log(rng, 1 << 12, 1 << (20 if directed else 22))
        return {"kind": kind, "graph": "lattice" if lattice else "rmat", "vertices": v,
                "ops": min(_log(rng, 1, 100_000), v // (64 if lattice else 4)),
                "insert": rng.choice((1.0, 0.7, 0.5, 0.3)), "directed": directed,
                "arrays": rng.choice(("host", "device"))}
    if kind == "bfs":
        if rng.random() < 0.35:
            return {"kind": kind, "graph": "lattice", "vertices": _log(rng, 32, 4096) ** 2, "directed": False}
        return {"kind": kind, "graph": "rmat", "vertices": _log(rng, 1 << 10, 1 << 22), "directed": rng.random() < 0.25}
    if kind == "multiroot":
        return {"kind": kind, "graph": "rmat", "vertices": _log(rng, 1 << 12, 1 << 20), "roots": _log(rng, 2, 256)}
    if kind == "stream":
        return {"kind": kind, "graph": "rmat", "vertices": _log(rng, 1 << 12, 1 << 20), "batches": _log(rng, 8, 512),
                "median": _log(rng, 16, 500), "counters": rng.random() < 0.25}
    if kind == "components":
        v = _log(rng, 1 << 12, 1 << 20)
        return {"kind": kind, "graph": "rmat", "vertices": v, "ops": min(_log(rng, 1, 20_000), v // 4),
                "insert": rng.choice((1.0, 0.7, 0.3))}
    return {"kind": kind, "graph": "rmat", "vertices": _log(rng, 1 << 10, 1 << 20), "directed": rng.random() < 0.25}


# ---------------------------------------------------------------- inputs ----

def _rmat(vertices, gen):
    """(16 * vertices, 2) int32 R-MAT pairs on the GPU, self-loops and duplicates kept."""
    scale = max(1, (vertices - 1).bit_length())
    n = EDGE_FACTOR * vertices
    u = torch.zeros(n, dtype=torch.int32, device="cuda")
    v = torch.zeros(n, dtype=torch.int32, device="cuda")
    for _ in range(scale):
        r = torch.rand(n, generator=gen, device="cuda")
        low = r >= 0.76
        u.mul_(2).add_(low)
        v.mul_(2).add_(((r >= 0.57) & ~low) | (r >= 0.95))
    if vertices != 1 << scale:
        u.remainder_(vertices)
        v.remainder_(vertices)
    return torch.stack((u, v), 1)


def _lattice(vertices, gen):
    """Side x side lattice edges and 0.1% uniform long-range ones."""
    side = math.isqrt(vertices)
    idx = torch.arange(side * side, dtype=torch.int32, device="cuda").view(side, side)
    right = torch.stack((idx[:, :-1].reshape(-1), idx[:, 1:].reshape(-1)), 1)
    down = torch.stack((idx[:-1].reshape(-1), idx[1:].reshape(-1)), 1)
    extra = int(round(0.001 * (right.shape[0] + down.shape[0])))
    far = torch.randint(0, vertices, (extra, 2), generator=gen, dtype=torch.int32, device="cuda")
    return torch.cat((right, down, far))


def _edges(case, gen):
    return (_lattice if case["graph"] == "lattice" else _rmat)(case["vertices"], gen)


def _graph(case, uv):
    g = vx.Graph(case["vertices"], case.get("directed", False))
    torch.cuda.synchronize()  # the edge array comes from torch's stream, the load runs on the graph's
    rc = vx.capi().vx_graph_bulk_load_device(ctypes.c_void_p(g.handle), ctypes.c_void_p(uv.data_ptr()),
                                             ctypes.c_size_t(uv.shape[0]))
    if rc:
        raise RuntimeError(vx.last_error())
    g.synchronize()
    return g


def _root(case, uv, gen):
    """The lattice's corner, or an endpoint of a random edge."""
    if case["graph"] == "lattice":
        return 0
    return int(uv[int(torch.randint(0, uv.shape[0], (1,), generator=gen, device="cuda")), 0])


def _ops(pool, vertices, ops, insert, gen):
    """`ops` update ops: uniform random insertions, and deletions drawn from the
    edges `pool`, mixed.  Returns host numpy arrays (src, dst, add)."""
    uv = torch.randint(0, vertices, (ops, 2), generator=gen, dtype=torch.int32, device="cuda")
    add = torch.rand(ops, generator=gen, device="cuda") < insert
    pick = torch.randint(0, pool.shape[0], (ops,), generator=gen, device="cuda")
    uv = torch.where(add[:, None], uv, pool[pick])
    src, dst = uv.t().contiguous().cpu().numpy().view(np.uint32)
    return src.copy(), dst.copy(), add.to(torch.uint8).cpu().numpy()


class _DeviceArray:
    """A device pointer as something torch can wrap without a copy.  The tensor
    keeps this object, and so the owner of the memory, alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i4", "data": (ptr, False), "version": 2}


def _view(state, ptr, shape, owner):
    """The owner's own buffer as a tensor, wrapped anew only when it moved."""
    if state.get("view_of") != (ptr, shape):
        state["view"] = torch.as_tensor(_DeviceArray(ptr, shape, owner), device="cuda")
        state["view_of"] = (ptr, shape)
    return state["view"]


def _distances(state):
    ptr, n = state["bfs"].distances_device_ptr()
    return _view(state, ptr, (n,), state["bfs"])


# --------------------------------------------------------------- prepare ----

def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    uv = _edges(case, gen)
    kind, vertices = case["kind"], case["vertices"]
    state = {"kind": kind, "vertices": vertices}
    if kind == "load":
        state["edges"] = uv.cpu().numpy().view(np.uint32)
        state["directed"] = case["directed"]
        state["root"] = _root(case, uv, gen)
        return state
    g = state["graph"] = _graph(case, uv)
    if kind == "multiroot":
        pick = torch.randint(0, uv.shape[0], (case["roots"],), generator=gen, device="cuda")
        roots = uv[pick, 0].cpu().numpy().view(np.uint32).copy()
        state["mr"] = _MultiRoot(g, roots)
        return state
    if kind == "components":
        src, dst, add = _ops(uv, vertices, case["ops"], case["insert"], gen)
        state["cc"] = vx.IncrementalComponents(g)
        state["batches"] = [(src, dst, (1 - add).astype(np.uint8)), (src, dst, add)]
        state["cc"].apply_arrays(src, dst, add)
        return state
    bfs = state["bfs"] = vx.IncrementalBFS(g, _root(case, uv, gen))
    if kind == "bfs":
        return state
    if kind == "stream":
        rng = np.random.default_rng(seed)
        half = max(1, case["batches"] // 2)
        sizes = np.clip(np.rint(np.exp(math.log(case["median"]) + 2.0 * rng.standard_normal(half))), 1,
                        min(200_000, vertices)).astype(np.int64)
        src, dst, add = _ops(uv, vertices, int(sizes.sum()), 0.7, gen)
        state["src"] = np.concatenate((src, src[::-1]))
        state["dst"] = np.concatenate((dst, dst[::-1]))
        state["add"] = np.concatenate((add, 1 - add[::-1])).astype(np.uint8)
        state["offsets"] = np.concatenate(([0], np.cumsum(np.concatenate((sizes, sizes[::-1]))))).astype(np.uint64)
        state["counters"] = case["counters"]
        g.reserve(int(sizes.max()), 2 * int(sizes.sum()))
        run(state)  # the stream's own end state is where every pass starts
        return state
    if case["graph"] == "lattice":
        d = _distances(state).to(torch.int64)
        far = torch.maximum(d[uv[:, 0].long()], d[uv[:, 1].long()])
        uv = uv[torch.argsort(far, stable=True)[: max(case["ops"], uv.shape[0] // 64)]]
    src, dst, add = _ops(uv, vertices, case["ops"], case["insert"], gen)
    g.reserve(case["ops"], 4 * case["ops"])
    state["batches"] = [(src, dst, (1 - add).astype(np.uint8)), (src, dst, add)]
    if case["arrays"] == "device":
        dev = [tuple(torch.from_numpy(x.view(np.int32) if x.dtype == np.uint32 else x).cuda() for x in b)
               for b in state["batches"]]
        state["device"] = dev
        state["batches"] = None
        state["pointers"] = [tuple(x.data_ptr() for x in b) for b in dev]
        torch.cuda.synchronize()
    bfs.apply_arrays(src, dst, add)
    return state


class _MultiRoot:
    """A multi-root handle of the C interface, whose distances stay on the device."""

    def __init__(self, graph, roots):
        self.graph, self.roots = graph, roots
        self.handle = ctypes.c_void_p()
        self._check(vx.capi().vx_mrbfs_create(ctypes.c_void_p(graph.handle),
                                              roots.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)),
                                              ctypes.c_size_t(roots.size), ctypes.byref(self.handle)))

    def __del__(self):
        vx.capi().vx_mrbfs_destroy(self.handle)

    @staticmethod
    def _check(rc):
        if rc:
            raise RuntimeError(vx.last_error())

    def run(self):
        self._check(vx.capi().vx_mrbfs_run(self.handle))

    def pointer(self):
        p, n = ctypes.c_void_p(), ctypes.c_size_t()
        self._check(vx.capi().vx_mrbfs_distances_device(self.handle, ctypes.byref(p), ctypes.byref(n)))
        return p.value, n.value


# ------------------------------------------------------------------- run ----

def _counters(bfs):
    """A batch's counters as a caller reads them after it.  A repair that fell
    back to a full recompute stops counting affected vertices at an
    unspecified point past the limit, so that count is left out."""
    s = bfs.stats()
    full = bool(s["last_used_full_recompute"])
    return [s["reachable_count"], s["last_deletion_candidates"], -1 if full else s["last_affected_vertices"], int(full)]


def run(state):
    kind = state["kind"]
    if kind == "update":
        bfs = state["bfs"]
        if state["batches"] is None:
            n = state["device"][0][0].numel()
            for src, dst, add in state["pointers"]:
                bfs.apply_device(src, dst, add, n, state["vertices"])
            return {"distances": _distances(state)}
        counters = []
        for src, dst, add in state["batches"]:
            bfs.apply_arrays(src, dst, add)
            counters.append(_counters(bfs))
        return {"distances": _distances(state), "counters": np.array(counters, np.int64)}
    if kind == "bfs":
        state["bfs"].recompute()
        return {"distances": _distances(state)}
    if kind == "multiroot":
        mr = state["mr"]
        mr.run()
        ptr, n = mr.pointer()
        return {"distances": _view(state, ptr, (n,), mr)}
    if kind == "stream":
        digests, stats = state["bfs"].apply_stream(state["src"], state["dst"], state["add"], state["offsets"],
                                                   digests=True, stats=state["counters"])
        out = {"distances": _distances(state), "digests": digests.view(np.int64)}
        if state["counters"]:
            # candidates, affected (unspecified after a fallback), fallback, reachable
            st = stats.astype(np.int64)
            st[st[:, 2] != 0, 1] = -1
            out["counters"] = st
        return out
    if kind == "components":
        cc = state["cc"]
        repaired = []
        for src, dst, add in state["batches"]:
            cc.apply_arrays(src, dst, add)
            repaired.append(cc.last_repaired_vertices)
        return {"labels": cc.labels_array().view(np.int32), "repaired": np.array(repaired, np.int64)}
    g = vx.Graph(state["vertices"], state["directed"])
    g.bulk_load_edges(state["edges"])
    bfs = vx.IncrementalBFS(g, state["root"])
    return {"distances": bfs.distances_array().view(np.int32), "arcs": g.edge_count_directed()}


# ------------------------------------------------------------------ work ----

def work(case):
    """Bytes a pass cannot do without: the op arrays (9 B an op) and the arcs
    they change, the graph's offsets and arcs where the whole graph is
    traversed (duplicate R-MAT pairs, a few percent, counted as arcs), and
    every result once.  No path does floating-point work."""
    v, kind = case["vertices"], case["kind"]
    sides = 1 if case.get("directed", False) else 2
    edges = (2 * v) if case["graph"] == "lattice" else EDGE_FACTOR * v
    traversal = 4.0 * sides * edges + 8.0 * (v + 1)
    if kind in ("update", "components"):
        b = 2.0 * case["ops"] * (9 + 4 * 2)
        b += 4.0 * v if kind == "components" else 0.0
    elif kind == "bfs":
        b = traversal + 4.0 * v
    elif kind == "multiroot":
        b = traversal + 4.0 * v * case["roots"]
    elif kind == "stream":
        ops = case["batches"] * min(float(v), case["median"] * math.exp(2.0))
        b = ops * (9 + 4 * 2) + 4.0 * v + 8.0 * case["batches"]
    else:
        b = 8.0 * edges + traversal + 4.0 * v
    return {"bytes": b, "flops": 0.0}
