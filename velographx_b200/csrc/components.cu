// Connected components of an undirected device graph, maintained across
// update batches (the reference's BasicIncrementalComponents,
// include/velographx/incremental/connected_components.hpp:16-165).
//
// Labels live in device memory as a compressed union-find forest: label[v] is
// the root of v's set, and every union hooks the larger root under the smaller
// one (atomicCAS), so a root is always the smallest vertex id of its
// component.  A batch is applied as the reference applies it:
//   1. the batch is canonicalised and classified against the pre-batch graph
//      (the graph's own staging: last op per edge, present-before bit);
//   2. the components of the endpoints of every effective deletion are marked
//      affected, and their vertices counted (last_repaired_vertices);
//   3. the batch is committed to the graph;
//   4. affected vertices are united anew along their arcs to other affected
//      vertices in the post-batch graph (unite_rows below);
//   5. the final additions are united;
//   6. every label is compressed to its root.
// Nothing of this waits on the host: without an effective deletion the kernels
// of steps 2 and 4 return at once, and the affected count is read when asked.
// The partition equals the reference's after every batch.  The labels are the
// components' smallest ids, where the reference's are whichever union-find
// roots its union order left (the reference's tests compare labels only for
// equality).
#include <algorithm>
#include <cstring>

#include "components.cuh"
#include "frontier.cuh"
#include "graph_dev.cuh"

namespace vxh {

namespace {

constexpr int kCcThreads = 256;

unsigned cc_grid(uint64_t n) {
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + kCcThreads - 1) / kCcThreads, 148ull * 64));
}

// Unites the sets of a and b (Rem's algorithm with splicing; concurrent as in
// Dhulipala, Hong and Shun, "ConnectIt", VLDB 2020).  The end with the larger parent
// goes under the other's parent; if it was no root, its old parent's set is still to
// be united, so the walk goes on from there.  Parents only ever move to smaller ids,
// and the walk ends where the parents are equal: without looking at the root, whose
// word all threads would load once the sets have grown together.  cc_link_kernel on
// a uniform graph of 2^20 vertices and 8M edges 763 to 1,123 us with a find of both
// roots, 125 so.
__device__ __forceinline__ void cc_union(uint32_t* label, uint32_t a, uint32_t b) {
  uint32_t pa = __ldcg(&label[a]), pb = __ldcg(&label[b]);
  while (pa != pb) {
    if (pa < pb) {
      const uint32_t t = a, tp = pa;
      a = b;
      pa = pb;
      b = t;
      pb = tp;
    }
    const uint32_t old = atomicMin(&label[a], pb);
    if (old == a) return;  // a root, now under pb
    a = old;
    pa = __ldcg(&label[a]);
    pb = __ldcg(&label[b]);
  }
}

__global__ void cc_identity_kernel(uint32_t* label, uint32_t lo, uint32_t hi) {
  for (uint32_t v = lo + blockIdx.x * blockDim.x + threadIdx.x; v < hi; v += gridDim.x * blockDim.x) label[v] = v;
}

// ---- uniting a vertex set along its arcs ------------------------------------
// All vertices (aff == null), or those of a bitmap, united along every live arc
// with both ends in the set.  Uniting arc by arc makes every arc of a skewed
// graph race for one root: R-MAT 2^20 (32M arcs) took 3.41 ms however little
// the batch cut.  Almost all of those arcs lie inside one giant component that
// two arcs per vertex already reveal, so (the sampling order of Sutton,
// Ben-Nun and Barak, "Optimizing parallel graph connectivity computation via
// subgraph sampling", IPDPS 2018):
//   hook    label[v] = the smaller of v and its first neighbour (rows are
//           sorted, so that is the smallest): one plain store each, no cycle;
//           the trees are then compressed;
//   link    v is united with its second neighbour (almost always equal by
//           now: two label loads);
//   sample  the commonest root of 256 vertices is taken for the giant one;
//   rows    only vertices of other sets unite along their whole rows.
// An arc between two sets is seen from an end outside the giant, as both
// directions are stored, so the partition is the same whichever root is taken
// (none when no sample hit the set).  Each pass is a coalesced sweep of the
// vertices with a few dependent loads each, bound by their latency; at R-MAT
// 2^20 they take some 90 us together (hook 13, compress 40, link 20, sample 6,
// rows 12).

constexpr uint32_t kNoRoot = 0xFFFFFFFFu;
constexpr uint32_t kProbe = 4;     // arcs of each row part looked at for a live neighbour in the set
constexpr uint32_t kSamples = 256;
constexpr uint32_t kLaneRow = 8;   // rows this short are walked by one lane

__device__ __forceinline__ bool in_set(const uint32_t* aff, uint32_t v) {
  return !aff || ((aff[v >> 5] >> (v & 31)) & 1u);
}

// The smallest neighbour of v above `after` in the set among the first kProbe
// arcs of its base row and of its delta row; kNoRoot if there is none.
__device__ __forceinline__ uint32_t probe_row(const vxb::DevAdj& a, uint32_t v, uint32_t V, const uint32_t* aff,
                                              uint32_t after, bool any_after) {
  uint64_t b, e;
  vxb::base_range(a, v, b, e);
  const uint2 dr = a.drow[v];
  uint32_t best = kNoRoot;
  for (uint32_t k = 0; k < kProbe && b + k < e; ++k) {
    const uint32_t x = a.col[b + k];
    if ((x & vxb::kTomb) || x >= V || (any_after && x <= after) || !in_set(aff, x)) continue;
    best = x;
    break;
  }
  for (uint32_t k = 0; k < kProbe && k < dr.y; ++k) {
    const uint32_t x = a.darena[dr.x + k];
    if (x >= V || (any_after && x <= after) || !in_set(aff, x)) continue;
    best = min(best, x);
    break;
  }
  return best;
}

__global__ void cc_hook_kernel(vxb::DevAdj a, uint32_t V, uint32_t n, uint32_t* label, const uint32_t* aff,
                               const uint32_t* any) {
  if (any && !*any) return;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    if (!in_set(aff, v)) continue;
    const uint32_t x = probe_row(a, v, V, aff, 0u, false);
    label[v] = min(v, x);
  }
}

__global__ void cc_link_kernel(vxb::DevAdj a, uint32_t V, uint32_t n, uint32_t* label, const uint32_t* aff,
                               const uint32_t* any) {
  if (any && !*any) return;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    if (!in_set(aff, v)) continue;
    const uint32_t x = probe_row(a, v, V, aff, 0u, false);
    if (x == kNoRoot) continue;
    const uint32_t y = probe_row(a, v, V, aff, x, true);
    if (x > v) cc_union(label, v, x);  // a vertex hooked to itself: its first arc is still to be united
    if (y != kNoRoot && __ldcg(&label[v]) != __ldcg(&label[y])) cc_union(label, v, y);
  }
}

// The root of v, read only (no halving: nothing is stored behind a union's back).
__device__ __forceinline__ uint32_t cc_root(const uint32_t* label, uint32_t v) {
  uint32_t p = __ldcg(&label[v]);
  while (p != v) {
    v = p;
    p = __ldcg(&label[v]);
  }
  return v;
}

// One block: the commonest root of kSamples vertices spread over [0, n), those
// outside the set not counted.
__global__ void __launch_bounds__(kSamples) cc_sample_kernel(const uint32_t* label, uint32_t n, const uint32_t* aff,
                                                             const uint32_t* any, uint32_t* giant) {
  __shared__ uint32_t root[kSamples];
  __shared__ unsigned long long best;
  if (any && !*any) return;
  const uint32_t t = threadIdx.x;
  // one vertex at a hashed place in each of kSamples equal parts
  const uint64_t lo = (uint64_t)n * t / kSamples, hi = (uint64_t)n * (t + 1) / kSamples;
  uint32_t r = kNoRoot;
  if (hi > lo) {
    const uint32_t v = (uint32_t)(lo + vxb::mix64(t) % (hi - lo));
    if (in_set(aff, v)) r = cc_root(label, v);
  }
  root[t] = r;
  if (t == 0) best = kNoRoot;  // no count, no root
  __syncthreads();
  if (r != kNoRoot) {
    uint32_t c = 0;
    for (uint32_t k = 0; k < kSamples; ++k) c += root[k] == r;
    atomicMax(&best, (unsigned long long)c << 32 | r);
  }
  __syncthreads();
  if (t == 0) *giant = (uint32_t)best;
}

// The rows of the set's vertices outside the giant: a lane each finds them and
// walks the short ones, the warp the others.  Rows of at most two arcs have been
// hooked and linked whole; a short row's arcs are united without a look for its
// root, which costs about as much.  A tree of 2^20 randomly numbered vertices with
// three children each: 759 us with a warp per row (and a find of both roots), now
// 70 to 95.
__global__ void cc_rows_kernel(vxb::DevAdj a, uint32_t V, uint32_t n, uint32_t* label, const uint32_t* aff,
                               const uint32_t* any, const uint32_t* giant) {
  if (any && !*any) return;
  const uint32_t big = *giant, lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; v0 < n; v0 += nw * 32) {
    const uint32_t v = v0 + lane;
    uint32_t deg = 0;
    if (v < n && in_set(aff, v) && __ldcg(&label[v]) != big) deg = frontier::degree_of(a, v);
    if (deg > kLaneRow && cc_root(label, v) == big) deg = 0;
    if (deg > 2u && deg <= kLaneRow) {
      uint64_t b, e;
      vxb::base_range(a, v, b, e);
      const uint2 dr = a.drow[v];
      const uint32_t nb = (uint32_t)(e - b);
      for (uint32_t k = 0; k < nb + dr.y; ++k) {
        const uint32_t x = k < nb ? a.col[b + k] : a.darena[dr.x + (k - nb)];
        if (!(x & vxb::kTomb) && x < V && in_set(aff, x)) cc_union(label, v, x);
      }
    }
    uint32_t rows = __ballot_sync(0xFFFFFFFFu, deg > kLaneRow);
    while (rows) {
      const uint32_t u = v0 + (uint32_t)__ffs(rows) - 1;
      rows &= rows - 1;
      auto visit = [&](bool valid, uint32_t x, uint32_t) {
        if (valid && x < V && in_set(aff, x)) cc_union(label, u, x);
      };
      frontier::warp_row(a, u, visit);
    }
  }
}

// Every label becomes its root.  The walk halves the paths it takes, so the long
// chains that hooking leaves on a lattice shorten for everybody (2048 x 2048,
// two batches and the label read: 3.8 ms against 15.4 ms without, and 5.5 ms
// arc by arc).  It lowers by atomicMin: ancestors are always
// smaller ids, so a thread that read an old parent cannot store it back over
// the root another thread stored meanwhile.
__global__ void cc_compress_kernel(uint32_t* label, uint32_t V, const uint32_t* any) {
  if (any && !*any) return;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const uint32_t first = __ldcg(&label[v]);
    uint32_t x = v, p = first;
    while (p != x) {
      const uint32_t gp = __ldcg(&label[p]);
      if (gp != p && x != v) atomicMin(&label[x], gp);
      x = p;
      p = gp;
    }
    if (x != first) atomicMin(&label[v], x);
  }
}

// Step 2: roots of the endpoints of effective deletions (present before the
// batch, final op a removal), among the pre-batch vertices.
__global__ void cc_mark_roots_kernel(const uint32_t* fu, const uint32_t* fv, const uint8_t* ff, const uint32_t* F,
                                     const uint32_t* label, uint32_t n_old, uint32_t* aroot, uint32_t* any) {
  const uint32_t nf = *F;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x) {
    const uint8_t f = ff[i];
    if ((f & kFAdd) || !(f & kFCur)) continue;
    const uint32_t u = fu[i], v = fv[i];
    if (u >= n_old || v >= n_old) continue;
    const uint32_t ru = label[u], rv = label[v];
    atomicOr(&aroot[ru >> 5], 1u << (ru & 31));
    atomicOr(&aroot[rv >> 5], 1u << (rv & 31));
    *any = 1u;
  }
}

// Affected vertices (their root is marked) as a bitmap, counted.
__global__ void cc_mark_vertices_kernel(const uint32_t* label, uint32_t n_old, const uint32_t* aroot, uint32_t* aff,
                                        const uint32_t* any, unsigned long long* count) {
  if (!*any) return;
  // a lane per vertex, so the labels are read whole lines at a time, a ballot
  // per bitmap word, and one counter update per block (one per warp serialised
  // on the counter: 28 us at 2^20 vertices)
  __shared__ uint32_t total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  uint32_t c = 0;
  const uint32_t lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < (n_old + 31) / 32; w += nw) {
    const uint32_t v = w * 32 + lane;
    bool hit = false;
    if (v < n_old) {
      const uint32_t r = label[v];
      hit = (aroot[r >> 5] >> (r & 31)) & 1u;
    }
    const uint32_t bits = __ballot_sync(0xFFFFFFFFu, hit);
    if (lane == 0) {
      aff[w] = bits;
      c += __popc(bits);
    }
  }
  if (lane == 0 && c) atomicAdd(&total, c);
  __syncthreads();
  if (threadIdx.x == 0 && total) atomicAdd(count, (unsigned long long)total);
}

// Step 5: the final additions of the batch (their edges exist now).
__global__ void cc_union_adds_kernel(const uint32_t* fu, const uint32_t* fv, const uint8_t* ff, const uint32_t* F,
                                     uint32_t* label, const uint32_t* graph_err, uint32_t* err) {
  // the graph's error word goes out with the affected count: a copy of its own was 7 us a read
  if (blockIdx.x == 0 && threadIdx.x == 0) *err = *graph_err;
  const uint32_t nf = *F;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x)
    if ((ff[i] & kFAdd) && fu[i] < fv[i]) cc_union(label, fu[i], fv[i]);
}

int ensure_labels(Components* c, size_t V) {
  if (V <= c->cap && c->label) return 0;
  size_t cap = std::max<size_t>(c->cap ? c->cap : 1024, 1024);
  while (cap < V) cap *= 2;
  cudaStream_t s = c->g->stream;
  uint32_t *label = nullptr, *aroot = nullptr, *aff = nullptr;
  const size_t words = cap / 32 + 1;
  if (cudaMalloc(&label, cap * 4) != cudaSuccess || cudaMalloc(&aroot, words * 4) != cudaSuccess ||
      cudaMalloc(&aff, words * 4) != cudaSuccess) {
    cudaFree(label);
    cudaFree(aroot);
    set_error("components: allocation for %zu vertices failed", cap);
    return -4;
  }
  VX_CUDA_TRY(cudaMemsetAsync(aroot, 0, words * 4, s));
  VX_CUDA_TRY(cudaMemsetAsync(aff, 0, words * 4, s));
  if (c->label && c->n) VX_CUDA_TRY(cudaMemcpyAsync(label, c->label, c->n * 4, cudaMemcpyDeviceToDevice, s));
  VX_CUDA_TRY(cudaStreamSynchronize(s));
  cudaFree(c->label);
  cudaFree(c->aroot);
  cudaFree(c->aff);
  c->label = label;
  c->aroot = aroot;
  c->aff = aff;
  c->cap = cap;
  return 0;
}

// Unites the vertices [0, n) of the set (all, or the affected ones, whose
// kernels run only when *any is set) in the graph of V vertices.  Labels of the
// set need not hold anything before; afterwards they lead to the sets' roots.
void unite_rows(Components* c, uint32_t V, uint32_t n, const uint32_t* aff, const uint32_t* any) {
  cudaStream_t s = c->g->stream;
  const vxb::DevAdj a = c->g->view().out;
  uint32_t* giant = c->ctr + 1;
  count_launch();
  cc_hook_kernel<<<cc_grid(n), kCcThreads, 0, s>>>(a, V, n, c->label, aff, any);
  count_launch();
  cc_compress_kernel<<<cc_grid(n), kCcThreads, 0, s>>>(c->label, n, any);
  count_launch();
  cc_link_kernel<<<cc_grid(n), kCcThreads, 0, s>>>(a, V, n, c->label, aff, any);
  count_launch();
  cc_sample_kernel<<<1, kSamples, 0, s>>>(c->label, n, aff, any, giant);
  count_launch();
  cc_rows_kernel<<<cc_grid(n), kCcThreads, 0, s>>>(a, V, n, c->label, aff, any, giant);
}

}  // namespace

int cc_rebuild(Components* c) {
  Graph* g = c->g;
  const size_t V = g->V;
  if (int rc = ensure_labels(c, std::max<size_t>(V, 1))) return rc;
  cudaStream_t s = g->stream;
  if (V) {
    unite_rows(c, (uint32_t)V, (uint32_t)V, nullptr, nullptr);
    count_launch();
    cc_compress_kernel<<<cc_grid(V), kCcThreads, 0, s>>>(c->label, (uint32_t)V, nullptr);
    VX_CUDA_TRY(cudaGetLastError());
  }
  c->n = V;
  c->last_repaired = V;
  c->repaired_pending = c->err_pending = false;
  return 0;
}

int cc_create(Components** out, Graph* g) {
  if (g->directed) {
    set_error("IncrementalComponents requires an undirected graph; use an explicitly defined weak/strong "
              "connectivity algorithm for directed graphs");
    return -1;
  }
  Components* c = new Components();
  c->g = g;
  if (cudaMalloc(&c->ctr, 32) != cudaSuccess) {
    set_error("components: counter allocation failed");
    cc_destroy(c);
    return -4;
  }
  if (int rc = cc_rebuild(c)) {
    cc_destroy(c);
    return rc;
  }
  *out = c;
  return 0;
}

void cc_destroy(Components* c) {
  if (!c) return;
  if (c->g && c->g->stream) cudaStreamSynchronize(c->g->stream);
  cudaFree(c->label);
  cudaFree(c->aroot);
  cudaFree(c->aff);
  cudaFree(c->ctr);
  delete c;
}

int cc_apply_staged(Components* c, size_t n, size_t vertex_bound) {
  Graph* g = c->g;
  cudaStream_t s = g->stream;
  c->last_repaired = 0;
  c->repaired_pending = false;
  if (n == 0) return 0;  // an empty batch changes nothing (connected_components.hpp:32-35)
  const uint32_t n_old = (uint32_t)c->n;
  if (int rc = graph_stage_batch(g, n, vertex_bound)) return rc;  // also grows the graph
  const size_t V = g->V;
  // before the marks: a growth replaces their bitmaps
  if (int rc = ensure_labels(c, std::max<size_t>(V, 1))) return rc;
  BatchBuffers& B = g->batch;
  const uint32_t* F = &g->ctr->final_arcs;
  const uint32_t words_old = (n_old + 31) / 32;
  uint32_t* any = c->ctr;                                                   // effective deletion seen
  unsigned long long* count = reinterpret_cast<unsigned long long*>(c->ctr + 2);  // affected vertices
  VX_CUDA_TRY(cudaMemsetAsync(c->ctr, 0, 20, s));
  const uint64_t m = 2 * n;  // canonical arcs of an undirected batch, at most
  if (n_old) {
    count_launch();
    cc_mark_roots_kernel<<<cc_grid(m), kCcThreads, 0, s>>>(B.fu, B.fv, B.ff, F, c->label, n_old, c->aroot, any);
    count_launch();
    cc_mark_vertices_kernel<<<std::min(cc_grid(n_old), 148u * 8u), kCcThreads, 0, s>>>(c->label, n_old, c->aroot, c->aff, any, count);
  }
  c->repaired_pending = c->err_pending = true;  // read by cc_sync
  if (int rc = graph_commit_batch(g)) return rc;
  if (V > n_old) {
    count_launch();
    cc_identity_kernel<<<cc_grid(V - n_old), kCcThreads, 0, s>>>(c->label, n_old, (uint32_t)V);
    VX_CUDA_TRY(cudaMemsetAsync(c->aff + words_old, 0, ((V + 31) / 32 + 1 - words_old) * 4, s));
  }
  if (n_old) unite_rows(c, (uint32_t)V, n_old, c->aff, any);
  count_launch();
  cc_union_adds_kernel<<<cc_grid(m), kCcThreads, 0, s>>>(B.fu, B.fv, B.ff, F, c->label, &g->ctr->err, c->ctr + 4);
  count_launch();
  cc_compress_kernel<<<cc_grid(V), kCcThreads, 0, s>>>(c->label, (uint32_t)V, nullptr);
  // the marks start clear for the next batch
  VX_CUDA_TRY(cudaMemsetAsync(c->aroot, 0, ((c->cap / 32) + 1) * 4, s));
  VX_CUDA_TRY(cudaMemsetAsync(c->aff, 0, ((c->cap / 32) + 1) * 4, s));
  VX_CUDA_TRY(cudaGetLastError());
  c->n = V;
  return 0;
}

// Waits for the stream; reads the last batch's affected count and the error word
// unless they have been read, and fails when a wait of the graph's sort ran out (the
// batch held no arcs then).
static int cc_sync(Components* c) {
  Graph* g = c->g;
  VX_CUDA_TRY(cudaStreamSynchronize(g->stream));
  if (!c->err_pending) return 0;
  volatile uint32_t* err = reinterpret_cast<uint32_t*>(g->pinned_scalar + 1);
  if (*err & vxb::kErrBarrierTimeout) {
    // (a load since then has cleared the graph's word)
    VX_CUDA_TRY(cudaMemcpyAsync(g->pinned_scalar + 1, &g->ctr->err, 4, cudaMemcpyDeviceToHost, g->stream));
    VX_CUDA_TRY(cudaStreamSynchronize(g->stream));
    if (*err & vxb::kErrBarrierTimeout) {
      set_error("components: a wait of the radix sort ran out");
      return -5;
    }
  }
  c->err_pending = false;
  if (c->repaired_pending) c->last_repaired = (size_t)g->pinned_scalar[0];
  c->repaired_pending = false;
  return 0;
}

// Enqueues the read that cc_sync looks at.
static int cc_ask(Components* c) {
  if (c->err_pending)
    VX_CUDA_TRY(cudaMemcpyAsync(c->g->pinned_scalar, c->ctr + 2, 12, cudaMemcpyDeviceToHost, c->g->stream));
  return 0;
}

int cc_last_repaired(Components* c, uint64_t* out) {
  if (c->repaired_pending) {
    if (int rc = cc_ask(c)) return rc;
    if (int rc = cc_sync(c)) return rc;
  }
  *out = c->last_repaired;
  return 0;
}

int cc_labels(Components* c, uint32_t* host_out, size_t cap, size_t* n) {
  *n = c->n;
  const size_t k = std::min(cap, c->n);
  if (int rc = cc_ask(c)) return rc;
  if (host_out && k) VX_CUDA_TRY(cudaMemcpyAsync(host_out, c->label, k * 4, cudaMemcpyDeviceToHost, c->g->stream));
  return cc_sync(c);
}

}  // namespace vxh
