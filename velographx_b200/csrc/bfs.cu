// Full BFS and incremental repair as persistent cooperative kernels.
//
// Two kernels, each a single co-resident grid that synchronises with the
// bounded grid_barrier: bfs_full_kernel runs the full BFS (kModeFull) and
// bfs_kernel the two repair modes.
//
//   kModeFull  recompute (bfs.hpp:100-120) as a direction-optimising BFS:
//              top-down levels expand a frontier queue with warp-cooperative
//              gathers (rows < 32 arcs flattened across the warp, medium rows
//              expanded by the whole warp, rows >= tune.large_row by the whole
//              grid; the smallest levels by one block alone), bottom-up levels
//              look through every block's own vertices and stop each scan at
//              the first parent in the frontier bitmap.  Top-down claims are
//              atomicOr on the visited bitmap; queues are appended through the
//              blocks' shared memory.
//   kModePre   the pre-batch part of apply (bfs.hpp:38-70, 222-259): deletion
//              candidates and the support-count fixpoint, run as one
//              asynchronous cascade over a work ring (no barrier per level).
//   kModePost  the post-batch part (bfs.hpp:72-97, 261-354): either the
//              fallback full BFS, or invalidation and boundary distances of
//              the affected vertices, then one asynchronous label-correcting
//              relaxation from them and from the heads of inserted arcs.
#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <vector>

#include "bfs.cuh"
#include "vstream.cuh"
#include "graph_dev.cuh"
#include "frontier.cuh"

namespace vxh {

using vxb::DevAdj;
using vxb::kIdMask;
using vxb::kTomb;
using vxb::kUnreachable;

namespace {

using namespace frontier;

constexpr int kThreads = 512;
enum { kModeFull = 0, kModePre = 1, kModePost = 2 };
// Slots of each bottom-up candidate list for V vertices: the blocks' segments
// of whole tiles (BuTiles) hold at most V / 16 + 32 vertices per block more
// than V (at most 1,024 blocks).
constexpr size_t list_slots(size_t V) { return V + V / 16 + 32 * 1024; }

struct Params {
  vxb::DevGraph g;
  uint32_t V;         // vertices of the graph in this phase
  uint32_t dist_len;  // logical length of the distance vector in this phase
  uint32_t source;
  uint32_t* dist;
  uint32_t* vis;
  uint32_t* fb[3];
  uint32_t* q[3];
  uint32_t* big;
  uint32_t* lst_a;
  uint32_t* lst_t;
  uint32_t* tent;
  uint32_t* bul;      // bottom-up candidate lists A (bul[0, bul_half)) and B (bul[bul_half, 2 * bul_half)),
  uint32_t bul_half;  // each cut into one segment per block (bul_half >= list_slots(V))
  unsigned long long* sw;  // support words of the pre-batch cascade (zero between batches)
  unsigned long long* ring;  // work ring of the repair phases (kSent between phases)
  uint32_t ring_mask;
  uint32_t* rq_head;       // ring counters, each on its own 128-byte line: the
  uint32_t* rq_tail;       // idle blocks poll them while the working ones push
  uint32_t* rq_done;
  uint32_t* rq_fin;        // set by the first block that sees the phase finished
  unsigned long long* rq_stat;  // drain statistics of the last phase (own line)
  uint32_t* aff;
  uint32_t* inq[2];
  const uint32_t* fu;
  const uint32_t* fv;
  const uint8_t* ff;
  const uint32_t* F;
  BfsCounters* c;
  unsigned long long total_arcs;
  unsigned long long fallback_limit;
  float handover;        // time budget of a repair phase, in multiples of the last full BFS's time
  uint32_t cascade_bfs;  // the cascade may hand over (the distance vector spans the graph)
  float alpha, beta;
  uint32_t large_row;
  uint32_t nblocks;
  uint32_t deltas;  // the graph may hold delta rows (zero: their table need not be read)
  const uint32_t* graph_err;  // the graph's error word (null: none)
  unsigned long long* trace;  // optional per-level {time, n_f | bottom-up << 63}
  // optional accounting of the update launch's algorithmic bytes (null: off):
  // [0] row arcs scanned by the repair, [1] vertices it visited, [2] delta-row
  // entries the commit read and wrote, [3] canonical arcs, [4] batches
  unsigned long long* acct;
  uint32_t* bar;              // grid barrier words
};

// What a repair launch's phases change of its parameters, a copy per block (thread 0
// writes it between block barriers; start_phases).  The other parameters are read
// where the launch put them: with all of them in shared memory every use was a load
// that no store could be moved past (a pair of 64-op batches at 2^20 vertices 67 us,
// now 63; a vertex of a cascade along a path 5.8 us, now 5.6).
struct PhaseParams {
  uint32_t V;             // vertices of the graph in this phase
  uint32_t dist_len;      // logical length of the distance vector in this phase
  uint32_t rq_base;       // slot of the ring's current epoch's first item (sync_rounds)
  uint32_t* rq_tail;      // the current epoch's length (Params::rq_tail + epoch)
  uint32_t touched_base;  // length of the touched list before touched_n counts
  uint32_t cascade_bfs;   // the cascade may hand over (the distance vector spans the graph)
  const uint32_t* fu;     // the batch's canonical arcs
  const uint32_t* fv;
  const uint8_t* ff;
  const uint32_t* F;
  unsigned long long fallback_limit;
};
__shared__ PhaseParams ph;

constexpr uint32_t kTraceLevels = 256;

// Time budgets of the repair phases.  On a deep graph one batch can move the
// distances of millions of vertices, and the cascade or the relaxation then
// walks them level by level, for far longer than a full BFS takes.  A phase
// that has run longer than handover x (the last full BFS's time + 0.1 ms) drops the rest of its queue and a BFS finishes its work, so a batch costs at most about
// twice the cheaper of the two; either way the result is the same.  The
// deadline is set by thread 0 before the barrier that precedes the phase's
// drain, which reads it once and compares it with the clock every round.  The cascade's BFS compares distances over every vertex of the
// phase graph, so it may hand over only when the distance vector spans it.
constexpr unsigned long long kNever = ~0ull;
// What handing over costs beside the BFS (clearing, the comparison pass,
// barriers, the launch's smaller blocks): without it 100,000-op batches at
// R-MAT 20, whose cascades take 110 us against a BFS of 70, hand over and take
// 280.
constexpr double kHandoverNs = 100e3;

__device__ __forceinline__ void set_deadline(const Params& p) {
  const float h = p.handover;
  const unsigned long long f = p.c->full_ns;
  p.c->deadline = h < 0.0f || (h > 0.0f && f == 0ull)
                      ? kNever
                      : globaltimer() + (unsigned long long)((double)h * ((double)f + kHandoverNs));
}

__device__ __forceinline__ void acct_add(const Params& p, int k, unsigned long long v) {
  if (p.acct && v) atomicAdd(&p.acct[k], v);
}

// A wait of the graph's sort that ran out (its batch holds no arcs then) becomes
// the object's error, so that the next synchronising call on it fails: one thread
// loads the word at the start of a launch and looks at it before the first barrier
// (with the words of every barrier it cost 1 us a batch).
__device__ __forceinline__ uint32_t sort_error(const Params& p) {
  return gtid() == 0 && p.graph_err ? __ldcg(p.graph_err) & vxb::kErrBarrierTimeout : 0u;
}

// Grid barrier; returns false once any block recorded a device error (a
// barrier that gave up waiting, a loop bound), so every persistent loop ends.
__device__ __forceinline__ bool sync_grid(const Params& p) {
  __shared__ uint32_t failed;
  vxb::grid_barrier_then(p.bar, p.nblocks, &p.c->err, [&] { failed = __ldcg(&p.c->err); });
  return failed == 0u;
}


// The row bounds of u; the delta row is read only where the graph may hold
// one (a loaded or compacted graph has none) and the row's dirty bit is set
// (every delta row's is): the table is one more random 32-byte sector per
// vertex, the bits stay in L2.  The bits are read past L1, which may hold them
// as they were before the launch's own insertions.
__device__ __forceinline__ void row_of(const Params& p, const DevAdj& a, uint32_t u, uint64_t& b, uint32_t& nb,
                                       uint2& dr) {
  uint64_t e;
  vxb::base_range(a, u, b, e);
  nb = (uint32_t)(e - b);
  dr = p.deltas && (ld_cg(&a.dirty[u >> 5]) >> (u & 31)) & 1u ? a.drow[u] : make_uint2(0u, 0u);
}

__device__ __forceinline__ uint32_t row_len(const Params& p, const DevAdj& a, uint32_t u) {
  uint64_t b;
  uint32_t nb;
  uint2 dr;
  row_of(p, a, u, b, nb, dr);
  return nb + dr.y;
}

// ------------------------------------------------------------ top-down --
//
// A level is a chain of dependent round trips per arc (column, visited word,
// claim), so its time is the number of steps a warp takes times that chain.
// Every path below hands TdVisit::visit four arcs per lane at once, whose
// loads and atomics are all in flight together.  A 4096 x 4096 lattice (160
// levels of up to 644,000 vertices with 4 arcs each): 4.15 -> 2.33 ms, with the
// one-block levels and the direction rule below; its widest levels (57 us) move
// some 200 MB of scattered sectors through L2.

constexpr int kVisit = 4;  // arcs a lane has in flight per step

template <class Queue, bool kTogether>
struct TdVisit {
  const Params* p;
  uint32_t* dist;
  uint32_t level;
  uint32_t* qout;
  uint32_t* fbn;  // bitmap of the next frontier, or null when no bottom-up level reads it as it is made
  uint32_t* cnt_n;
  Queue* bq;
  unsigned long long mloc;  // arcs of the vertices this lane claimed
  // Claims the heads of one step's arcs for the next level (warp-uniform);
  // bit 31 of an entry marks a dead arc or none.
  __device__ __forceinline__ void visit(const uint32_t (&x)[kVisit]) {
    uint32_t w[kVisit];
#pragma unroll
    for (int j = 0; j < kVisit; ++j) w[j] = (x[j] & kTomb) ? FULL : p->vis[x[j] >> 5];
    // the row lengths are loaded before the claims, so both are in flight together
    uint32_t deg[kVisit];
#pragma unroll
    for (int j = 0; j < kVisit; ++j) deg[j] = (w[j] >> (x[j] & 31)) & 1u ? 0u : row_len(*p, p->g.out, x[j]);
    // Heads side by side (a hub's leaves) share a word: where 16 lanes or more do, one
    // of them claims for all, as atomics of a warp on one word are served one by one (a
    // star of 2^20 leaves 154 us, with eight arcs per lane in flight 73, so 39).  Not in
    // levels of one block (a 59 x 59 lattice 78 us, so 87) and not with 1,024 threads,
    // which have no registers left for it (R-MAT of 3.9M vertices 134 us, so 136).
    uint32_t m[kVisit];  // lanes whose claim is made together
#pragma unroll
    for (int j = 0; j < kVisit; ++j) {
      const uint32_t bit = 1u << (x[j] & 31), word = x[j] >> 5;
      const bool need = !(w[j] & bit);
      uint32_t op = need ? bit : 0u;
      m[j] = 0u;
      if (kTogether) {
        const uint32_t middle = __shfl_sync(FULL, word, 16);  // every lane takes part
        m[j] = __ballot_sync(FULL, need && word == middle);
      }
      if (kTogether && __popc(m[j]) >= 16) {
        const bool in = (m[j] >> (threadIdx.x & 31)) & 1u;
        const uint32_t all = __reduce_or_sync(FULL, in ? bit : 0u);
        if (__popc(all) != __popc(m[j])) m[j] = 0u;  // a head twice
        else if (in) op = (m[j] & vxb::lanemask_lt()) == 0u ? all : 0u;
      } else {
        m[j] = 0u;
      }
      if (op) w[j] = atomicOr(&p->vis[word], op);
    }
#pragma unroll
    for (int j = 0; j < kVisit; ++j) {
      const uint32_t bit = 1u << (x[j] & 31);
      if (kTogether && m[j]) {  // warp-uniform
        const uint32_t old = __shfl_sync(FULL, w[j], __ffs(m[j]) - 1);
        if ((m[j] >> (threadIdx.x & 31)) & 1u) w[j] = old;
      }
      const bool claim = !(w[j] & bit);
      if (claim) {
        mloc += deg[j];
        dist[x[j]] = level + 1;
      }
      if (fbn) {
        uint32_t op = claim ? bit : 0u;
        if (kTogether && m[j]) {
          const bool in = (m[j] >> (threadIdx.x & 31)) & 1u;
          const uint32_t all = __reduce_or_sync(FULL, in ? op : 0u);
          if (in) op = (m[j] & vxb::lanemask_lt()) == 0u ? all : 0u;
        }
        if (op) atomicOr(&fbn[x[j] >> 5], op);
      }
      m[j] = __ballot_sync(FULL, claim);
    }
    bq_push_n(*bq, m, x, cnt_n, qout);
  }
};

// Rows arr[start, start + len) of the lanes (len 0: none): rows of >= 32 arcs
// walked by the whole warp, shorter ones as one flattened list (a warp scan of
// the lengths, then each arc's owner by a 5-step shuffle search), 128 arcs
// per step either way.
template <class Visit>
__device__ __forceinline__ void td_rows(Visit& t, const uint32_t* arr, uint64_t start, uint32_t len) {
  const int lane = threadIdx.x & 31;
  uint32_t med = __ballot_sync(FULL, len >= 32);
  while (med) {
    const int l = __ffs(med) - 1;
    med &= med - 1;
    const uint64_t s = __shfl_sync(FULL, start, l);
    const uint32_t n = __shfl_sync(FULL, len, l);
    for (uint32_t k0 = 0; k0 < n; k0 += 32 * kVisit) {
      uint32_t x[kVisit];
#pragma unroll
      for (int j = 0; j < kVisit; ++j) {
        const uint32_t k = k0 + 32 * j + lane;
        x[j] = k < n ? arr[s + k] : kTomb;
      }
      t.visit(x);
    }
  }
  if (len >= 32) len = 0;
  uint32_t incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  const uint32_t excl = incl - len;
  const uint32_t total = __shfl_sync(FULL, incl, 31);
  start -= excl;  // arc k of the list is arr[start + k] in its owner's lane
  for (uint32_t k0 = 0; k0 < total; k0 += 32 * kVisit) {
    uint32_t x[kVisit];
#pragma unroll
    for (int j = 0; j < kVisit; ++j) {
      const uint32_t k = k0 + 32 * j + lane;
      int owner = 0;
#pragma unroll
      for (int step = 16; step >= 1; step >>= 1) {
        const uint32_t ex = __shfl_sync(FULL, excl, owner + step);
        if (ex <= k) owner += step;
      }
      const uint64_t s = __shfl_sync(FULL, start, owner);
      x[j] = k < total ? arr[s + k] : kTomb;
    }
    t.visit(x);
  }
}

// A wide frontier: up to 32 of its vertices per warp, fewer
// when that leaves warps without any.  Rows of at least large_row arcs are
// listed (p.big, their lengths in p.bul, free outside the bottom-up levels)
// for grid_rows.
template <class Visit>
__device__ void td_level(const Params& p, Visit& t, const uint32_t* qin, uint32_t n_f, uint32_t* cnt_big) {
  const DevAdj& a = p.g.out;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t per = min(32u, (n_f + nwarps() - 1) / nwarps());
  for (uint32_t base = gwarp() * per; base < n_f; base += nwarps() * per) {
    const bool act = lane < per && base + lane < n_f;
    const uint32_t u = act ? qin[base + lane] : 0u;
    uint64_t b = 0;
    uint32_t nb = 0;
    uint2 dr = make_uint2(0u, 0u);
    if (act) row_of(p, a, u, b, nb, dr);
    const bool big = act && nb + dr.y >= p.large_row;
    const uint32_t slot = vxb::warp_append(big, cnt_big);
    if (big) {
      p.big[slot] = u;
      p.bul[slot] = nb + dr.y;
      nb = dr.y = 0;
    }
    td_rows(t, a.col, b, nb);
    if (p.deltas) td_rows(t, a.darena, dr.x, dr.y);
  }
}

// Top-down expansion of a small frontier (n_f <= kLbMax) as one flat edge
// space: every block stages the frontier's row ranges and their degree prefix
// in shared memory, then each warp takes 32 consecutive edges per step and
// finds their owners by binary search -- the same number of edges per warp
// however skewed the rows are (a 30-vertex frontier of hubs included).
constexpr uint32_t kLbMax = 1024;
// Levels of the grid take the flat edge space up to here: staging 1,024 rows of four
// arcs made a level 7.3 us, by td_level it takes 6.9.
constexpr uint32_t kFlatMax = 1000;
struct LbStage {
  uint32_t pref[kLbMax + 1];
  uint64_t base[kLbMax];
  uint32_t blen[kLbMax];
  uint32_t dx[kLbMax];
};

template <int kT>
__device__ void lb_stage(const Params& p, const uint32_t* qin, uint32_t n_f, LbStage& st) {
  const DevAdj& a = p.g.out;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kPer = kLbMax / kT;  // frontier entries per thread
  uint32_t len[kPer], sum = 0;
#pragma unroll
  for (int h = 0; h < kPer; ++h) {
    const uint32_t i = threadIdx.x * kPer + h;
    len[h] = 0;
    if (i < n_f) {
      uint64_t b;
      uint32_t nb;
      uint2 dr;
      row_of(p, a, qin[i], b, nb, dr);
      st.base[i] = b;
      st.blen[i] = nb;
      st.dx[i] = dr.x;
      len[h] = nb + dr.y;
    }
    sum += len[h];
  }
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  __shared__ uint32_t wsum[kT / 32];
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < kT / 32 ? wsum[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < kT / 32) wsum[lane] = wi - w;
  }
  __syncthreads();
  uint32_t ex = wsum[warp] + incl - sum;
#pragma unroll
  for (int h = 0; h < kPer; ++h) {
    const uint32_t i = threadIdx.x * kPer + h;
    if (i < n_f) st.pref[i] = ex;
    ex += len[h];
    if (i + 1 == n_f) st.pref[n_f] = ex;
  }
  __syncthreads();
}

// The staged rows' arcs, 32 per warp and round over `warps` warps, four rounds
// at a time (a frontier of fewer arcs still spreads over every warp).
template <class Visit>
__device__ void lb_visit(const Params& p, Visit& t, uint32_t n_f, const LbStage& st, uint32_t warp, uint32_t warps) {
  const DevAdj& a = p.g.out;
  const uint32_t M = st.pref[n_f];
  for (uint32_t e0 = warp * 32; e0 < M; e0 += warps * 32 * kVisit) {
    uint32_t x[kVisit];
#pragma unroll
    for (int j = 0; j < kVisit; ++j) {
      const uint32_t e = e0 + j * warps * 32 + (threadIdx.x & 31);
      x[j] = kTomb;
      if (e < M) {
        uint32_t lo = 0, hi = n_f;  // last i with pref[i] <= e
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) >> 1;
          if (st.pref[mid] <= e) lo = mid;
          else hi = mid;
        }
        const uint32_t k = e - st.pref[lo];
        x[j] = k < st.blen[lo] ? a.col[st.base[lo] + k] : a.darena[st.dx[lo] + (k - st.blen[lo])];
      }
    }
    t.visit(x);
  }
}

// The listed rows of at least large_row arcs, in slices of 128 arcs dealt to
// the warps of the grid.
template <class Visit>
__device__ void grid_rows(const Params& p, Visit& t, uint32_t n) {
  const DevAdj& a = p.g.out;
  const uint32_t lane = threadIdx.x & 31;
  constexpr uint32_t kSlice = 32 * kVisit;
  for_my_rows(p.bul, n, kSlice, [&](uint32_t r, uint32_t len, uint32_t s0) {
    uint64_t b;
    uint32_t nb;
    uint2 dr;
    row_of(p, a, p.big[r], b, nb, dr);
    for (uint64_t k0 = (uint64_t)s0 * kSlice; k0 < len; k0 += (uint64_t)nwarps() * kSlice) {
      uint32_t x[kVisit];
#pragma unroll
      for (int j = 0; j < kVisit; ++j) {
        const uint64_t k = k0 + 32 * j + lane;
        x[j] = k >= len ? kTomb : (k < nb ? a.col[b + k] : a.darena[dr.x + (uint32_t)(k - nb)]);
      }
      t.visit(x);
    }
  });
}

// What a block adds up over a level and reads back after it (shared memory).
struct LevelWords {
  unsigned long long m;   // arcs of the vertices the block claimed
  uint32_t n;             // vertices it claimed without queueing them
  uint32_t failed, n_f, nbig;
  unsigned long long m_f;
};

// The end of a level's pass: the block's sums and queued vertices go out (one
// update of each counter per block), the grid meets, and the block reads the
// level's figures.  Block-uniform; false once any block recorded an error.
template <class Queue>
__device__ __forceinline__ bool level_end(const Params& p, LevelWords& lw, Queue& bq, uint32_t nloc,
                                          unsigned long long mloc, uint32_t slot, uint32_t* nbig) {
  BfsCounters* c = p.c;
  constexpr uint32_t kCap = sizeof(bq.items) / sizeof(bq.items[0]);
  mloc = vxb::warp_sum(mloc);
  nloc = vxb::warp_sum(nloc);
  if ((threadIdx.x & 31) == 0) {
    if (mloc) atomicAdd(&lw.m, mloc);
    if (nloc) atomicAdd(&lw.n, nloc);
  }
  __syncthreads();
  const uint32_t q = min(bq.cnt, kCap);
  if (threadIdx.x == 0) {
    const uint32_t n = lw.n;
    if (lw.m) atomicAdd(&c->lvl_m[slot], lw.m);
    if (q + n) bq.gbase = atomicAdd(&c->lvl_n[slot], q + n);  // queued or counted, not both
    lw.m = 0;
    lw.n = 0;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < q; i += blockDim.x) p.q[slot][bq.gbase + i] = bq.items[i];
  if (threadIdx.x == 0) bq.cnt = 0;  // read by every thread before the block barrier above
  vxb::grid_barrier_then(p.bar, p.nblocks, &c->err, [&] {
    lw.failed = __ldcg(&c->err);
    lw.n_f = ld_cg(&c->lvl_n[slot]);
    lw.m_f = __ldcg(&c->lvl_m[slot]);
    lw.nbig = nbig ? ld_cg(nbig) : 0u;
  });
  return lw.failed == 0u;
}

// The block's sum of v (every thread gets it; red is per-block scratch).
template <int kT>
__device__ __forceinline__ unsigned long long block_sum(unsigned long long v, unsigned long long* red) {
  v = vxb::warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long s = 0;
#pragma unroll
  for (int k = 0; k < kT / 32; ++k) s += red[k];
  return s;
}

// ---- levels of one block ----
// A frontier of a few hundred vertices keeps one block busy for about as long
// as the grid takes to meet at a barrier: block 0 runs such levels by itself,
// frontier in shared memory and block barriers only, until the frontier
// outgrows it, while the others wait at the grid barrier that ends the
// stretch.  A level takes 3 us instead of 8 to 10.  The limit is where a level of
// one block (one step of four arcs per thread) costs what a level of the grid
// does, 7 to 8 us: lattices 512 wide 8.3 us a level by one block, 600 wide 10.7 by
// one block in two steps and 8.1 by the grid, 1,024 wide 18.6 and 9.4.  A stretch is
// bounded so that the waiting blocks' barrier is.
constexpr uint32_t kSoloArcs = 2048;
constexpr uint32_t kSoloLevels = 4096;

// Words of the barrier array past the barrier word (zero between searches):
// what a stretch hands back (two sets of 8), the length of a queue made from a
// bitmap, and the lengths of the arc lists of a batch that the update launch
// canonicalises itself.
constexpr uint32_t kSoloWord = 8, kQueueWord = 28, kRawWord = 30;
static_assert(kRawWord + 2 <= vxb::kBarrierWords, "the barrier array holds these words");

struct SoloState {
  uint32_t level, n_f, reached;
  unsigned long long m_f, m_visited;
};

__device__ __forceinline__ bool solo_fits(uint32_t n_f, unsigned long long m_f) {
  return n_f <= kLbMax && m_f <= kSoloArcs;
}

// Block 0, block-uniform: levels from s.level on, the frontier in qin; the
// frontier after the last one is left in qout (its size added to *cnt_n).
template <int kT, class Queue>
__device__ void solo_levels(const Params& p, uint32_t* dist, const uint32_t* qin, uint32_t* qout, uint32_t* cnt_n,
                            Queue& bq, LbStage& st, unsigned long long* red, unsigned long long* trace,
                            SoloState& s) {
  const uint32_t* in = qin;
  for (uint32_t k = 0; s.n_f && solo_fits(s.n_f, s.m_f) && k < kSoloLevels; ++k, ++s.level) {
    s.reached += s.n_f;
    s.m_visited += s.m_f;
    if (trace && threadIdx.x == 0 && s.level < kTraceLevels) {
      trace[2 * s.level] = globaltimer();
      trace[2 * s.level + 1] = s.n_f;
    }
    lb_stage<kT>(p, in, s.n_f, st);  // ends with a block barrier: the entries are read
    in = bq.items;
    if (threadIdx.x == 0) bq.cnt = 0;
    __syncthreads();
    // an overflow of bq's slots goes to qout: more than kLbMax entries, so it is the last level here
    TdVisit<Queue, false> t{&p, dist, s.level, qout, nullptr, cnt_n, &bq, 0ull};
    lb_visit(p, t, s.n_f, st, threadIdx.x >> 5, kT / 32);
    s.m_f = block_sum<kT>(t.mloc, red);  // its barriers also cover the pushes
    s.n_f = bq.cnt;
    __threadfence_block();
  }
  bq_flush(bq, cnt_n, qout);
}

// ----------------------------------------------------------- bottom-up --

// Appends v where pred holds to a block-private list segment (seg, counter
// n in shared memory), in lane order within the warp.  Warp-uniform.
__device__ __forceinline__ void seg_append(bool pred, uint32_t v, uint32_t* seg, uint32_t* n) {
  const uint32_t m = __ballot_sync(FULL, pred);
  if (!m) return;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(n, (uint32_t)__popc(m));
  base = __shfl_sync(FULL, base, leader);
  if (pred) seg[base + __popc(m & vxb::lanemask_lt())] = v;
}

// A bottom-up level scans the in-rows of the unvisited vertices for a parent
// in the frontier bitmap.  Each scan is a chain of round trips (columns, bitmap
// words), a warp has some 500 vertices, and most of them find their parent
// among the first arcs (rows are sorted, and in skewed graphs the hubs that
// fill the frontier sit at small ids): the level's time is the number of steps
// a warp takes times one step's chain.  So a warp gathers its vertices in a
// ring in shared memory until every lane of a step has kR of them (R-MAT graphs
// have two isolated vertices in five), reads the first 8 arcs of each (kR x 4
// loads in flight), and scans the longer rows still looking four at a time,
// eight lanes each (one after another by the whole warp, each paid its own
// chain).  R-MAT 22, the level that reaches 1.8M of 2.4M vertices: 103 us with
// one vertex per lane and step, 87 us with two (the whole launch moves 193 MB
// of DRAM traffic, mostly single 32-byte sectors: 30 us at the copy rate); one is enough, and 10% faster in all, on
// graphs of a few thousand arcs per block, which kT = 512 serves.  Putting the
// long rows back into the ring instead (24 or 56 arcs left): no gain on large
// graphs, 41 -> 44 us in all at 30,000 vertices.
constexpr uint32_t kBuStep = 8;  // arcs of a vertex a lane scans by itself

constexpr uint64_t kBuDelta = 1ull << 63;
struct BuEntry {
  uint64_t at;    // next arc: base position, or arena position with kBuDelta set
  uint32_t v;
  uint32_t left;  // arcs left of that part of the row
};

// The vertices waiting for a step, per warp: fewer than 32 * kR before a
// refill of 32 or a step's returns (for their delta rows).
template <int kT, int kR>
struct BuStage {
  BuEntry e[kT / 32][32 * kR * 2];
};

// The vertices of a block in bottom-up levels: tiles of 2^shift bitmap words
// dealt to the blocks in turn, at least 16 a block where the graph has them
// (so that no block has all the small ids, an R-MAT graph's hubs; one range per
// block measured the same within 2% at R-MAT 20 to 22).
struct BuTiles {
  uint32_t shift, per_block;  // words per tile (log2), tiles of each block
  __device__ BuTiles(uint32_t words, uint32_t blocks) {
    shift = 0;
    while (shift < 6 && (words >> (shift + 1)) >= blocks * 16u) ++shift;
    const uint32_t tiles = (words + (1u << shift) - 1) >> shift;
    per_block = (tiles + blocks - 1) / blocks;
  }
  // the block's words are 0 .. words() - 1 in its own count
  __device__ uint32_t words() const { return per_block << shift; }
  __device__ uint32_t word_of(uint32_t local) const {
    return (((local >> shift) * gridDim.x + blockIdx.x) << shift) + (local & ((1u << shift) - 1u));
  }
  __device__ uint32_t local_of(uint32_t word) const {
    return (((word >> shift) / gridDim.x) << shift) + (word & ((1u << shift) - 1u));
  }
};

// Where a level's finds and misses go.  Vertices found may be counted and set
// in the bitmaps only (bq null): the queue is then made from the bitmap if a
// top-down level follows (queueing 1.8M vertices past the blocks' buffers took
// tens of thousands of updates of one counter).  A block's bitmap words are its
// own, so their bits are gathered in shared memory where it holds them.
template <class Queue>
struct BuOut {
  uint32_t* dist;
  uint32_t level;
  const uint32_t* fbc;
  uint32_t* fbn;
  uint32_t* bits;   // the block's words in shared memory, or null
  BuTiles tiles;
  uint32_t* lout;   // this block's segment of the next list, and its length (shared memory)
  uint32_t* nout;
  Queue* bq;        // the next frontier's queue, or null
  uint32_t* qout;
  uint32_t* cnt_n;
  uint32_t nloc;    // vertices this lane found and did not queue
};

// Every scan stops at the first parent.  refill(ring, cnt) appends up to 32
// vertices, false when there are no more.  Whole warp.
template <int kR, class Queue, class Refill>
__device__ __forceinline__ void bu_scan(const Params& p, BuOut<Queue>& o, BuEntry* ring, Refill&& refill) {
  const DevAdj& a = p.g.in;
  const uint32_t lane = threadIdx.x & 31, lt = vxb::lanemask_lt();
  uint32_t cnt = 0;
  bool more = true;
  for (;;) {
    while (more && cnt < 32 * kR) more = refill(ring, cnt);
    if (!cnt) break;
    __syncwarp();
    const uint32_t n = min(cnt, 32u * kR);
    cnt -= n;
    BuEntry e[kR];
    bool found[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const uint32_t k = 32 * r + lane;
      e[r] = k < n ? ring[cnt + k] : BuEntry{0ull, kUnreachable, 0u};
      found[r] = false;
    }
    __syncwarp();
#pragma unroll
    for (uint32_t k0 = 0; k0 < kBuStep; k0 += 4) {
      uint32_t x[kR][4];
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        const uint32_t* arr = (e[r].at & kBuDelta ? a.darena : a.col) + (e[r].at & ~kBuDelta) + k0;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) x[r][j] = !found[r] && k0 + j < e[r].left ? arr[j] : kTomb;
      }
#pragma unroll
      for (int r = 0; r < kR; ++r)
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) found[r] = found[r] || (!(x[r][j] & kTomb) && test_bit(o.fbc, x[r][j]));
    }
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      // long rows: four at a time, eight lanes each, 32 arcs per step
      uint32_t coop = __ballot_sync(FULL, !found[r] && e[r].left > kBuStep);
      while (coop) {
        const uint32_t sub = lane >> 3, g = lane & 7;
        int l = -1;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
          if (k == sub) l = __ffs(coop) - 1;
          coop &= coop - 1;
        }
        const uint64_t at = __shfl_sync(FULL, e[r].at, l < 0 ? 0 : l) + kBuStep;
        const uint32_t tot = __shfl_sync(FULL, e[r].left, l < 0 ? 0 : l) - kBuStep;
        const uint32_t* arr = (at & kBuDelta ? a.darena : a.col) + (at & ~kBuDelta);
        bool on = l >= 0, hit_l = false;
        for (uint32_t k0 = 0; __any_sync(FULL, on); k0 += 32) {
          uint32_t x[4];
          bool hit = false;
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j) x[j] = on && k0 + 8 * j + g < tot ? arr[k0 + 8 * j + g] : kTomb;
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j) hit = hit || (!(x[j] & kTomb) && test_bit(o.fbc, x[j]));
          if ((__ballot_sync(FULL, hit) >> (8 * sub)) & 0xFFu) {
            hit_l = true;
            on = false;
          }
          on = on && k0 + 32 < tot;
        }
        const uint32_t got = __reduce_or_sync(FULL, hit_l && g == 0 ? 1u << l : 0u);
        found[r] = found[r] || ((got >> lane) & 1u);
      }
      const uint32_t v = e[r].v;
      const bool real = v != kUnreachable;
      bool look = false;
      if (p.deltas && real && !found[r] && !(e[r].at & kBuDelta)) {  // back for the delta row
        const uint2 dr = a.drow[v];
        e[r].at = dr.x | kBuDelta;
        e[r].left = dr.y;
        look = dr.y != 0u;
      }
      if (found[r]) {
        o.dist[v] = o.level + 1;
        const uint32_t bit = 1u << (v & 31);
        if (o.bits) {
          atomicOr(&o.bits[o.tiles.local_of(v >> 5)], bit);
        } else {
          atomicOr(&p.vis[v >> 5], bit);
          atomicOr(&o.fbn[v >> 5], bit);
        }
        o.nloc += o.bq == nullptr;
      }
      if (o.bq) bq_push(*o.bq, found[r], v, o.cnt_n, o.qout);
      seg_append(real && !found[r] && !look, v, o.lout, o.nout);
      const uint32_t back = __ballot_sync(FULL, look);
      if (look) ring[cnt + __popc(back & lt)] = e[r];
      cnt += __popc(back);
    }
  }
}

// The first arcs of v's in-row for the ring.
__device__ __forceinline__ BuEntry bu_entry(uint32_t v, uint64_t b, uint32_t nb, uint2 dr) {
  return nb ? BuEntry{b, v, nb} : BuEntry{dr.x | kBuDelta, v, dr.y};
}

// The first bottom-up level: every unvisited vertex of the block's tiles with a
// nonempty in-row; a warp reads the visited words and row bounds of 32 vertices
// at a time, one refill ahead.  (Listing the candidates in the initialisation
// pass instead cost a chain of loads per 512 vertices of a block there, also in
// searches that never go bottom-up.)
template <int kT, int kR, class Queue>
__device__ void bu_first_level(const Params& p, uint32_t V, BuOut<Queue>& o, BuStage<kT, kR>& st) {
  const DevAdj& a = p.g.in;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t nw = o.tiles.words();
  uint32_t w = warp, v = 0, vis0 = FULL, n0 = 0;  // v: this lane's vertex of the word loaded
  uint64_t b0 = 0;
  uint2 d0 = make_uint2(0u, 0u);
  auto load = [&] {
    vis0 = FULL;
    if (w >= nw) return;
    const uint64_t x = (uint64_t)o.tiles.word_of(w) * 32 + lane;
    if (x >= V) return;
    v = (uint32_t)x;
    vis0 = p.vis[v >> 5];
    row_of(p, a, v, b0, n0, d0);
  };
  load();
  bu_scan<kR>(p, o, st.e[warp], [&](BuEntry* ring, uint32_t& cnt) {
    if (w >= nw) return false;
    const bool cand = !((vis0 >> lane) & 1u) && n0 + d0.y != 0u;
    const uint32_t m = __ballot_sync(FULL, cand);
    if (cand) ring[cnt + __popc(m & vxb::lanemask_lt())] = bu_entry(v, b0, n0, d0);
    cnt += __popc(m);
    w += kT / 32;
    load();
    return w < nw;
  });
}

// Later bottom-up levels: the block's segment lin[0, nin) of the list the
// level before left (entries visited since are skipped).  Entries are loaded
// two refills ahead, their visited words and row bounds one.
template <int kT, int kR, class Queue>
__device__ void bu_list_level(const Params& p, BuOut<Queue>& o, BuStage<kT, kR>& st, const uint32_t* lin,
                              uint32_t nin) {
  const DevAdj& a = p.g.in;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t base = warp * 32;
  uint32_t v0 = base + lane < nin ? lin[base + lane] : kUnreachable;
  uint32_t v1 = base + kT + lane < nin ? lin[base + kT + lane] : kUnreachable;
  uint32_t vis0 = FULL, n0 = 0;
  uint64_t b0 = 0;
  uint2 d0 = make_uint2(0u, 0u);
  auto load = [&] {
    vis0 = FULL;
    if (v0 != kUnreachable) {
      vis0 = p.vis[v0 >> 5];
      row_of(p, a, v0, b0, n0, d0);
    }
  };
  load();
  bu_scan<kR>(p, o, st.e[warp], [&](BuEntry* ring, uint32_t& cnt) {
    if (base >= nin) return false;
    const uint32_t v = v0;
    const bool cand = !((vis0 >> (v & 31)) & 1u);
    const uint32_t m = __ballot_sync(FULL, cand);
    if (cand) ring[cnt + __popc(m & vxb::lanemask_lt())] = bu_entry(v, b0, n0, d0);
    cnt += __popc(m);
    base += kT;
    v0 = v1;
    const uint32_t i = base + kT + lane;
    v1 = i < nin ? lin[i] : kUnreachable;
    load();
    return base < nin;
  });
}

// ------------------------------------------------------------ full BFS --

// kT threads per block; lbst and bu may share memory.  wbits[0, wbits_n): shared
// words for the block's part of a bitmap.
template <bool kInRepair, int kT, int kR, class Queue>
__device__ void full_bfs(const Params& p, Queue& bq, LbStage& lbst, BuStage<kT, kR>& bu, uint32_t* wbits,
                         uint32_t wbits_n, uint32_t* dist, unsigned long long* trace) {
  BfsCounters* c = p.c;
  const unsigned long long t_start = gtid() == 0 ? globaltimer() : 0ull;  // the repair phases' time budget
  const uint32_t sort_err = kInRepair ? 0u : sort_error(p);
  __shared__ uint32_t seg_n[2];  // entries of this block's segment of each candidate list
  __shared__ unsigned long long red[kT / 32];
  __shared__ LevelWords lw;
  if (threadIdx.x == 0) {
    bq.cnt = 0;
    lw.m = 0;
    lw.n = 0;
  }
  uint32_t V = p.V;
  if constexpr (kInRepair) V = ph.V;
  const uint32_t words = (V + 31) >> 5;
  // one pass sets every vertex unreached and the source at level 0 (bits
  // past V count as visited, so bottom-up never scans them)
  const uint32_t s = p.source;
  const bool has_source = s < V;
  if ((reinterpret_cast<uintptr_t>(dist) & 15) == 0) {  // a caller's own buffer may start anywhere
    const uint4 none = make_uint4(kUnreachable, kUnreachable, kUnreachable, kUnreachable);
    for (uint32_t i = gtid(); i < V / 4; i += nthreads()) {
      uint4 d = none;
      if (i == s / 4) d = make_uint4(s % 4 == 0 ? 0u : d.x, s % 4 == 1 ? 0u : d.y, s % 4 == 2 ? 0u : d.z, s % 4 == 3 ? 0u : d.w);
      reinterpret_cast<uint4*>(dist)[i] = d;
    }
    for (uint32_t i = V / 4 * 4 + gtid(); i < V; i += nthreads()) dist[i] = i == s ? 0u : kUnreachable;
  } else {
    for (uint32_t i = gtid(); i < V; i += nthreads()) dist[i] = i == s ? 0u : kUnreachable;
  }
  for (uint32_t i = gtid(); i < words; i += nthreads()) {
    const uint32_t lo = i * 32;
    const uint32_t sbit = has_source && i == (s >> 5) ? 1u << (s & 31) : 0u;
    p.vis[i] = ((lo + 32 <= V) ? 0u : (FULL << (V - lo))) | sbit;
    p.fb[0][i] = p.fb[1][i] = p.fb[2][i] = 0u;
  }
  if (gtid() == 0) {
    if (sort_err) atomicOr(&c->err, sort_err);
    for (int k = 0; k < 3; ++k) {
      c->lvl_n[k] = 0;
      c->lvl_big[k] = 0;
      c->lvl_m[k] = 0;
    }
    if (has_source) {
      p.q[0][0] = s;
      c->lvl_n[0] = 1;
      c->lvl_m[0] = row_len(p, p.g.out, s);
    } else {
      c->reachable = 0;
      c->levels = 0;
      c->arcs = 0;
    }
  }
  if (!sync_grid(p) || !has_source) return;
  unsigned long long m_visited = 0;
  uint32_t reached = 0;
  bool bottom_up = false, left_bu = false, bu_listed = false;
  bool queued = true;  // the current frontier is in its queue
  uint32_t prev_n = 0;
  uint32_t level = 0;
  // the frontier size and arc count of the current level, read once after the
  // barrier that ends the level before it; a bottom-up level does not count arcs
  uint32_t n_f = ld_cg(&c->lvl_n[0]);
  unsigned long long m_f = __ldcg(&c->lvl_m[0]);
  bool m_known = true;
  // bottom-up candidate lists, cut into one segment per block: the first
  // bottom-up level leaves list 0
  const BuTiles tiles(words, gridDim.x);
  const uint32_t seg = tiles.words() * 32;  // vertices (and list slots) per block
  uint32_t lin = 1;
  uint32_t bits = 0;  // bit k: fb[k] holds the bits of its level's frontier
  // queues, bitmaps and counters rotate over three slots; a stretch of one
  // block's levels takes one turn
  for (uint32_t turn = 0;; ++turn) {
    if (level > V + 1) {
      if (gtid() == 0) atomicOr(&c->err, vxb::kErrLoopBound);
      break;
    }
    const uint32_t cur = turn % 3, nxt = (turn + 1) % 3, clr = (turn + 2) % 3;
    if (n_f == 0) break;
    if (gtid() == 0) {
      c->lvl_n[clr] = 0;
      c->lvl_m[clr] = 0;
      c->lvl_big[clr] = 0;
    }
    if (bottom_up && (double)n_f * p.beta < (double)V && n_f < prev_n) {
      bottom_up = false;
      left_bu = true;
      if (!queued) {  // the frontier's queue, from its bitmap (at most once per search)
        for (uint32_t i0 = gtid() & ~31u; i0 < words; i0 += nthreads()) {
          const uint32_t i = i0 + (threadIdx.x & 31);
          uint32_t w = i < words ? p.fb[cur][i] : 0u;
          while (__any_sync(FULL, w != 0u)) {
            bq_push(bq, w != 0u, i * 32 + (uint32_t)__ffs(w) - 1, p.bar + kQueueWord, p.q[cur]);
            w &= w - 1;
          }
        }
        bq_flush(bq, p.bar + kQueueWord, p.q[cur]);
        if (!sync_grid(p)) return;
        if (gtid() == 0) p.bar[kQueueWord] = 0u;
        queued = true;
      }
    }
    if (!bottom_up && m_known && solo_fits(n_f, m_f)) {
      for (uint32_t k = 0; k < 3; ++k)
        if ((bits >> k) & 1u)
          for (uint32_t i = gtid(); i < words; i += nthreads()) p.fb[k][i] = 0u;
      bits = 0;
      // the state after the stretch, one set per parity of the turn (a block
      // may still read the last stretch's set while block 0 runs the next)
      uint32_t* out = p.bar + kSoloWord + 8 * (turn & 1);
      if (blockIdx.x == 0) {
        SoloState st{level, n_f, reached, m_f, m_visited};
        solo_levels<kT>(p, dist, p.q[cur], p.q[nxt], &c->lvl_n[nxt], bq, lbst, red, trace, st);
        if (threadIdx.x == 0) {
          out[0] = st.level;
          out[1] = st.reached;
          *reinterpret_cast<unsigned long long*>(out + 2) = st.m_visited;
          c->lvl_m[nxt] = st.m_f;
        }
      }
      __shared__ SoloState after;
      vxb::grid_barrier_then(p.bar, p.nblocks, &c->err, [&] {
        lw.failed = __ldcg(&c->err);
        after = SoloState{ld_cg(&out[0]), ld_cg(&c->lvl_n[nxt]), ld_cg(&out[1]), __ldcg(&c->lvl_m[nxt]),
                          __ldcg(reinterpret_cast<unsigned long long*>(out + 2))};
      });
      if (lw.failed) return;
      prev_n = n_f;
      level = after.level;
      n_f = after.n_f;
      reached = after.reached;
      m_f = after.m_f;
      m_visited = after.m_visited;
      continue;
    }
    reached += n_f;
    m_visited += m_f;
    if (!bottom_up && !left_bu && level > 0) {
      // bottom-up when the frontier's rows hold more than 1 / alpha of the
      // arcs of unvisited vertices, and (at the default alpha) nearly as many
      // arcs as there are vertices: the first bottom-up level sweeps every
      // vertex, so a thin frontier of a low-degree graph is cheaper pushed (4096 x
      // 4096 lattice, 620,000 vertices of frontier: three bottom-up levels took 480
      // us, top-down ones take 170; the hub of a star of 2^20 leaves, seen from a
      // leaf: 15 us swept, 45 pushed).  Or when few vertices are left beside a wide
      // frontier, whatever its arcs: the last levels of trees (262,144 and then
      // 782,000 leaves of 2^20 vertices: 30 + 3 us, pushed 202 + 21).  A frontier
      // vertex costs some 90 ps pushed, an unvisited one 15 ps looked at, and every
      // vertex 2 ps swept.
      const unsigned long long m_u = p.total_arcs > m_visited ? p.total_arcs - m_visited : 0ull;
      const double am = (double)m_f * p.alpha;
      const bool few_left = (unsigned long long)(V - reached) <= 4ull * n_f && V <= 16ull * n_f;
      bottom_up = am > (double)m_u && (am > 12.0 * (double)V || few_left);
    }
    if (gtid() == 0 && trace && level < kTraceLevels) {
      trace[2 * level] = globaltimer();
      trace[2 * level + 1] = (unsigned long long)n_f | ((unsigned long long)bottom_up << 63);
    }
    if ((bits >> clr) & 1u)
      for (uint32_t i = gtid(); i < words; i += nthreads()) p.fb[clr][i] = 0u;
    bits &= ~(1u << clr);
    unsigned long long mloc = 0;
    uint32_t nloc = 0;
    const bool td = !bottom_up;
    if (bottom_up) {
      if (!((bits >> cur) & 1u)) {  // the level before kept no bitmap
        for (uint32_t i = gtid(); i < n_f; i += nthreads()) {
          const uint32_t v = p.q[cur][i];
          atomicOr(&p.fb[cur][v >> 5], 1u << (v & 31));
        }
        if (!sync_grid(p)) return;
        bits |= 1u << cur;
      }
      const uint32_t lout = lin ^ 1u;
      if (threadIdx.x == 0) seg_n[lout] = 0;
      // the queue is kept where the block's shared buffer takes it whole or the
      // level is not the first (which reaches most of a graph's vertices)
      const bool push = seg <= sizeof(bq.items) / sizeof(bq.items[0]) || bu_listed;
      const uint32_t nwords = tiles.words();
      const bool local = nwords <= wbits_n;
      if (local)
        for (uint32_t i = threadIdx.x; i < nwords; i += kT) wbits[i] = 0u;
      __syncthreads();
      uint32_t* lists = p.bul + (size_t)blockIdx.x * seg;
      BuOut<Queue> o{dist,  level, p.fb[cur], p.fb[nxt], local ? wbits : nullptr, tiles, lists + (size_t)lout * p.bul_half,
                     &seg_n[lout], push ? &bq : nullptr, p.q[nxt], &c->lvl_n[nxt], 0u};
      if (!bu_listed) bu_first_level(p, V, o, bu);
      else bu_list_level(p, o, bu, lists + (size_t)lin * p.bul_half, seg_n[lin]);
      if (local) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < nwords; i += kT) {
          const uint32_t w = wbits[i];
          if (!w) continue;
          const uint32_t g = tiles.word_of(i);  // no other block writes it
          p.vis[g] |= w;
          p.fb[nxt][g] = w;
        }
      }
      bu_listed = true;
      lin = lout;
      bits |= 1u << nxt;
      m_known = false;
      nloc = o.nloc;
      queued = push;
    } else {
      // a small frontier's level keeps the bitmap (few claims); after a
      // larger one a bottom-up level makes it from the queue
      const bool keep = n_f <= kFlatMax && !left_bu;
      TdVisit<Queue, kT <= 512> t{&p, dist, level, p.q[nxt], keep ? p.fb[nxt] : nullptr, &c->lvl_n[nxt], &bq, 0ull};
      if (n_f <= kFlatMax) {
        lb_stage<kT>(p, p.q[cur], n_f, lbst);
        lb_visit(p, t, n_f, lbst, gwarp(), nwarps());
      } else {
        td_level(p, t, p.q[cur], n_f, &c->lvl_big[cur]);
      }
      if (keep) bits |= 1u << nxt;
      m_known = true;
      queued = true;
      mloc = t.mloc;
    }
    if (!level_end(p, lw, bq, nloc, mloc, nxt, td ? &c->lvl_big[cur] : nullptr)) return;
    prev_n = n_f;
    if (lw.nbig) {  // hub rows remain
      TdVisit<Queue, kT <= 512> t{&p, dist, level, p.q[nxt], nullptr, &c->lvl_n[nxt], &bq, 0ull};
      grid_rows(p, t, lw.nbig);
      if (!level_end(p, lw, bq, 0u, t.mloc, nxt, nullptr)) return;
    }
    n_f = lw.n_f;
    m_f = lw.m_f;
    ++level;
  }
  if (gtid() == 0) {
    c->reachable = reached;
    c->levels = level;
    c->arcs = m_visited;
    // for the repair phases' time budget: the kernel's time (inside an update
    // launch, 512 threads per SM take 1.2 to 1.45 times as long at R-MAT 20 to 22
    // and on the lattice)
    const unsigned long long t = globaltimer() - t_start;
    c->full_ns = kInRepair ? t - t / 4 : t;
    if (trace && level < kTraceLevels) {
      trace[2 * level] = globaltimer();
      trace[2 * level + 1] = 0;
    }
  }
}

// ------------------------------------------------------------- helpers --

__device__ __forceinline__ bool is_sp(const Params& p, uint32_t u, uint32_t v) {
  if (u >= ph.dist_len || v >= ph.dist_len) return false;
  const uint32_t du = p.dist[u], dv = p.dist[v];
  return du != kUnreachable && dv != kUnreachable && du + 1 == dv;
}

__device__ __forceinline__ void reach_add(const Params& p, long long d) {
  if (d) atomicAdd(&p.c->reachable, (unsigned long long)d);
}

// ------------------------------------------------- asynchronous work ring --
// The repair phases are dependency chains a few vertices wide and as deep as
// the tree below a deletion or an insertion.  Level-synchronous rounds would
// pay a grid barrier per level; instead each phase drains a work ring: blocks
// claim items, expand their rows, and push the vertices they change, with no
// barrier until the ring is empty.
//
// The ring holds 64-bit items (kSent = empty slot) at slot[i & ring_mask]:
// bits 0-30 a vertex, bit 31 the cascade's expand kind, bits 32-62 the chunk
// of the vertex's row the item covers (rows longer than kChunk arcs are split
// by the block that claims their first chunk, so a hub is spread over
// blocks), bit 63 the cascade's chunk-check kind;
// head / tail / done count claimed, pushed and finished items.  A block ends
// the phase once it sees done == tail (read in that order): every push happens
// while its pusher's item is unfinished, so at that moment nothing is in
// flight.  Every wait is bounded and records kErrDrainTimeout when it gives up.

constexpr unsigned long long kSent = ~0ull;
constexpr uint32_t kChunk = 128;  // arcs of one ring item: a 32-item round stays within 4096 arcs

// Bit test through L2: bits another block sets during a phase.
__device__ __forceinline__ bool test_bit_cg(const uint32_t* bm, uint32_t v) {
  return (__ldcg(&bm[v >> 5]) >> (v & 31)) & 1u;
}
constexpr uint32_t kKindBit = 0x80000000u;  // cascade items: set = expand an affected vertex
constexpr unsigned long long kChunkCheckBit = 1ull << 63;  // cascade items: one chunk of a long check
constexpr uint32_t kDrainIdleLimit = 1u << 20;  // idle rounds of a block (up to 2 us each)

__device__ __forceinline__ void ring_push(const Params& p, bool pred, unsigned long long item) {
  const uint32_t s = vxb::warp_append(pred, ph.rq_tail);  // warp-uniform
  if (pred) __stcg(&p.ring[(ph.rq_base + s) & p.ring_mask], item);
}

__device__ __forceinline__ uint32_t item_vertex(unsigned long long it) { return (uint32_t)it & ~kKindBit; }
__device__ __forceinline__ uint32_t item_chunk(unsigned long long it) { return (uint32_t)(it >> 32) & 0x7FFFFFFFu; }

// Stages the rows of n <= kThreads items (one per thread; kSent items have no
// row) with their degree prefix in shared memory, then every warp of the block
// takes 32 consecutive arcs of the flattened range per step, so one long row
// is spread over the whole block.  f(valid, x, j) gets the owning item's index
// and is called warp-uniformly.  With 64-bit ring items (p non-null) an item
// covers one kChunk-arc chunk of its row, and the claimer of a row's first
// chunk pushes the rest as items of their own.
template <class T, class F>
__device__ void block_rows(const DevAdj& a, const T* items, uint32_t n, LbStage& st, F& f,
                           const Params* p = nullptr, unsigned long long* acct = nullptr) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ uint32_t wsum[kThreads / 32];
  uint32_t len = 0;
  if (threadIdx.x < n) {
    const T it = items[threadIdx.x];
    uint64_t b = 0, e = 0;
    uint2 dr = make_uint2(0, 0);
    if (it != (T)kSent) {
      const uint32_t u = (uint32_t)it & ~kKindBit;
      vxb::base_range(a, u, b, e);
      dr = a.drow[u];
    }
    uint32_t blen = (uint32_t)(e - b), dx = dr.x, dlen = dr.y;
    if (p && it != (T)kSent) {
      const uint32_t total = blen + dlen, c = (uint32_t)((unsigned long long)it >> 32) & 0x7FFFFFFFu;
      const uint32_t lo = c * kChunk, hi = min(total, lo + kChunk);
      if (c == 0 && total > kChunk) {  // hand the other chunks to other blocks
        const uint32_t more = (total - 1) / kChunk;
        const uint32_t s0 = ph.rq_base + atomicAdd(ph.rq_tail, more);
        for (uint32_t k = 0; k < more; ++k)
          __stcg(&p->ring[(s0 + k) & p->ring_mask], ((unsigned long long)it & 0xFFFFFFFFull) |
                                                        ((unsigned long long)(k + 1) << 32));
      }
      const uint32_t bl = lo < blen ? min(blen, hi) - lo : 0u;
      const uint32_t dl = hi > max(lo, blen) ? hi - max(lo, blen) : 0u;
      b += lo < blen ? lo : blen;
      dx += lo > blen ? lo - blen : 0u;
      blen = bl;
      dlen = dl;
    }
    st.base[threadIdx.x] = b;
    st.blen[threadIdx.x] = blen;
    st.dx[threadIdx.x] = dx;
    len = blen + dlen;
  }
  uint32_t incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < kThreads / 32 ? wsum[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < kThreads / 32) wsum[lane] = wi - w;
  }
  __syncthreads();
  const uint32_t ex = wsum[warp] + incl - len;
  if (threadIdx.x < n) st.pref[threadIdx.x] = ex;
  if (threadIdx.x + 1 == n) st.pref[n] = ex + len;
  __syncthreads();
  const uint32_t M = n ? st.pref[n] : 0u;
  if (acct && threadIdx.x == 0 && M) atomicAdd(&acct[0], (unsigned long long)M);
  for (uint32_t e0 = (uint32_t)warp * 32; e0 < M; e0 += kThreads) {
    const uint32_t e = e0 + lane;
    bool valid = false;
    uint32_t x = 0, j = 0;
    if (e < M) {
      uint32_t lo = 0, hi = n;  // last j with pref[j] <= e
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (st.pref[mid] <= e) lo = mid;
        else hi = mid;
      }
      j = lo;
      const uint32_t k = e - st.pref[j];
      if (k < st.blen[j]) {
        x = a.col[st.base[j] + k];
        valid = !(x & kTomb);
        x &= kIdMask;
      } else {
        x = a.darena[st.dx[j] + (k - st.blen[j])];
        valid = true;
      }
    }
    f(valid, x, j);
  }
  __syncthreads();  // st is reused by the next call
}

// The words a repair phase decides by, as of the last grid barrier.
struct RepairWords {
  unsigned long long deadline;
  uint32_t failed, candidates, touched, affected, fallback, cbig, rbig, tail, big_b, later, raw_f[2];
};

// Grid barrier of the repair phases: thread 0 of each block loads the words
// above once, all in flight together (each phase loading what it needs in
// every thread cost a dependent round trip per word and thousands of requests
// for one line).  A block may load them while another is already in the next
// phase, so a word may be used only where the next phase does not change it, or
// only in a direction that does not change what is decided by it.  False once
// any block recorded a device error.
__device__ __forceinline__ bool sync_words(const Params& p, RepairWords& w) {
  BfsCounters* c = p.c;
  vxb::grid_barrier_then(p.bar, p.nblocks, &c->err, [&] {
    RepairWords r;
    r.failed = __ldcg(&c->err);
    r.candidates = ld_cg(&c->cand_n);
    r.touched = ph.touched_base + ld_cg(&c->touched_n);
    r.affected = ld_cg(&c->a_n);
    r.fallback = ld_cg(&c->fallback);
    r.cbig = ld_cg(&c->cbig);
    r.rbig = ld_cg(&c->rbig);
    r.tail = ld_cg(ph.rq_tail);
    r.big_b = ld_cg(&c->big_b);
    r.later = ld_cg(&c->later);
    r.raw_f[0] = ld_cg(p.bar + kRawWord);
    r.raw_f[1] = ld_cg(p.bar + kRawWord + 1);
    r.deadline = __ldcg(&c->deadline);
    w = r;
  });
  return w.failed == 0u;
}

// Warps (threads) numbered across the blocks first, so that a few items spread
// over every SM.
__device__ __forceinline__ uint32_t dealt_warp() { return (threadIdx.x >> 5) * gridDim.x + blockIdx.x; }
__device__ __forceinline__ uint32_t dealt_thread() { return threadIdx.x * gridDim.x + blockIdx.x; }

// Shared memory of one block for the repair phases.
struct RepairSmem {
  unsigned long long items[kThreads];  // claimed ring items
  uint32_t sv[kThreads];     // check items (vertex); boundary chunk vertices
  unsigned long long ex[kThreads];     // expand items (vertex, chunk)
  uint32_t cnt[kThreads];    // chunk + 1 of a chunk-check sv item (0: plain check); boundary minima
  uint32_t d[kThreads];      // distance of each staged item
  uint32_t g0, n, stop, nsv, nex, fallback;
  uint32_t late;     // the round started past the phase's deadline (its items are dropped)
  uint32_t flagged;  // this block has raised the phase's handover flag
  RepairWords w;     // kept across a BFS in the memory before it
};

// The full BFS inside a repair kernel, in the shared memory its phases do not
// hold at that point.  It is a function of its own (called, not inlined), which reads
// the parameters faster from a copy in shared memory than by reference from the
// kernel's (fallback batches on a 512 x 512 lattice 1,127 us each, so 1,080).
__device__ __noinline__ void bfs_in_repair(const Params& p, RepairSmem& sm, LbStage& lb, BlockQueue& bq, uint32_t* dist,
                              unsigned long long* trace) {
  using Stage = BuStage<kThreads, 1>;
  static_assert(sizeof(Stage) <= sizeof(LbStage) && alignof(LbStage) >= alignof(Stage), "the two share memory");
  static_assert(sizeof(Params) % 4 == 0, "copied by words");
  __shared__ Params own;
  for (uint32_t i = threadIdx.x; i < sizeof(Params) / 4; i += kThreads)
    reinterpret_cast<uint32_t*>(&own)[i] = reinterpret_cast<const uint32_t*>(&p)[i];
  __syncthreads();
  full_bfs<true>(own, bq, lb, reinterpret_cast<Stage&>(lb), reinterpret_cast<uint32_t*>(&sm),
                 (uint32_t)(offsetof(RepairSmem, w) / 4), dist, trace);
}

// Drains the ring; W::process(sm, n) handles sm.items[0, n) block-uniformly,
// with sm.late set for a round that starts at or past the deadline (a
// globaltimer value read once per round by warp 0, no memory access).
//
// A block takes a ticket of kClaim consecutive ring indices (one atomicAdd,
// which never fails) and warp 0 polls the ticket's own slots: items pushed
// into them are processed as they arrive, and the next ticket is taken once
// the current one is used up.  Indices past the tail belong to whichever
// block holds them, so pushes spread over the blocks waiting for work, and no
// two blocks poll the same address.  Every few idle rounds a block checks
// done == tail; the first to see it raises rq_fin, which the other idle
// blocks read every round, and all leave the phase.
constexpr uint32_t kClaim = 32;

template <class W>
__device__ void drain(const Params& p, RepairSmem& sm, W& w, unsigned long long deadline) {
  BfsCounters* c = p.c;
  const int lane = threadIdx.x & 31;
  uint32_t cur = 0, end = 0;  // warp 0's ticket [cur, end), uniform over its lanes
  uint32_t idle = 0;
  if (threadIdx.x == 0) sm.flagged = 0;
  for (;;) {
    if (threadIdx.x < 32) {
      uint32_t n = 0, stop = 0;
      if (ld_cg(&c->err)) {
        stop = 1;
      } else {
        if (cur == end) {
          uint32_t s0 = 0;
          if (lane == 0) {
            s0 = atomicAdd(p.rq_head, kClaim);
            atomicAdd(&p.rq_stat[1], 1ull);
          }
          cur = __shfl_sync(FULL, s0, 0);
          end = cur + kClaim;
        }
        const uint32_t k = cur + lane;
        unsigned long long v = kSent;
        if (k < end) v = __ldcg(&p.ring[(ph.rq_base + k) & p.ring_mask]);
        const uint32_t have = __ballot_sync(FULL, v != kSent);
        n = have == FULL ? 32u : (uint32_t)(__ffs(~have) - 1);  // leading filled slots
        if ((uint32_t)lane < n) {
          sm.items[lane] = v;
          __stcg(&p.ring[(ph.rq_base + k) & p.ring_mask], kSent);
        }
        cur += n;
        if (n == 0) {
          uint32_t st = 0;
          if (lane == 0) {
            st = ld_cg(p.rq_fin);
            if (!st && (idle & 3) == 3) {
              const uint32_t dn = ld_cg(p.rq_done);
              __threadfence();
              st = dn == ld_cg(ph.rq_tail);
              if (st) atomicExch(p.rq_fin, 1u);  // releases the other blocks at their next idle round
              atomicAdd(&p.rq_stat[3], 1ull);
            }
          }
          stop = __shfl_sync(FULL, st, 0);
        }
      }
      if (lane == 0) {
        sm.n = n;
        sm.stop = stop;
        sm.late = n && globaltimer() >= deadline;
      }
    }
    __syncthreads();
    const uint32_t n = sm.n, stop = sm.stop;
    __syncthreads();  // every thread has read the words before warp 0 rewrites them
    if (stop) break;
    if (n == 0) {
      if (threadIdx.x == 0) atomicAdd(&p.rq_stat[2], 1ull);
      if (++idle > kDrainIdleLimit) {
        if (threadIdx.x == 0) atomicOr(&c->err, vxb::kErrDrainTimeout);
        break;
      }
      __nanosleep(32u << min(idle >> 2, 4u));  // back off to 512 ns
      continue;
    }
    idle = 0;
    const long long t0 = clock64();
    w.process(sm, n);
    __syncthreads();
    if (threadIdx.x == 0) {
      acct_add(p, 1, n);
      __threadfence();  // this block's pushes are visible before its items count as done
      atomicAdd(p.rq_done, n);
      atomicAdd(&p.rq_stat[0], 1ull);
      const unsigned long long dt = (unsigned long long)(clock64() - t0);
      atomicAdd(&p.rq_stat[4], dt);
      atomicMax(&p.rq_stat[5], dt);
    }
  }
}

// A phase's first items are taken in rounds with a grid barrier between them, a
// warp per item, before the ring is drained asynchronously: most batches leave a
// few dozen items of one or two hops, and a drain's tickets, polls and
// termination test take longer than a barrier (1,000 directed ops at 300,000
// vertices, 2 items: cascade 20 us drained, 16 in rounds; 10,000 ops at R-MAT 22, 58
// items: 33 and 27).  A phase that is not done after kSyncRounds rounds,
// or has more items than blocks, is deep or wide enough to drain.  w.one
// handles an item (whole warp) that it has taken out of the ring.  sm.w is of
// the last barrier; true when the ring is empty, false to drain (or on an
// error, sm.w.failed).
//
// What a round pushes is an epoch of its own, with its own length word and the
// slots behind the epoch before: a block that is late to read a round's length
// must not see pushes of the next round in it.  (A first epoch that is drained
// only grows, past the limit that sends it to the drain.)
constexpr uint32_t kSyncRounds = 2;

// One thread of a block.
__device__ __forceinline__ void ring_epoch(const Params& p, uint32_t epoch, uint32_t base) {
  ph.rq_tail = p.rq_tail + epoch;
  ph.rq_base = base;
}

template <class W>
__device__ bool sync_rounds(const Params& p, RepairSmem& sm, W& w) {
  if (p.handover == 0.0f) return false;  // hands over at its first drain round
  for (uint32_t r = 0; r < kSyncRounds; ++r) {
    const uint32_t lo = ph.rq_base, n = sm.w.tail;
    if (n == 0) return true;
    if (n > gridDim.x) return false;
    __syncthreads();  // every warp has read the epoch before
    if (threadIdx.x == 0) ring_epoch(p, r + 1, lo + n);
    __syncthreads();
    const uint32_t i = dealt_warp();
    if (i < n) {
      unsigned long long* slot = &p.ring[(lo + i) & p.ring_mask];
      const unsigned long long it = __ldcg(slot);
      __syncwarp();
      if ((threadIdx.x & 31) == 0) {
        __stcg(slot, kSent);
        acct_add(p, 1, 1);
      }
      w.one(it);
    }
    if (!sync_words(p, sm.w)) return false;
  }
  return sm.w.tail == 0;
}

// --------------------------------------------------- pre-batch fixpoint --
//
// compute_affected_prebatch (bfs.hpp:222-259): a touched vertex x at
// distance d is affected iff none of its shortest parents survives -- every
// in-neighbour at d-1 is reached over a deleted arc or is affected itself
// (the reference's lost >= support).  The fixpoint does not depend on the
// order, so it runs as one asynchronous cascade with a witness per vertex:
//
//   check(x)   scan x's in-row from the saved position for the first parent
//              that survives and is not affected; record it as the witness,
//              or mark x affected when the row is exhausted.  Affectedness
//              only grows, so a rescan never goes back.
//   expand(y)  y became affected: its children whose witness is y (or that
//              no check has touched yet) get a check.
//
// In-rows longer than kChunk arcs are checked in chunks by many warps at once
// (chunk_check); their passes always start from the row's beginning.
//
// sw[x] packs bit 63 touched, bits 32-62 witness + 1 (0 = none yet), bits
// 0-31 the scan position.  A check stores its witness, fences, and re-reads
// the witness's affected bit; mark_affected sets the bit and fences before
// the expand item is pushed -- so either the check sees the parent affected
// and scans on, or the expansion sees the witness and asks for a recheck.
// Requests are deduplicated by a bit in inq[1], cleared when a check starts.

constexpr unsigned long long kSwTouched = 1ull << 63;

// Marks v affected once (the affected bit decides); true for the caller that set it.
__device__ __forceinline__ bool mark_affected(const Params& p, uint32_t v) {
  const uint32_t bit = 1u << (v & 31);
  if (atomicOr(&p.aff[v >> 5], bit) & bit) return false;
  const uint32_t slot = atomicAdd(&p.c->a_n, 1u);
  p.lst_a[slot] = v;
  if (slot + 1 > ph.fallback_limit) p.c->fallback = 1;
  __threadfence();  // the affected bit is visible before the expand item is
  return true;
}

// Warp-uniform: request a check of x where pred holds (first touch is recorded
// in sw and in the touched list; a pending request is not repeated).  The
// touched-list and ring reservations are one atomic each, both in flight
// before either result is used.
__device__ __forceinline__ void request_check(const Params& p, bool pred, uint32_t x) {
  bool first = false, push = false;
  if (pred) {
    first = !(atomicOr(&p.sw[x], kSwTouched) & kSwTouched);
    const uint32_t bit = 1u << (x & 31);
    push = !(atomicOr(&p.inq[1][x >> 5], bit) & bit);
  }
  const uint32_t mf = __ballot_sync(FULL, first), mp = __ballot_sync(FULL, push);
  if (!(mf | mp)) return;
  const int lane = threadIdx.x & 31;
  const int lf = mf ? __ffs(mf) - 1 : 0, lp = mp ? __ffs(mp) - 1 : 0;
  uint32_t bf = 0, bp = 0;
  if (mf && lane == lf) bf = atomicAdd(&p.c->touched_n, (uint32_t)__popc(mf));
  if (mp && lane == lp) bp = atomicAdd(ph.rq_tail, (uint32_t)__popc(mp));
  bf = __shfl_sync(FULL, bf, lf);
  bp = __shfl_sync(FULL, bp, lp);
  const uint32_t lt = vxb::lanemask_lt();
  if (first) p.lst_t[ph.touched_base + bf + __popc(mf & lt)] = x;
  if (push) __stcg(&p.ring[(ph.rq_base + bp + __popc(mp & lt)) & p.ring_mask], (unsigned long long)x);
}

// expand(y) for a newly affected y at distance dy, applied to one arc (y, x)
// of y's out-row (warp-uniform): x gets a check if it sits at dy + 1 and its
// witness is y or no check has touched it yet.
constexpr uint32_t kInlineExpand = 64;  // out-rows this short are expanded by the warp that marked y
struct ExpandChildren {
  const Params* p;
  uint32_t y, dy;
  __device__ __forceinline__ void operator()(bool valid, uint32_t x, uint32_t) {
    bool need = false;
    if (valid && x < ph.dist_len) {
      const uint32_t dx = p->dist[x];
      const unsigned long long w = __ldcg(&p->sw[x]);
      const uint32_t wit = (uint32_t)(w >> 32) & 0x7FFFFFFFu;
      need = dx == dy + 1 && (!(w & kSwTouched) || wit == y + 1);
    }
    request_check(*p, need, x);
  }
};

// First position k in [lo, hi) of x's in-row (base part [b, b + nb), delta
// part from darena[dx]) whose tail y survives, sits at distance d - 1 and is
// not affected; whole warp, warp-uniform result.  Each step covers 128 arcs:
// every lane issues its four column loads, then the four distance and
// affected-bit loads, so a step costs two dependent round trips however many
// of its arcs are needed.
__device__ __forceinline__ bool find_parent(const Params& p, const DevAdj& a, uint64_t b, uint32_t nb, uint32_t dx,
                                            uint32_t lo, uint32_t hi, uint32_t d, uint32_t& kw, uint32_t& yw) {
  const int lane = threadIdx.x & 31;
  for (uint32_t k0 = lo; k0 < hi; k0 += 128) {
    if (lane == 0) acct_add(p, 0, min(128u, hi - k0));
    uint32_t y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t k = k0 + 32 * j + lane;
      y[j] = kTomb;  // no arc
      if (k < hi) y[j] = k < nb ? a.col[b + k] : a.darena[dx + (k - nb)];
    }
    uint32_t dy[4], aw[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool live = !(y[j] & kTomb) && y[j] < ph.dist_len;
      dy[j] = live ? p.dist[y[j]] : kUnreachable;
      aw[j] = live ? __ldcg(&p.aff[y[j] >> 5]) : 0u;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool ok = dy[j] != kUnreachable && dy[j] + 1 == d && !((aw[j] >> (y[j] & 31)) & 1u);
      const uint32_t ball = __ballot_sync(FULL, ok);
      if (ball) {
        const int f = __ffs(ball) - 1;
        kw = k0 + 32 * j + (uint32_t)f;
        yw = __shfl_sync(FULL, y[j], f);
        return true;
      }
    }
  }
  return false;
}

// check(x), whole warp.  The scan resumes at the position saved in sw[x]:
// affectedness only grows and distances are fixed during the cascade, so an
// arc that failed once fails again.  In-rows longer than kChunk arcs are
// scanned in place over their first chunk only; when it holds no witness the
// rest goes to a chunked pass (chunk_check), and the saved position kChunk
// tells later checks to go straight to a new pass.  A candidate's first check
// (kFirst) answers no request and starts at position 0: nothing relies on it
// clearing the request bit, and neither that nor the saved state is a round
// trip of its chain.
template <bool kFirst>
__device__ void check_vertex(const Params& p, uint32_t x) {
  const DevAdj& a = p.g.in;
  const int lane = threadIdx.x & 31;
  // x's distance and row bounds do not change during the cascade: they load
  // together with the clearing of the request bit
  const uint32_t d = p.dist[x];
  uint64_t b, e;
  vxb::base_range(a, x, b, e);
  const uint2 dr = a.drow[x];
  if (!kFirst) {
    if (lane == 0) atomicAnd(&p.inq[1][x >> 5], ~(1u << (x & 31)));
    __syncwarp();
    __threadfence();  // the request bit is clear before the state (witness, affected bits) is read
  }
  const uint32_t nb = (uint32_t)(e - b), total = nb + dr.y;
  const uint32_t lim = min(total, kChunk);
  uint32_t k0 = kFirst ? 0u : (uint32_t)__ldcg(&p.sw[x]);
  bool resolved = false;
  uint32_t kw = 0, yw = 0;
  while (k0 < lim && !resolved) {
    if (!find_parent(p, a, b, nb, dr.x, k0, lim, d, kw, yw)) break;
    bool still = false;
    if (lane == 0) {
      __stcg(&p.sw[x], kSwTouched | ((unsigned long long)(yw + 1) << 32) | kw);
      __threadfence();
      still = !test_bit_cg(p.aff, yw);
    }
    resolved = __shfl_sync(FULL, still, 0);
    k0 = kw + 1;  // the witness turned affected meanwhile: scan on past it
  }
  if (resolved) return;
  if (total > kChunk) {
    // the rest of a long in-row: one chunk-check item per kChunk arcs past the
    // first, scanned by many warps; tent[x] counts the chunks of the pass in
    // flight.  A request that finds a pass in flight is covered by it: the
    // pass clears tent[x] before it verifies its final witness.
    const uint32_t K = (total + kChunk - 1) / kChunk - 1;
    bool start = false;
    if (lane == 0) {
      __stcg(&p.sw[x], kSwTouched | (unsigned long long)kChunk);
      start = atomicCAS(&p.tent[x], 0u, K) == 0u;
    }
    start = __shfl_sync(FULL, start, 0);
    if (start)
      for (uint32_t c0 = 0; c0 < K; c0 += 32)
        ring_push(p, c0 + lane < K, kChunkCheckBit | ((unsigned long long)(c0 + lane + 1) << 32) | x);
    return;
  }
  bool marked = false;
  if (lane == 0) {
    __stcg(&p.sw[x], kSwTouched | (unsigned long long)total);
    marked = mark_affected(p, x);
  }
  marked = __shfl_sync(FULL, marked, 0);
  bool inlined = false;
  if (marked) {
    // a short out-row is expanded here instead of through one more ring round;
    // every lane fences after the affected bit (set and fenced by lane 0)
    // before it reads a child's witness, as the expanding block does after
    // claiming an expand item
    __syncwarp();
    __threadfence();
    // past the fallback limit the block path drops expansions; so does
    // this one (past the deadline its later rounds drop what this pushes)
    const uint32_t odeg = degree_of(p.g.out, x);
    if (odeg <= kInlineExpand && !ld_cg(&p.c->fallback)) {
      if (lane == 0) acct_add(p, 0, odeg);
      ExpandChildren ec{&p, x, d};
      warp_row(p.g.out, x, ec);
      inlined = true;
    }
  }
  ring_push(p, marked && !inlined && lane == 0, (unsigned long long)(x | kKindBit));
}

// One chunk c >= 1 of a long check (whole warp): scan [c * kChunk,
// (c + 1) * kChunk) of x's in-row for a surviving, non-affected parent, unless
// another chunk found one already (kFoundBit in tent[x]).  The last chunk of
// the pass clears tent[x], then either verifies the recorded witness (asking
// for a new check if it turned affected) or, when no chunk found one, marks x
// affected.  Witnesses are recorded with the saved position kChunk (the first
// chunk is known to hold none).
constexpr uint32_t kFoundBit = 0x80000000u;

__device__ void chunk_check(const Params& p, uint32_t x, uint32_t c) {
  const DevAdj& a = p.g.in;
  const int lane = threadIdx.x & 31;
  const uint32_t d = p.dist[x];
  uint64_t b, e;
  vxb::base_range(a, x, b, e);
  const uint2 dr = a.drow[x];
  const uint32_t nb = (uint32_t)(e - b), total = nb + dr.y;
  const uint32_t hi = min(total, (c + 1) * kChunk);
  uint32_t k0 = c * kChunk;
  bool found = (ld_cg(&p.tent[x]) & kFoundBit) != 0u;
  uint32_t kw = 0, yw = 0;
  while (k0 < hi && !found) {
    if (!find_parent(p, a, b, nb, dr.x, k0, hi, d, kw, yw)) break;
    bool good = false;
    if (lane == 0) {
      __stcg(&p.sw[x], kSwTouched | ((unsigned long long)(yw + 1) << 32) | kChunk);
      __threadfence();
      good = !test_bit_cg(p.aff, yw);
      if (good) atomicOr(&p.tent[x], kFoundBit);
    }
    found = __shfl_sync(FULL, good, 0);
    k0 = kw + 1;
  }
  bool recheck = false, aff = false;
  if (lane == 0) {
    __threadfence();
    const uint32_t old = atomicSub(&p.tent[x], 1u);
    if ((old & ~kFoundBit) == 1u) {  // the pass's last chunk
      atomicExch(&p.tent[x], 0u);
      __threadfence();
      if (old & kFoundBit) {
        const uint32_t w1 = (uint32_t)(__ldcg(&p.sw[x]) >> 32) & 0x7FFFFFFFu;
        recheck = w1 == 0u || test_bit_cg(p.aff, w1 - 1);
      } else {
        aff = mark_affected(p, x);
      }
    }
  }
  request_check(p, recheck, x);
  ring_push(p, aff, (unsigned long long)(x | kKindBit));
}

// An expand item (y, chunk) by one warp: the item's arcs of y's out-row, all of
// a short row's; the other chunks of a longer one are queued by its first.
__device__ void expand_one(const Params& p, unsigned long long it) {
  const DevAdj& a = p.g.out;
  const uint32_t lane = threadIdx.x & 31, y = item_vertex(it), c = item_chunk(it);
  const uint32_t dy = p.dist[y];
  uint64_t b, e;
  vxb::base_range(a, y, b, e);
  const uint2 dr = a.drow[y];
  const uint32_t nb = (uint32_t)(e - b), total = nb + dr.y;
  const uint32_t hi = min(total, (c + 1) * kChunk);
  if (c == 0)
    for (uint32_t k = 1 + lane; (k - lane) * kChunk < total; k += 32)
      ring_push(p, k * kChunk < total, (unsigned long long)(y | kKindBit) | ((unsigned long long)k << 32));
  if (lane == 0) acct_add(p, 0, hi - c * kChunk);
  ExpandChildren ec{&p, y, dy};
  for (uint32_t k0 = c * kChunk; k0 < hi; k0 += 32) {
    const uint32_t k = k0 + lane;
    const uint32_t x = k >= hi ? kTomb : k < nb ? a.col[b + k] : a.darena[dr.x + (k - nb)];
    ec(!(x & kTomb), x & kIdMask, 0u);
  }
}

struct Cascade {
  const Params* p;
  LbStage* lb;
  // One item by one warp.  Past the fallback limit it is dropped like process
  // drops its items.
  __device__ void one(unsigned long long it) {
    if (ld_cg(&p->c->fallback)) {
      if (!(it & kChunkCheckBit) && !((uint32_t)it & kKindBit) && (threadIdx.x & 31) == 0)
        atomicAnd(&p->inq[1][(uint32_t)it >> 5], ~(1u << ((uint32_t)it & 31)));
      return;
    }
    __threadfence();  // expand items were pushed after their affected bits
    if (it & kChunkCheckBit) chunk_check(*p, item_vertex(it), item_chunk(it));
    else if ((uint32_t)it & kKindBit) expand_one(*p, it);
    else check_vertex<false>(*p, (uint32_t)it);
  }
  __device__ void process(RepairSmem& sm, uint32_t n) {
    const Params& P = *p;
    BfsCounters* c = P.c;
    const uint32_t t = threadIdx.x;
    if (t == 0) {
      sm.nsv = 0;
      sm.nex = 0;
      // past its deadline the cascade drops the rest of its queue like the
      // fallback does; a BFS then gives the affected set (cascade_by_bfs)
      if (sm.late && !sm.flagged) {
        atomicOr(&c->cbig, 1u);
        sm.flagged = 1;
      }
      sm.fallback = ld_cg(&c->fallback) | sm.late;
    }
    __syncthreads();
    if (t < n) {
      const unsigned long long it = sm.items[t];
      if (it != kSent) {
        if (it & kChunkCheckBit) {
          const uint32_t k = atomicAdd(&sm.nsv, 1u);
          sm.sv[k] = item_vertex(it);
          sm.cnt[k] = item_chunk(it) + 1;
        } else if ((uint32_t)it & kKindBit) {
          sm.ex[atomicAdd(&sm.nex, 1u)] = it;
        } else {
          const uint32_t k = atomicAdd(&sm.nsv, 1u);
          sm.sv[k] = (uint32_t)it;
          sm.cnt[k] = 0u;
        }
      }
    }
    __threadfence();  // expand items were pushed after their affected bits
    __syncthreads();
    if (sm.fallback) {
      // past the fallback limit or the budget: drop the items, keeping the
      // request bits clear
      for (uint32_t i = t; i < sm.nsv; i += kThreads)
        if (sm.cnt[i] == 0u) atomicAnd(&P.inq[1][sm.sv[i] >> 5], ~(1u << (sm.sv[i] & 31)));
      return;
    }
    const uint32_t nsv = sm.nsv, nex = sm.nex;
    for (uint32_t i = t >> 5; i < nsv; i += kThreads / 32) {
      if (sm.cnt[i]) chunk_check(P, sm.sv[i], sm.cnt[i] - 1);
      else check_vertex<false>(P, sm.sv[i]);
    }
    if (nex) {
      if (t < nex) sm.d[t] = P.dist[item_vertex(sm.ex[t])];
      __syncthreads();
      auto expand = [&](bool valid, uint32_t x, uint32_t j) {
        bool need = false;
        if (valid && x < ph.dist_len) {  // both loads in flight together
          const uint32_t dx = P.dist[x];
          const unsigned long long w = __ldcg(&P.sw[x]);
          const uint32_t wit = (uint32_t)(w >> 32) & 0x7FFFFFFFu;
          need = dx == sm.d[j] + 1 && (!(w & kSwTouched) || wit == item_vertex(sm.ex[j]) + 1);
        }
        request_check(P, need, x);
      };
      block_rows(P.g.out, sm.ex, nex, *lb, expand, &P, P.acct);
    }
  }
};

// Between a barrier after the ring's last use and one before its next.
__device__ void reset_ring(const Params& p) {
  if (threadIdx.x == 0) ring_epoch(p, 0, 0);
  if (gtid() == 0) {
    *p.rq_head = 0;
    for (uint32_t k = 0; k <= kSyncRounds; ++k) p.rq_tail[k] = 0;
    *p.rq_done = 0;
    *p.rq_fin = 0;
    for (int k = 0; k < 6; ++k) p.rq_stat[k] = 0;
  }
}

__device__ __forceinline__ void stamp(const Params& p, int k) {
  if (gtid() == 0) p.c->rtrace[k] = globaltimer();
}

// Deletion candidates (bfs.hpp:52-63): heads of deleted shortest-parent arcs.
// The first touch of each records it in the touched list, so the list's
// first cand_n entries are the candidates.  Warp-uniform.
__device__ void register_candidates(const Params& p) {
  BfsCounters* c = p.c;
  const int lane = threadIdx.x & 31;
  const uint32_t F = *ph.F;
  for (uint32_t base = gwarp() * 32; base < F; base += nwarps() * 32) {
    const uint32_t i = base + lane;
    bool first = false;
    uint32_t v = 0;
    if (i < F) {
      const uint8_t f = ph.ff[i];
      const uint32_t u = ph.fu[i];
      v = ph.fv[i];
      if (!(f & kFAdd) && (f & kFCur) && is_sp(p, u, v)) first = !(atomicOr(&p.sw[v], kSwTouched) & kSwTouched);
    }
    const uint32_t slot = vxb::warp_append(first, &c->touched_n);
    if (first) p.lst_t[slot] = v;
    vxb::warp_append(first, &c->cand_n);
  }
}

__device__ void clear_workspace(const Params& p, uint32_t touched, uint32_t affected);

// The cascade past its time budget (a cut near the root of a deep graph
// leaves millions of vertices affected, and the cascade walks them level by
// level).
// A vertex keeps its distance through the batch's deletions iff one of its
// shortest paths survives them, i.e. iff it has a surviving parent that is not
// affected itself: the affected vertices are exactly those whose distance in
// the graph without the deletions exceeds their old one.  One BFS of that graph
// (the deletions are committed, the insertions not yet) gives them: its
// distances replace the old ones, the count of raised vertices is the batch's
// affected count (and decides the fallback as the cascade's would), and the
// affected list stays empty, so the post-batch repair only relaxes the
// insertions.  The BFS distances go to tent (zero between phases), which the
// comparison pass zeroes again.
__device__ __noinline__ bool cascade_by_bfs(const Params& p, RepairSmem& sm, BlockQueue& bq, LbStage& lb) {
  BfsCounters* c = p.c;
  clear_workspace(p, sm.w.touched, sm.w.affected);
  reset_ring(p);
  if (!sync_grid(p)) return false;
  unsigned long long arcs = 0;
  uint32_t levels = 0;
  if (gtid() == 0) {  // the last full BFS's figures stand
    arcs = c->arcs;
    levels = c->levels;
    c->touched_n = 0;
    c->a_n = 0;
    c->a_bfs = 0;
  }
  bfs_in_repair(p, sm, lb, bq, p.tent, nullptr);  // also sets the reachable count of the graph without the deletions
  if (!sync_grid(p)) return false;
  uint32_t raised = 0;
  for (uint32_t v = gtid(); v < ph.dist_len; v += nthreads()) {
    const uint32_t d0 = p.dist[v], d1 = p.tent[v];
    p.tent[v] = 0u;
    raised += d0 != kUnreachable && d1 > d0;
    p.dist[v] = d1;
  }
  raised = vxb::warp_sum(raised);
  if ((threadIdx.x & 31) == 0 && raised) atomicAdd(&c->a_bfs, raised);
  if (!sync_grid(p)) return false;
  if (gtid() == 0) {
    const uint32_t na = c->a_bfs;
    c->affected = na;
    if (na > ph.fallback_limit) c->fallback = 1;  // bfs.hpp:249, 258: more than the limit falls back
    c->arcs = arcs;
    c->levels = levels;
    c->cbig = 0u;
    c->a_bfs = 0u;
    c->handovers[0] += 1;
  }
  return true;
}

// The cascade after the candidates are registered (and the batch's deletions
// committed): every candidate is checked in place, one warp each; the ring
// is drained only when a check left work in it (an affected vertex to expand,
// chunks of a long in-row), which most small batches never do.  Records the
// batch's affected count.
__device__ bool cascade(const Params& p, RepairSmem& sm, LbStage& lb, BlockQueue& bq, uint32_t ncand) {
  if (gtid() == 0) set_deadline(p);
  for (uint32_t i = dealt_warp(); i < ncand; i += nwarps()) check_vertex<true>(p, p.lst_t[i]);
  if (!sync_words(p, sm.w)) return false;
  if (sm.w.tail) {
    Cascade w{&p, &lb};
    if (!sync_rounds(p, sm, w)) {
      if (sm.w.failed) return false;
      drain(p, sm, w, ph.cascade_bfs ? sm.w.deadline : kNever);
      if (!sync_words(p, sm.w)) return false;
    }
  }
  if (gtid() == 0) {  // the drain statistics of the phase trace
    p.c->rtrace[7] = ph.rq_base + sm.w.tail;
    for (int k = 0; k < 6; ++k) p.c->rtrace[9 + k] = __ldcg(&p.rq_stat[k]);
  }
  if (sm.w.cbig) return cascade_by_bfs(p, sm, bq, lb);
  if (gtid() == 0) p.c->affected = sm.w.affected;
  return true;
}

__device__ void repair_pre(const Params& p, RepairSmem& sm, LbStage& lb, BlockQueue& bq) {
  BfsCounters* c = p.c;
  stamp(p, 0);
  reset_ring(p);
  if (!sync_grid(p)) return;
  register_candidates(p);
  if (!sync_grid(p)) return;
  stamp(p, 1);
  const uint32_t ncand = ld_cg(&c->cand_n);
  if (gtid() == 0) c->candidates = ncand;
  if (ncand == 0) return;
  if (!cascade(p, sm, lb, bq, ncand)) return;
  stamp(p, 2);
  reset_ring(p);  // for the post-batch kernel
}

// -------------------------------------------------- post-batch repair --

__device__ void clear_workspace(const Params& p, uint32_t nt, uint32_t na) {
  for (uint32_t i = gtid(); i < nt; i += nthreads()) {
    p.sw[p.lst_t[i]] = 0ull;
    p.tent[p.lst_t[i]] = 0u;  // chunk counts left by a pass the fallback dropped
  }
  for (uint32_t i = gtid(); i < na; i += nthreads()) p.aff[p.lst_a[i] >> 5] = 0u;
}

// Lower dist[x] to cand; true when this thread lowered it (INF -> finite
// counted in reach).
__device__ __forceinline__ bool lower(const Params& p, uint32_t x, uint32_t cand, long long& reach) {
  if (cand >= ld_cg(&p.dist[x])) return false;
  const uint32_t old = atomicMin(&p.dist[x], cand);
  if (old <= cand) return false;
  if (old == kUnreachable) ++reach;
  return true;
}

// Queue x unless it is queued already (inq bit; cleared when claimed).
__device__ __forceinline__ void lower_and_push(const Params& p, bool lowered, uint32_t x) {
  bool push = false;
  if (lowered) {
    const uint32_t bit = 1u << (x & 31);
    push = !(atomicOr(&p.inq[0][x >> 5], bit) & bit);
  }
  ring_push(p, push, x);
}

// Per-lane form of a queued push (any lane, no warp aggregation).
__device__ __forceinline__ void push_one(const Params& p, uint32_t x) {
  const uint32_t bit = 1u << (x & 31);
  if (atomicOr(&p.inq[0][x >> 5], bit) & bit) return;
  const uint32_t s = ph.rq_base + atomicAdd(ph.rq_tail, 1u);
  __stcg(&p.ring[s & p.ring_mask], (unsigned long long)x);
}

constexpr uint32_t kInlineRelax = 8;  // rows this short are relaxed where they are lowered

// Arcs [lo, hi) of u's row relaxed from label du, whole warp, four arcs per
// lane in flight; the vertices lowered are queued.
__device__ __forceinline__ void relax_arcs(const Params& p, uint64_t b, uint32_t nb, uint32_t dx, uint32_t lo, uint32_t hi,
                                           uint32_t du, long long& reach) {
  const DevAdj& a = p.g.out;
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t k0 = lo; k0 < hi; k0 += 128) {
    uint32_t x[4], d[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      const uint32_t k = k0 + 32 * j + lane;
      x[j] = k >= hi ? kTomb : k < nb ? a.col[b + k] : a.darena[dx + (k - nb)];
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) d[j] = !(x[j] & kTomb) && x[j] < ph.dist_len ? ld_cg(&p.dist[x[j]]) : 0u;
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
      if (d[j] > du + 1 && lower(p, x[j], du + 1, reach)) push_one(p, x[j]);
  }
}

constexpr uint32_t kInlineRows = 4;    // longer rows of one warp's seeds relaxed in place
constexpr uint32_t kInlineArcs = 512;  // their length

// A seed v just lowered: a short row is relaxed here by its lane (the
// vertices it lowers are queued), a few longer ones by the warp, others are
// queued (a batch whose seeds queue nothing ends without draining the ring).  Any later lowering
// of v queues v again, so relaxing from the current label loses nothing.
__device__ void seed_relax(const Params& p, bool lowered, uint32_t v, long long& reach) {
  const DevAdj& a = p.g.out;
  bool queue = false;
  uint64_t b = 0;
  uint32_t nb = 0, deg = 0;
  uint2 dr = make_uint2(0u, 0u);
  if (lowered) {
    uint64_t e;
    vxb::base_range(a, v, b, e);
    dr = a.drow[v];
    nb = (uint32_t)(e - b);
    deg = nb + dr.y;
    if (deg > kInlineRelax) {
      queue = true;
    } else {
      acct_add(p, 0, deg);
      // the row's columns, then their labels, are in flight together
      const uint32_t dv = ld_cg(&p.dist[v]);
      uint32_t x[kInlineRelax], dx[kInlineRelax];
#pragma unroll
      for (uint32_t k = 0; k < kInlineRelax; ++k)
        x[k] = k < nb ? a.col[b + k] : k < deg ? a.darena[dr.x + (k - nb)] : kTomb;
#pragma unroll
      for (uint32_t k = 0; k < kInlineRelax; ++k)
        dx[k] = !(x[k] & kTomb) && x[k] < ph.dist_len ? ld_cg(&p.dist[x[k]]) : 0u;
#pragma unroll
      for (uint32_t k = 0; k < kInlineRelax; ++k)
        if (dx[k] > dv + 1 && lower(p, x[k], dv + 1, reach)) push_one(p, x[k]);
    }
  }
  uint32_t rows = __ballot_sync(FULL, queue && deg <= kInlineArcs);
  if (rows && __popc(rows) <= kInlineRows) {
    if ((rows >> (threadIdx.x & 31)) & 1u) queue = false;
    while (rows) {
      const int l = __ffs(rows) - 1;
      rows &= rows - 1;
      const uint32_t n = __shfl_sync(FULL, deg, l);
      if ((threadIdx.x & 31) == 0) acct_add(p, 0, n);
      relax_arcs(p, __shfl_sync(FULL, b, l), __shfl_sync(FULL, nb, l), __shfl_sync(FULL, dr.x, l), 0u, n,
                 ld_cg(&p.dist[__shfl_sync(FULL, v, l)]), reach);
    }
  }
  lower_and_push(p, queue, v);
}

// Label-correcting relaxation (the settle of repair_affected, bfs.hpp:272-310,
// and propagate_decreases, :341-354, as one phase): every label is an upper
// bound of the post-batch distance, and relaxing from every changed label
// until nothing lowers gives the exact distances in any order.
struct Relax {
  const Params* p;
  LbStage* lb;
  long long* reach;
  // One item by one warp (the other chunks of a long row are queued by its first).
  __device__ void one(unsigned long long it) {
    const Params& P = *p;
    const DevAdj& a = P.g.out;
    const uint32_t lane = threadIdx.x & 31, u = item_vertex(it), c = item_chunk(it);
    if (c == 0) {
      if (lane == 0) atomicAnd(&P.inq[0][u >> 5], ~(1u << (u & 31)));
      __syncwarp();
      __threadfence();  // the queued bit is clear before the label is read
    }
    const uint32_t du = ld_cg(&P.dist[u]);
    uint64_t b, e;
    vxb::base_range(a, u, b, e);
    const uint2 dr = a.drow[u];
    const uint32_t nb = (uint32_t)(e - b), total = nb + dr.y;
    const uint32_t hi = min(total, (c + 1) * kChunk);
    if (c == 0)
      for (uint32_t k = 1 + lane; (k - lane) * kChunk < total; k += 32)
        ring_push(P, k * kChunk < total, (unsigned long long)u | ((unsigned long long)k << 32));
    if (du == kUnreachable) return;
    if (lane == 0) acct_add(P, 0, hi - c * kChunk);
    relax_arcs(P, b, nb, dr.x, c * kChunk, hi, du, *reach);
  }
  __device__ void process(RepairSmem& sm, uint32_t n) {
    const Params& P = *p;
    const uint32_t t = threadIdx.x;
    // past its deadline the relaxation drops the rest of its queue: the
    // batch's distances then come from a full BFS of the post-batch graph
    // (the same distances)
    if (t == 0 && sm.late && !sm.flagged) {
      atomicOr(&P.c->rbig, 1u);
      sm.flagged = 1;
    }
    if (t < n) {
      const unsigned long long it = sm.items[t];
      uint32_t du = kUnreachable;
      if (it != kSent) {
        const uint32_t u = item_vertex(it);
        if (item_chunk(it) == 0) atomicAnd(&P.inq[0][u >> 5], ~(1u << (u & 31)));
        if (sm.late) sm.items[t] = kSent;  // dropped
        else du = ld_cg(&P.dist[u]);
      }
      sm.d[t] = du;
    }
    __syncthreads();
    auto relax = [&](bool valid, uint32_t x, uint32_t j) {
      const uint32_t du = sm.d[j];
      const bool lowered = valid && du != kUnreachable && x < ph.dist_len && lower(P, x, du + 1, *reach);
      lower_and_push(P, lowered, x);
    };
    block_rows(P.g.out, sm.items, n, *lb, relax, &P, P.acct);
  }
};

// Boundary distances (best_boundary_distance, bfs.hpp:261-269) of the
// affected vertices, a block-sized chunk of them at a time: min of dist + 1
// over non-affected in-neighbours, folded per vertex in shared memory; each
// finite one seeds the relaxation.
constexpr uint32_t kBigBoundary = 4096;  // in-rows this long go to the grid-wide pass

__device__ void boundary_seeds(const Params& p, RepairSmem& sm, LbStage& lb, uint32_t na, long long& reach) {
  const uint32_t per = min((uint32_t)kThreads, max(1u, (na + gridDim.x - 1) / gridDim.x));
  for (uint32_t i0 = blockIdx.x * per; i0 < na; i0 += gridDim.x * per) {
    const uint32_t k = min(per, na - i0);
    if (threadIdx.x < k) {
      uint32_t v = p.lst_a[i0 + threadIdx.x];
      if (degree_of(p.g.in, v) > kBigBoundary) {  // a hub: the whole grid scans it after the barrier
        p.tent[i0 + threadIdx.x] = kUnreachable;
        p.big[atomicAdd(&p.c->big_b, 1u)] = i0 + threadIdx.x;
        v = 0xFFFFFFFFu;  // no row in this pass
      }
      sm.sv[threadIdx.x] = v;
      sm.cnt[threadIdx.x] = kUnreachable;
    }
    __syncthreads();
    auto bmin = [&](bool valid, uint32_t x, uint32_t j) {
      if (!valid || x >= ph.dist_len || test_bit(p.aff, x)) return;
      const uint32_t dx = p.dist[x];
      if (dx != kUnreachable) atomicMin(&sm.cnt[j], dx + 1);
    };
    block_rows(p.g.in, sm.sv, k, lb, bmin, nullptr, p.acct);
    bool seed = false;
    uint32_t v = 0;
    if (threadIdx.x < k && sm.sv[threadIdx.x] != 0xFFFFFFFFu) {
      v = sm.sv[threadIdx.x];
      const uint32_t best = sm.cnt[threadIdx.x];
      // by atomicMin: an inserted arc may lower v first
      if (best != kUnreachable) seed = lower(p, v, best, reach);
    }
    seed_relax(p, seed, v, reach);
    __syncthreads();
  }
}

// A few affected vertices (no more than the grid has warps): a warp each, no
// block barriers; the blocks' last warps take them first, so that the inserted
// arcs' seeds, which the first ones take, run beside them.
__device__ void boundary_seeds_few(const Params& p, uint32_t na, long long& reach) {
  const DevAdj& a = p.g.in;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t i = (blockDim.x / 32 - 1 - (threadIdx.x >> 5)) * gridDim.x + blockIdx.x;
  if (i >= na) return;
  const uint32_t v = p.lst_a[i];
  uint64_t b, e;
  vxb::base_range(a, v, b, e);
  const uint2 dr = a.drow[v];
  const uint32_t nb = (uint32_t)(e - b), total = nb + dr.y;
  if (total > kBigBoundary) {
    if (lane == 0) {
      p.tent[i] = kUnreachable;
      p.big[atomicAdd(&p.c->big_b, 1u)] = i;
    }
    return;
  }
  if (lane == 0) acct_add(p, 0, total);
  uint32_t best = kUnreachable;
  for (uint32_t k0 = 0; k0 < total; k0 += 128) {
    uint32_t x[4], dx[4], aw[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t k = k0 + 32 * j + lane;
      x[j] = k < nb ? a.col[b + k] : k < total ? a.darena[dr.x + (k - nb)] : kTomb;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool live = !(x[j] & kTomb) && x[j] < ph.dist_len;
      dx[j] = live ? p.dist[x[j]] : kUnreachable;
      aw[j] = live ? p.aff[x[j] >> 5] : FULL;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (dx[j] != kUnreachable && !((aw[j] >> (x[j] & 31)) & 1u)) best = min(best, dx[j] + 1);
  }
  best = __reduce_min_sync(FULL, best);
  bool seed = false;
  if (lane == 0 && best != kUnreachable) seed = lower(p, v, best, reach);
  seed_relax(p, seed, v, reach);
}

// Boundary distances of the hub entries p.big[0, nb) (indices into lst_a):
// each hub gets its own group of nwarps / nb warps (at least one), which fold
// 32-arc slices of its row into p.tent[i] by atomicMin, so many hubs are
// scanned side by side; the rows' seeds are taken after a barrier.
__device__ void grid_boundary_min(const Params& p, uint32_t nb) {
  const DevAdj& a = p.g.in;
  const int lane = threadIdx.x & 31;
  const uint32_t W = nwarps(), w = gwarp();
  const uint32_t G = max(1u, W / nb), R = W / G;  // warps per hub, hubs per round
  if (w >= R * G) return;
  for (uint32_t r = w / G; r < nb; r += R) {
    const uint32_t i = p.big[r];
    const uint32_t v = p.lst_a[i];
    uint32_t best = kUnreachable;
    uint64_t b, e;
    vxb::base_range(a, v, b, e);
    const uint2 dr = a.drow[v];
    const uint64_t nbase = e - b, total = nbase + dr.y;
    if (w % G == 0 && lane == 0) acct_add(p, 0, total);
    for (uint64_t k = (uint64_t)(w % G) * 32 + lane; k < total; k += (uint64_t)G * 32) {
      uint32_t x;
      if (k < nbase) {
        x = a.col[b + k];
        if (x & kTomb) continue;
      } else {
        x = a.darena[dr.x + (uint32_t)(k - nbase)];
      }
      if (x >= ph.dist_len || test_bit(p.aff, x)) continue;
      const uint32_t dx = p.dist[x];
      if (dx != kUnreachable && dx + 1 < best) best = dx + 1;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(FULL, best, o));
    if (lane == 0 && best != kUnreachable) atomicMin(&p.tent[i], best);
  }
}

// The post-batch repair proper (everything but the fallback); true when the
// batch's distances are to come from a full BFS of the post-batch graph
// instead (the relaxation passed its budget), with the workspace cleared.
// kInvalidated: the caller invalidated the affected vertices (invalidate) and
// sm.w holds the words of the barrier after that.
__device__ __forceinline__ void invalidate(const Params& p, uint32_t na) {
  for (uint32_t i = dealt_thread(); i < na; i += nthreads()) p.dist[p.lst_a[i]] = kUnreachable;
  if (gtid() == 0 && na) {
    reach_add(p, -(long long)na);
    p.c->big_b = 0;
  }
}

template <bool kInvalidated>
__device__ bool repair_relax(const Params& p, RepairSmem& sm, LbStage& lb) {
  BfsCounters* c = p.c;
  const int lane = threadIdx.x & 31;
  // the ring counters are zero here: the pre-batch kernel (or the previous
  // batch) left them so, and the first push comes after a barrier of this
  // kernel or a kernel boundary
  stamp(p, 3);
  if (gtid() == 0) set_deadline(p);
  // the lists' lengths as of the barrier before: gtid 0 resets them once the
  // repair is done, when another block may just be reading the last barrier's words
  const uint32_t na = kInvalidated ? sm.w.affected : ld_cg(&c->a_n);
  const uint32_t nt = kInvalidated ? sm.w.touched : ld_cg(&c->touched_n);
  if (gtid() == 0) acct_add(p, 1, na);  // invalidated and re-seeded
  long long reach = 0;
  if (na > 0) {
    if (!kInvalidated) {  // the affected vertices (repair_affected, bfs.hpp:272-283)
      invalidate(p, na);
      if (!sync_words(p, sm.w)) return false;
    }
    stamp(p, 4);
    if (na <= nwarps()) boundary_seeds_few(p, na, reach);
    else boundary_seeds(p, sm, lb, na, reach);
  }
  // inserted arcs relax their heads (bfs.hpp:91-96)
  const uint32_t F = *ph.F;
  for (uint32_t base = (dealt_thread() - lane * gridDim.x); base < F; base += nthreads()) {
    const uint32_t i = base + lane * gridDim.x;
    bool lowered = false;
    uint32_t v = 0;
    if (i < F && (ph.ff[i] & kFAdd)) {
      const uint32_t u = ph.fu[i];
      v = ph.fv[i];
      if (u < ph.dist_len && v < ph.dist_len) {
        const uint32_t du = ld_cg(&p.dist[u]);
        if (du != kUnreachable) lowered = lower(p, v, du + 1, reach);
      }
    }
    seed_relax(p, lowered, v, reach);
  }
  if (!sync_words(p, sm.w)) return false;
  const uint32_t nbig = na ? sm.w.big_b : 0u;
  if (nbig) {
    grid_boundary_min(p, nbig);
    if (!sync_words(p, sm.w)) return false;
    for (uint32_t base = gwarp() * 32; base < nbig; base += nwarps() * 32) {
      const uint32_t r = base + lane;
      bool seed = false;
      uint32_t v = 0;
      if (r < nbig) {
        const uint32_t i = p.big[r];
        v = p.lst_a[i];
        const uint32_t best = ld_cg(&p.tent[i]);
        p.tent[i] = 0u;  // tent is all-zero between phases (the cascade's chunk counts)
        if (best != kUnreachable) seed = lower(p, v, best, reach);
      }
      seed_relax(p, seed, v, reach);
    }
    if (!sync_words(p, sm.w)) return false;
  }
  stamp(p, 5);
  if (sm.w.tail) {  // the relaxation runs only when a seed left work queued
    Relax w{&p, &lb, &reach};
    if (!sync_rounds(p, sm, w)) {
      if (sm.w.failed) return false;
      drain(p, sm, w, sm.w.deadline);
      if (!sync_words(p, sm.w)) return false;
    }
    if (sm.w.rbig) {
      // the relaxation passed its budget: a full BFS of the post-batch graph
      // gives the distances and the reachable count (the repair's counters
      // -- candidates, affected, no full recompute -- stand)
      clear_workspace(p, nt, na);
      reset_ring(p);
      return true;
    }
  }
  stamp(p, 6);
  if (gtid() == 0) {
    c->rtrace[8] = ph.rq_base + sm.w.tail;
    for (int k = 0; k < 6; ++k) c->rtrace[15 + k] = __ldcg(&p.rq_stat[k]);
  }
  reach = vxb::warp_sum(reach);
  if (lane == 0) reach_add(p, reach);
  clear_workspace(p, nt, na);
  reset_ring(p);
  return false;
}

// Post-batch repair (bfs.hpp:72-97): the fallback's full BFS or the repair,
// which may itself hand over to a full BFS; one call site serves both.
template <bool kInvalidated>
__device__ void repair_post(const Params& p, RepairSmem& sm, LbStage& lb, BlockQueue& bq) {
  BfsCounters* c = p.c;
  const bool fallback = kInvalidated ? sm.w.fallback != 0u : ld_cg(&c->fallback) != 0u;
  if (fallback) {
    if (kInvalidated) clear_workspace(p, sm.w.touched, sm.w.affected);
    else clear_workspace(p, ld_cg(&c->touched_n), ld_cg(&c->a_n));
  } else if (!repair_relax<kInvalidated>(p, sm, lb)) {
    return;
  }
  if (!sync_grid(p)) return;
  bfs_in_repair(p, sm, lb, bq, p.dist, p.trace);
  if (gtid() == 0) {
    if (fallback) {
      c->full = 1;
    } else {
      c->rbig = 0u;
      c->handovers[1] += 1;
    }
  }
}

// ------------------------------------------------------- batched stream --
//
// A whole update stream applied in one persistent launch: the batches' canonical
// arcs come sorted by (batch, u, v) from one stream-wide sort, and every batch
// runs classify + tombstones, delta removals + deletion candidates, the
// cascade, tombstone revivals + delta insertions, and the post-batch repair,
// separated by grid barriers, with no launch or host synchronisation between
// batches.  The result after every batch is the one IncrementalBFS::apply
// gives (bfs.hpp:29-98); an optional per-batch digest of the distances and
// per-batch counters make every batch checkable.

struct StreamArgs {
  // canonical arcs of the stream, batch-major: [0] of the out-adjacency, sorted
  // by (u, v); [1] of a directed graph's in-adjacency, the same arcs as (v, u)
  const uint32_t* fu[2];
  const uint32_t* fv[2];
  uint8_t* ff[2];            // in: desired state (bit 0); out: classification flags
  uint64_t* fpos[2];
  const uint32_t* cnt[2];    // arc counts: nb of them for [0], one for [1]
  uint32_t* scratch[2];      // one batch's arcs: the insertions of each row run
  const uint32_t* boff;      // nb + 1 offsets of the batches' arcs (null: one batch)
  const uint32_t* vpost;     // vertex count after each batch
  unsigned long long* digest;  // nb digests of the distances (optional)
  uint32_t* bstats;          // nb x 4: candidates, affected, full recompute, reachable (optional)
  GraphCounters* gc;
  unsigned long long arena_cap[2];
  double frac;
  uint32_t nb, V0, len0;
  uint32_t v_single;    // vertex count after the batch when vpost is null (one staged batch)
  uint32_t classified;  // the arcs carry their classification already (a staged batch)
  // raw_n > 0: one batch whose op arrays the launch canonicalises itself (the
  // arc lists above are written by it); ids take b bits, below bound, and
  // raw_sh bits hold an op's index and its add flag
  const uint32_t* raw_src;
  const uint32_t* raw_dst;
  const uint8_t* raw_add;
  uint32_t* over;  // canon_grid: per block, rows left to the grid, then two counts
  uint32_t raw_n, raw_b, raw_sh, raw_bound;
};

// A batch of at most kRawOps ops is canonicalised inside the launch: every block
// reads all ops and keeps the arcs whose row hashes to it (a dozen of 2,000), sorts
// them, keeps the last of each arc and appends them to the batch's list, so
// the arcs of a row are consecutive there and the block that has them in
// shared memory can process them at once.  Rows of more arcs than a block sorts are
// listed by the whole grid (canon_grid).  A launch of its own with a cluster's
// barriers between the radix passes took 12 to 44 us; every block sorting
// all arcs 2 us for 128 arcs but 7 for 1,024 and 13 for 2,048, bound by the
// instructions of the one block an SM runs; now 2 to 8 (10,000 ops).  The limit keeps a
// block's reading (9 bytes an op from L2) at a few microseconds.
constexpr uint32_t kRawOps = 16384;
constexpr uint32_t kRawKeys = 2048;  // arcs a block sorts at once (canon_grid beyond)
constexpr uint32_t kRawBlocks = 512;  // blocks of a launch at most
constexpr unsigned long long kRawDir = 1ull << 63;  // a directed graph's reversed arcs sort last
// A block with more arcs than this (hub rows) leaves them to the whole grid,
// behind a barrier; with more than kRawWarps it gives each a lane, not a warp.
constexpr uint32_t kRawMine = 1024;
constexpr uint32_t kRawWarps = 32;
constexpr uint8_t kFPending = 0x80;  // flag of an arc left to the grid
constexpr uint32_t kNoRoom = 0xFFFFFFFFu;
struct RawArcs {
  unsigned long long key[kRawKeys];  // [dir] | u | v | op index | add
  uint32_t wsum[kThreads / 32];
  uint32_t n[2];                     // arcs, and those of direction 0 among them
  uint32_t base[2];                  // their places in the batch's lists
  uint32_t over[kRawBlocks / 32];    // canon_grid: blocks whose rows are left to the grid
  uint32_t sum[4];
};
static_assert(sizeof(RawArcs) <= sizeof(LbStage), "the arcs are kept in the row stage's memory");

// Bitonic sort of a warp's 32 * E keys, key e * 32 + lane in x[e].  The loops
// over the steps stay rolled: the code runs once per launch, and unrolled it
// is bound by fetching its instructions.
template <int E>
__device__ __forceinline__ void warp_sort(unsigned long long (&x)[E]) {
  const uint32_t lane = threadIdx.x & 31;
  auto exchange = [&](uint32_t e, uint32_t o, uint32_t k) {
    if ((x[e] > x[o]) == (((e * 32 + lane) & k) == 0)) {
      const unsigned long long t = x[e];
      x[e] = x[o];
      x[o] = t;
    }
  };
#pragma unroll 1
  for (uint32_t k = 2; k <= 32 * E; k <<= 1) {
    if (E == 4 && k == 128) {
      exchange(0, 2 % E, k);
      exchange(1 % E, 3 % E, k);
    }
    if (E >= 2 && k >= 64) {
      exchange(0, 1 % E, k);
      if (E == 4) exchange(2 % E, 3 % E, k);
    }
#pragma unroll 1
    for (uint32_t j = min(k >> 1, 16u); j > 0; j >>= 1) {
      const bool low = (lane & j) == 0;
#pragma unroll
      for (uint32_t e = 0; e < E; ++e) {
        const bool up = ((e * 32 + lane) & k) == 0;
        const unsigned long long y = __shfl_xor_sync(FULL, x[e], j);
        x[e] = (x[e] < y) == (low == up) ? x[e] : y;
      }
    }
  }
}

// Sorts the block's n arc keys, padded to N (a power of two, 32 * E per warp in
// use), and, unless all are wanted, keeps the last of each arc.  Every warp sorts
// its keys in registers; the runs are then merged pairwise, each key finding its
// place by a binary search of the other run.
template <int E>
__device__ void canon_sort(const StreamArgs& s, bool directed, RawArcs& r, uint32_t n, uint32_t N, bool all) {
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool on = warp * 32 * E < N;
  unsigned long long x[E];
  uint32_t g[E];  // the keys' places
#pragma unroll
  for (uint32_t e = 0; e < E; ++e) {
    g[e] = warp * 32 * E + e * 32 + lane;
    x[e] = g[e] < n ? r.key[g[e]] : ~0ull;
  }
  __syncthreads();  // every key is read
  if (on) {
    warp_sort<E>(x);
#pragma unroll
    for (uint32_t e = 0; e < E; ++e) r.key[g[e]] = x[e];
  }
  if (t < 2) r.n[t] = 0;
  __syncthreads();
#pragma unroll 1
  for (uint32_t L = 32 * E; L < N; L <<= 1) {
    uint32_t to[E];
    if (on) {
      uint32_t lo[E];
      const unsigned long long* other[E];
      bool right[E];
#pragma unroll
      for (uint32_t e = 0; e < E; ++e) {
        lo[e] = 0;
        right[e] = (g[e] & L) != 0;
        other[e] = r.key + ((g[e] & ~(L - 1)) ^ L);
      }
      // padding keys are equal: those of the left run stay first
#pragma unroll 1
      for (uint32_t step = L >> 1; step > 0; step >>= 1) {
#pragma unroll
        for (uint32_t e = 0; e < E; ++e) {
          const unsigned long long y = other[e][lo[e] + step - 1];
          if (y < x[e] || (right[e] && y == x[e])) lo[e] += step;
        }
      }
#pragma unroll
      for (uint32_t e = 0; e < E; ++e) {
        const unsigned long long y = other[e][lo[e]];
        if (y < x[e] || (right[e] && y == x[e])) ++lo[e];
        to[e] = (g[e] & ~(2 * L - 1)) + (g[e] & (L - 1)) + lo[e];
      }
    }
    __syncthreads();
    if (on) {
#pragma unroll
      for (uint32_t e = 0; e < E; ++e) {
        g[e] = to[e];
        r.key[g[e]] = x[e];
      }
    }
    __syncthreads();
  }
  if (all) return;
  // the last key of every arc, compacted in place
  unsigned long long keep[E];
  uint32_t cnt = 0, cnt0 = 0;
#pragma unroll
  for (uint32_t h = 0; h < E; ++h) {
    const uint32_t j = t * E + h;
    keep[h] = ~0ull;
    if (j < N) {
      const unsigned long long k = r.key[j], y = j + 1 < N ? r.key[j + 1] : ~0ull;
      if (k != ~0ull && (k >> s.raw_sh) != (y >> s.raw_sh)) {
        keep[h] = k;
        ++cnt;
        cnt0 += !(directed && (k & kRawDir));
      }
    }
  }
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, incl, o);
    if ((int)lane >= o) incl += y;
  }
  cnt0 = __reduce_add_sync(FULL, cnt0);
  if (lane == 31) r.wsum[warp] = incl;
  if (lane == 0 && cnt0) atomicAdd(&r.n[1], cnt0);
  __syncthreads();  // every key is read, too
  uint32_t pos = incl - cnt;
  for (uint32_t k = 0; k < warp; ++k) pos += r.wsum[k];
#pragma unroll
  for (uint32_t h = 0; h < E; ++h)
    if (keep[h] != ~0ull) r.key[pos++] = keep[h];
  if (t == kThreads - 1) r.n[0] = pos;
  __syncthreads();
}

// The keys of op i's arcs whose row hashes to a block that mine(block) takes,
// f(key) each.  first: reports ids out of bound.
template <class Mine, class F>
__device__ __forceinline__ void raw_op(const StreamArgs& s, bool directed, uint32_t i, bool first, Mine&& mine, F&& f) {
  const uint32_t a = s.raw_src[i], b = s.raw_dst[i];
  const unsigned long long low = ((unsigned long long)i << 1) | (s.raw_add[i] ? 1ull : 0ull);
  bool ok = a != b;
  if (ok && (a >= s.raw_bound || b >= s.raw_bound)) {
    if (first && blockIdx.x == 0) atomicOr(&s.gc->err, vxb::kErrBadVertex);
    ok = false;
  }
  if (!ok) return;
#pragma unroll
  for (int rev = 0; rev < 2; ++rev) {
    const unsigned long long u = rev ? b : a, v = rev ? a : b;
    if (!mine(__umulhi((uint32_t)u * 0x9E3779B1u, gridDim.x))) continue;
    f((directed && rev ? kRawDir : 0ull) | (u << (s.raw_b + s.raw_sh)) | (v << s.raw_sh) | low);
  }
}

__device__ void canon_keys(const StreamArgs& s, bool directed, RawArcs& r, uint32_t n, bool all = false) {
  uint32_t N = 32;
  while (N < n) N <<= 1;
  static_assert(kRawKeys == 4 * kThreads, "four keys per thread at most");
  if (N <= kThreads) canon_sort<1>(s, directed, r, n, N, all);
  else if (N <= 2 * kThreads) canon_sort<2>(s, directed, r, n, N, all);
  else canon_sort<4>(s, directed, r, n, N, all);
}

// The block's arcs of the batch in r, and their places in the batch's lists
// (whose lengths are f[0] and f[1], zero before); true, and no arcs, when the block
// has too many: canon_grid lists them.  Block-uniform.
__device__ bool canon_raw(const StreamArgs& s, bool directed, RawArcs& r, uint32_t* f) {
  if (threadIdx.x < 2) r.n[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < s.raw_n; i += kThreads)
    raw_op(s, directed, i, true, [&](uint32_t b) { return b == blockIdx.x; }, [&](unsigned long long key) {
      if (*(volatile uint32_t*)&r.n[0] > kRawKeys) return;
      const uint32_t k = atomicAdd(&r.n[0], 1u);
      if (k < kRawKeys) r.key[k] = key;
    });
  __syncthreads();
  const uint32_t n = r.n[0];
  __syncthreads();
  const bool fits = n <= kRawKeys;
  if (threadIdx.x == 0) {
    r.n[0] = 0;
    s.over[blockIdx.x] = fits ? 0u : 1u;
  }
  __syncthreads();
  if (fits) canon_keys(s, directed, r, n);
  if (threadIdx.x < 2) {
    const uint32_t k = threadIdx.x ? r.n[0] - r.n[1] : r.n[1], room = directed ? s.raw_n : 2 * s.raw_n;
    const uint32_t at = k ? atomicAdd(&f[threadIdx.x], k) : 0u;
    r.base[threadIdx.x] = at <= room && k <= room - at ? at : kNoRoom;
  }
  __syncthreads();
  // A launch that ended on a device error left its lengths behind: the batches
  // after it, whose launches end at their first barrier, must not run past the lists.
  if (r.base[0] == kNoRoom || r.base[1] == kNoRoom) {
    __syncthreads();
    if (threadIdx.x < 2) r.n[threadIdx.x] = 0;
    __syncthreads();
  }
  return !fits;
}

// Ascending ranges of [lo, hi) of the arcs' (dir, u, v) value whose arcs fit r,
// halved and doubled as they come: emit() for each, its arcs in r (the last op of
// each, r.n as canon_keys leaves it).  One range, the whole of it, where
// canon_grid's samples do not deceive.  Returns their number.  Block-uniform.
template <class Mine, class Emit>
__device__ uint32_t raw_ranges(const StreamArgs& s, bool directed, RawArcs& r, unsigned long long lo,
                               unsigned long long end, Mine&& mine, Emit&& emit) {
  const uint32_t bits = 2 * s.raw_b;
  auto value = [&](unsigned long long key) {
    return ((key & ~kRawDir) >> s.raw_sh) | (key & kRawDir ? 1ull << bits : 0ull);
  };
  unsigned long long width = end - lo;
  uint32_t ranges = 0;
  while (lo < end) {
    const unsigned long long hi = end - lo < width ? end : lo + width;
    __syncthreads();  // the range before is done with
    if (threadIdx.x < 2) r.n[threadIdx.x] = 0;
    if (threadIdx.x == 0) r.key[0] = 0;
    __syncthreads();
    uint32_t n;
    if (hi - lo == 1) {  // one arc, of any number of ops: its last
      unsigned long long last = 0;
      for (uint32_t i = threadIdx.x; i < s.raw_n; i += kThreads)
        raw_op(s, directed, i, false, mine, [&](unsigned long long key) {
          if (value(key) == lo && key > last) last = key;
        });
      if (last) atomicMax(&r.key[0], last);  // ids of an arc differ, so no key is 0
      __syncthreads();
      n = r.key[0] ? 1u : 0u;
    } else {
      for (uint32_t i = threadIdx.x; i < s.raw_n; i += kThreads)
        raw_op(s, directed, i, false, mine, [&](unsigned long long key) {
          const unsigned long long x = value(key);
          if (x < lo || x >= hi || *(volatile uint32_t*)&r.n[0] > kRawKeys) return;
          const uint32_t k = atomicAdd(&r.n[0], 1u);
          if (k < kRawKeys) r.key[k] = key;
        });
      __syncthreads();
      n = r.n[0];
    }
    __syncthreads();
    if (n > kRawKeys) {
      width = (hi - lo + 1) / 2;
      continue;
    }
    if (threadIdx.x < 2) r.n[threadIdx.x] = 0;
    __syncthreads();
    canon_keys(s, directed, r, n);
    emit();
    ++ranges;
    if (n < kRawKeys / 2 && width <= (end - lo) / 2) width *= 2;
    lo = hi;
  }
  return ranges;
}

// The arcs of rows whose block has too many of them, listed by the whole grid in
// the order of their (dir, u, v) value: all blocks sort the same sample of the
// ops, take the range between two of its entries each, sort their range's arcs,
// and write them behind those of the blocks before (marked kFPending: a row's arcs
// lie with several blocks).  An arc that fills a block's share of the sample or
// more is a range by itself.  The hub's block alone, range after range of 2,048
// arcs, took the launch 1.5 ms longer than a cluster's sort of the batch does
// (16,384 ops on one row at R-MAT 20: 2.88 ms a call against 1.38).  words: as of
// the last barrier; false on a device error.  Grid-uniform.
constexpr uint32_t kRawSamples = 512;  // ops
__device__ __noinline__ bool canon_grid(const Params& p, const StreamArgs& s, RawArcs& r,
                                        const RepairWords& words) {
  const bool directed = p.g.directed;
  const uint32_t t = threadIdx.x, G = gridDim.x, b = blockIdx.x;
  if (t < 2) r.n[t] = 0;
  if (t < 4) r.sum[t] = 0;
  for (uint32_t i = t; i < kRawBlocks / 32; i += kThreads) r.over[i] = 0;
  __syncthreads();
  for (uint32_t i = t; i < G; i += kThreads)
    if (ld_cg(&s.over[i])) atomicOr(&r.over[i >> 5], 1u << (i & 31));
  __syncthreads();
  auto left = [&](uint32_t block) { return (r.over[block >> 5] >> (block & 31)) & 1u; };
  const uint32_t S = min(s.raw_n, kRawSamples);
  for (uint32_t i = t; i < S; i += kThreads) {
    const uint32_t lo = (uint32_t)((uint64_t)i * s.raw_n / S), hi = (uint32_t)((uint64_t)(i + 1) * s.raw_n / S);
    raw_op(s, directed, lo + (uint32_t)(vxb::mix64(i) % (hi - lo)), false, left,
           [&](unsigned long long key) { r.key[atomicAdd(&r.n[0], 1u)] = key; });
  }
  __syncthreads();
  const uint32_t ns = r.n[0];
  __syncthreads();
  static_assert(2 * kRawSamples <= kRawKeys, "the samples' arcs are sorted at once");
  canon_keys(s, directed, r, ns, true);
  const uint32_t bits = 2 * s.raw_b;
  auto split = [&](uint32_t k) {  // first value of block k's range
    if (k == 0 || ns == 0) return k < G ? 0ull : (directed ? 2ull : 1ull) << bits;
    if (k >= G) return (directed ? 2ull : 1ull) << bits;
    const unsigned long long key = r.key[(uint64_t)k * ns / G];
    return ((key & ~kRawDir) >> s.raw_sh) | (key & kRawDir ? 1ull << bits : 0ull);
  };
  unsigned long long lo = split(b), hi = split(b + 1);
  const bool again = b > 0 && split(b - 1) == lo;  // the block before begins at the same arc
  if (lo == hi) hi = again ? lo : lo + 1;          // the first of them takes that arc,
  else if (again) ++lo;                            // the last what lies behind it
  uint32_t kept[2] = {0, 0};
  const uint32_t ranges = raw_ranges(s, directed, r, lo, hi, left, [&] {
    kept[0] += r.n[1];
    kept[1] += r.n[0] - r.n[1];
  });
  if (t == 0) {
    s.over[G + b] = kept[0];
    s.over[2 * G + b] = kept[1];
  }
  if (!sync_grid(p)) return false;
  for (uint32_t i0 = t & ~31u; i0 < G; i0 += kThreads) {
    const uint32_t i = i0 + (t & 31);
    for (uint32_t d = 0; d < 2; ++d) {
      const uint32_t c = i < G ? ld_cg(&s.over[(d + 1) * G + i]) : 0u;
      const uint32_t before = __reduce_add_sync(FULL, i < b ? c : 0u), sum = __reduce_add_sync(FULL, c);
      if ((t & 31) == 0) {
        atomicAdd(&r.sum[d], before);
        atomicAdd(&r.sum[2 + d], sum);
      }
    }
  }
  __syncthreads();
  uint32_t place[2] = {words.raw_f[0] + r.sum[0], words.raw_f[1] + r.sum[1]};
  if (gtid() == 0) {  // the lists' new lengths, read behind the next barrier
    p.bar[kRawWord] = words.raw_f[0] + r.sum[2];
    p.bar[kRawWord + 1] = words.raw_f[1] + r.sum[3];
  }
  auto write = [&] {
    const uint32_t n = r.n[0], n0 = r.n[1];
    for (uint32_t i = t; i < n; i += kThreads) {
      const int dir = i >= n0;
      const uint32_t at = place[dir] + i - (dir ? n0 : 0u);
      const unsigned long long k = r.key[i];
      const_cast<uint32_t*>(s.fu[dir])[at] = (uint32_t)((k & ~kRawDir) >> (s.raw_b + s.raw_sh));
      const_cast<uint32_t*>(s.fv[dir])[at] = (uint32_t)(k >> s.raw_sh) & ((1u << s.raw_b) - 1u);
      s.ff[dir][at] = (uint8_t)(k & 1ull) | kFPending;
    }
    place[0] += n0;
    place[1] += n - n0;
  };
  if (ranges == 1) write();
  else if (ranges) raw_ranges(s, directed, r, lo, hi, left, write);
  __syncthreads();  // r is used by others
  return true;
}

// Order-independent 64-bit digest of dist[0, n): sum of splitmix64(v << 32 | dist[v]).
using vxb::mix64;

__device__ void digest_pass(const uint32_t* dist, uint32_t n, unsigned long long* out) {
  unsigned long long h = 0;
  for (uint32_t v = gtid(); v < n; v += nthreads()) h += mix64(((unsigned long long)v << 32) | ld_cg(&dist[v]));
  h = vxb::warp_sum(h);
  if ((threadIdx.x & 31) == 0 && h) atomicAdd(out, h);
}

// End of the row run of canonical arcs starting at s (same u), whole warp: 32
// probes a step, 1, 32, 1,024 ... arcs apart while all of them are the row's, then
// closer again (a row's arcs are consecutive).
__device__ __forceinline__ uint32_t run_end(const uint32_t* fu, uint32_t s, uint32_t F) {
  const uint32_t lane = threadIdx.x & 31, u = fu[s];
  uint64_t last = s, stride = 1;  // last: an arc of the row
  for (;;) {
    const uint64_t i = last + (lane + 1) * stride;
    const uint32_t m = __ballot_sync(FULL, i >= F || fu[i] != u);
    last += (m ? (uint32_t)(__ffs(m) - 1) : 32u) * stride;
    if (!m) stride *= 32;
    else if (stride == 1) return (uint32_t)last + 1;
    else stride /= 32;
  }
}

__device__ __forceinline__ bool delta_op(uint8_t f, bool insertion) {
  return !(f & kFInBase) && (f & kFChanged) && (((f & kFAdd) != 0) == insertion);
}

// Delta removals of one row run (whole warp): the row's sorted delta list
// keeps every entry that is not a removal of the run (delta_remove_kernel of
// the per-batch path, on the canonical arcs directly).  128 entries a step, their
// searches in the run side by side: a hub's run is one warp's chain.  9,000 ops on
// one row at R-MAT 20, 6,300 removals: with run_end's probes the pass takes 232 us
// instead of 337, and the insertions back 92 instead of 176.
__device__ void run_remove(const vxb::DevAdj& a, int dir, const uint32_t* fv, const uint8_t* ff, uint32_t s, uint32_t e,
                           uint32_t u, GraphCounters* gc, unsigned long long* acct) {
  constexpr int kStep = 4;
  const int lane = threadIdx.x & 31;
  bool any = false;
  for (uint32_t k = s + lane; k < e; k += 32) any |= delta_op(ff[k], false);
  if (!__any_sync(FULL, any)) return;
  const uint2 row = a.drow[u];
  uint32_t* A = a.darena + row.x;
  uint32_t written = 0;
  for (uint32_t base = 0; base < row.y; base += 32 * kStep) {
    uint32_t x[kStep], lo[kStep];
#pragma unroll
    for (int r = 0; r < kStep; ++r) {
      const uint32_t j = base + 32 * r + lane;
      x[r] = j < row.y ? A[j] : 0u;
      lo[r] = s;
    }
    for (uint32_t len = e - s; len > 1;) {  // x's place in the run is lo or, at the end, lo + 1
      const uint32_t half = len >> 1;
#pragma unroll
      for (int r = 0; r < kStep; ++r)
        if (fv[lo[r] + half - 1] < x[r]) lo[r] += half;
      len -= half;
    }
    __syncwarp();  // every entry of the step is read
#pragma unroll
    for (int r = 0; r < kStep; ++r) {
      if (base + 32 * r >= row.y) break;
      const uint32_t q = lo[r] + (fv[lo[r]] < x[r] ? 1u : 0u);
      const bool keep = base + 32 * r + lane < row.y && !(q < e && fv[q] == x[r] && delta_op(ff[q], false));
      const uint32_t mask = __ballot_sync(FULL, keep);
      if (keep) A[written + __popc(mask & vxb::lanemask_lt())] = x[r];
      written += __popc(mask);
    }
    __syncwarp();
  }
  if (lane == 0) {
    a.drow[u].y = written;
    if (acct) atomicAdd(acct, (unsigned long long)(row.y + written));
    atomicAdd(&gc->delta_live[dir], (unsigned long long)(-(long long)(row.y - written)));
    gdev::mark_dirty(a.dirty, u, &gc->dirty_rows[dir]);
  }
}

// Delta insertions of one row run (whole warp): the run's insertions are
// compacted into scratch[s, s + nB) and merged into the row's delta list, in
// place when its block has room, else into a new power-of-two arena block
// (delta_insert_kernel of the per-batch path).
__device__ void run_insert(const vxb::DevAdj& a, int dir, const uint32_t* fv, const uint8_t* ff, uint32_t* scratch,
                           uint32_t s, uint32_t e, uint32_t u, GraphCounters* gc, unsigned long long arena_cap,
                           unsigned long long* acct) {
  const int lane = threadIdx.x & 31;
  uint32_t nB = 0;
  for (uint32_t base = s; base < e; base += 128) {  // 128 arcs in flight
    uint32_t v[4];
    bool ins[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t k = base + 32 * r + lane;
      ins[r] = k < e && delta_op(ff[k], true);
      v[r] = k < e ? fv[k] : 0u;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t m = __ballot_sync(FULL, ins[r]);
      if (ins[r]) scratch[s + nB + __popc(m & vxb::lanemask_lt())] = v[r];
      nB += __popc(m);
    }
  }
  if (nB == 0) return;
  __syncwarp();
  const uint2 row = a.drow[u];
  const uint32_t cap = a.dcap[u];
  const uint32_t cnew = row.y + nB;
  if (cnew <= cap) {
    gdev::warp_merge_inplace(a.darena + row.x, row.y, scratch + s, nB);
    if (lane == 0) a.drow[u].y = cnew;
  } else {
    uint32_t ncap = 8;
    while (ncap < cnew) ncap <<= 1;
    unsigned long long off = 0;
    if (lane == 0) off = atomicAdd(&gc->arena_top[dir], (unsigned long long)ncap);
    off = __shfl_sync(FULL, off, 0);
    if (off + ncap > arena_cap) {
      if (lane == 0) atomicOr(&gc->err, vxb::kErrArenaOverflow);
      return;
    }
    gdev::warp_merge_to(a.darena + off, a.darena + row.x, row.y, scratch + s, nB);
    if (lane == 0) {
      a.drow[u] = make_uint2((uint32_t)off, cnew);
      a.dcap[u] = ncap;
    }
  }
  if (lane == 0) {
    atomicAdd(&gc->delta_live[dir], (unsigned long long)nB);
    if (acct) atomicAdd(acct, (unsigned long long)(row.y + cnew));
    gdev::mark_dirty(a.dirty, u, &gc->dirty_rows[dir]);
  }
}

// ---- the commit's two passes over the canonical arcs ----
//
// Removals first (before the cascade reads the rows), insertions after it.
// Arcs of one row are consecutive (a run) and only they touch that row, so
// whoever takes an arc that is a run by itself -- most of a batch -- classifies
// it, tombstones it or edits its delta row and registers it as a deletion
// candidate in one go.  Delta removals of longer runs need the whole run's
// classification: they are left to a second pass behind a grid barrier, which
// a batch without any skips.  On a delta row of at most 7 arcs (8 for a removal)
// one lane does a single arc: the row's block (capacity >= 8, 8-aligned in the
// arena) is loaded as two 16-byte words, edited in registers and stored back; a
// row without a block gets 8 slots from one warp-aggregated arena allocation.
// The rest is queued in shared memory and done by the block's warps (run_insert,
// run_remove).  Arcs are dealt round-robin (arc i to block i mod gridDim), so a
// small batch still spreads over every block.

// Position of x in the sorted a[lo, hi), compared by the low 31 bits, or hi
// where it is missing; whole warp: 32 pivots per round trip.
__device__ __forceinline__ uint64_t warp_find(const uint32_t* a, uint64_t lo, uint64_t hi, uint32_t x) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t end = hi;
  while (hi - lo > 32) {
    const uint64_t step = (hi - lo + 31) / 32;
    const uint64_t k = lo + step * (lane + 1) - 1;  // last entry of this lane's part
    const bool below = k < hi && (a[k] & kIdMask) < x;
    const uint32_t n = __popc(__ballot_sync(FULL, below));  // parts before the one that may hold x
    lo += step * n;
    if (lo >= hi) return end;
    hi = hi < lo + step ? hi : lo + step;
  }
  const bool hit = lo + lane < hi && (a[lo + lane] & kIdMask) == x;
  const uint32_t m = __ballot_sync(FULL, hit);
  return m ? lo + (uint32_t)(__ffs(m) - 1) : end;
}

struct ArcWork {
  const Params* p;
  const StreamArgs* s;
  const vxb::DevAdj* a;
  int dir;
  const uint32_t* fu;  // the batch's arcs
  const uint32_t* fv;
  uint8_t* ff;
  uint64_t* fpos;
  uint32_t F;
  // the arcs this block canonicalised, F of them, whose list place is base on
  // (null: the whole batch's, in fu, fv, ff)
  const unsigned long long* raw;
  uint32_t base;
  bool pending;        // only the arcs marked kFPending
  long long tombs;     // this lane's change of the tombstone count, and rows it dirtied
  uint32_t dirtied;

  // A deletion candidate (bfs.hpp:52-63) is the head of a deleted
  // shortest-parent arc; its first touch records it at the front of the touched
  // list.  Warp-uniform.
  __device__ __forceinline__ void candidate(bool arc, uint32_t u, uint32_t v, uint8_t f) {
    if (dir) return;
    bool first = false;
    if (arc && !(f & kFAdd) && (f & kFCur) && is_sp(*p, u, v))
      first = !(atomicOr(&p->sw[v], kSwTouched) & kSwTouched);
    const uint32_t slot = vxb::warp_append(first, &p->c->cand_n);
    if (first) p->lst_t[slot] = v;
  }

  __device__ __forceinline__ uint32_t tail_of(uint32_t i) const {
    return raw ? (uint32_t)((raw[i] & ~kRawDir) >> (s->raw_b + s->raw_sh)) : fu[i];
  }
  // Arc i; a block's own are also written to the list the later passes read.
  __device__ __forceinline__ void arc(uint32_t i, uint32_t& u, uint32_t& v, uint8_t& f) const {
    if (raw) {
      const unsigned long long k = raw[i];
      u = tail_of(i);
      v = (uint32_t)(k >> s->raw_sh) & ((1u << s->raw_b) - 1u);
      f = (uint8_t)(k & 1ull);
      const_cast<uint32_t*>(fu)[base + i] = u;
      const_cast<uint32_t*>(fv)[base + i] = v;
    } else {
      u = fu[i];
      v = fv[i];
      f = ff[i];
    }
  }
  // Whether arc i's row has other arcs in the batch.
  __device__ __forceinline__ bool in_run(uint32_t i, uint32_t u) const {
    return (i > 0 && tail_of(i - 1) == u) || (i + 1 < F && tail_of(i + 1) == u);
  }

  // Arc (u, v) leaves u's delta row; whole warp.
  __device__ void remove_one(uint32_t u, uint32_t v) {
    const uint32_t lane = threadIdx.x & 31;
    const uint2 row = a->drow[u];
    uint32_t* A = a->darena + row.x;
    uint32_t written = 0;
    for (uint32_t base = 0; base < row.y; base += 32) {
      const uint32_t x = base + lane < row.y ? A[base + lane] : v;
      const uint32_t mask = __ballot_sync(FULL, x != v);
      if (x != v) A[written + __popc(mask & vxb::lanemask_lt())] = x;
      written += __popc(mask);
      __syncwarp();
    }
    if (lane == 0) {
      a->drow[u].y = written;
      acct_add(*p, 2, (unsigned long long)row.y + written);
      atomicAdd(&s->gc->delta_live[dir], (unsigned long long)(-(long long)(row.y - written)));
      gdev::mark_dirty(a->dirty, u, &s->gc->dirty_rows[dir]);
    }
  }

  // The sums of the pass into the graph's counters.
  __device__ __forceinline__ void flush() {
    tombs = vxb::warp_sum(tombs);
    dirtied = vxb::warp_sum(dirtied);
    if ((threadIdx.x & 31) == 0 && tombs) atomicAdd(&s->gc->tombs[dir], (unsigned long long)tombs);
    if ((threadIdx.x & 31) == 0 && dirtied) atomicAdd(&s->gc->dirty_rows[dir], (unsigned long long)dirtied);
    tombs = 0;
    dirtied = 0;
  }
};

// A delta row of at most 8 arcs in registers: its block's 8 slots.
struct SmallRow {
  uint32_t x[8];
  __device__ __forceinline__ void load(const uint32_t* block) {
    const uint4* q = reinterpret_cast<const uint4*>(block);
    const uint4 q0 = q[0], q1 = q[1];
    x[0] = q0.x, x[1] = q0.y, x[2] = q0.z, x[3] = q0.w;
    x[4] = q1.x, x[5] = q1.y, x[6] = q1.z, x[7] = q1.w;
  }
  __device__ __forceinline__ uint32_t below(uint32_t n, uint32_t v) const {  // entries < v among the first n
    uint32_t k = 0;
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) k += (j < n && x[j] < v) ? 1u : 0u;
    return k;
  }
  __device__ __forceinline__ bool holds(uint32_t n, uint32_t v) const {
    bool h = false;
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) h = h || (j < n && x[j] == v);
    return h;
  }
};

// What the first removal pass left for later (bits of BfsCounters::later).
constexpr uint32_t kLaterRuns = 1u;  // delta removals of runs of several arcs
constexpr uint32_t kLaterArcs = 2u;  // arcs marked kFPending
constexpr uint32_t kLaterRows = 4u;  // rows of blocks with too many arcs (canon_grid)

// The removal pass.  A batch of few arcs takes a warp per arc: its row searches
// read 32 pivots per round trip instead of 7, and the chain of such a batch is
// its longest row's.  With the classification, the removals and the candidates
// in three passes and two barriers 950 arcs at R-MAT 20 took 20 us, now 7 to 8;
// 20,000 arcs at R-MAT 22 22 us, now 15.  Block-uniform.
__device__ void removal_pass(ArcWork& w, RepairSmem& sm) {
  if (w.raw && w.F > kRawMine) {  // hub rows: listed, and left to the grid
    for (uint32_t i = threadIdx.x; i < w.F; i += kThreads) {
      uint32_t u, v;
      uint8_t f;
      w.arc(i, u, v, f);
      w.ff[w.base + i] = f | kFPending;
    }
    if (threadIdx.x == 0) atomicOr(&w.p->c->later, kLaterArcs);
    return;
  }
  const Params& p = *w.p;
  const vxb::DevAdj& a = *w.a;
  const uint32_t lane = threadIdx.x & 31;
  bool multi = false;  // a delta removal left to removal_runs
  const uint32_t base = w.base;
  if (w.raw ? w.F <= kRawWarps : w.F <= 2 * nwarps()) {
    for (uint32_t i = w.raw ? threadIdx.x >> 5 : dealt_warp(); i < w.F; i += w.raw ? kThreads / 32 : nwarps()) {
      uint32_t u, v;
      uint8_t f;
      w.arc(i, u, v, f);
      if (w.pending && !(f & kFPending)) continue;
      uint64_t b, e;
      vxb::base_range(a, u, b, e);
      const uint2 row = a.drow[u];
      const bool small = row.y <= 32u, run = w.in_run(i, u);
      const uint32_t x = small && lane < row.y ? a.darena[row.x + lane] : 0u;  // in flight with the base search
      uint64_t q = ~0ull;
      const uint32_t held = __ballot_sync(FULL, small && lane < row.y && x == v);
      if (!w.s->classified) {
        const uint64_t at = warp_find(a.col, b, e, v);
        bool cur;
        f &= kFAdd;
        if (at < e) {
          f |= kFInBase;
          cur = !(a.col[at] & kTomb);
          q = at;
        } else {
          cur = small ? held != 0u : warp_find(a.darena, row.x, row.x + row.y, v) < row.x + row.y;
        }
        if (cur) f |= kFCur;
        if (cur != ((f & kFAdd) != 0)) f |= kFChanged;
        if (lane == 0) {
          w.ff[base + i] = f;
          w.fpos[base + i] = q;
        }
      } else {
        q = w.fpos[base + i];
      }
      // lane 0 does what is not a search
      if (lane == 0) w.tombs += gdev::tomb_arc(a, u, f, q, 0, w.dirtied);
      w.candidate(lane == 0, u, v, f);
      if (!delta_op(f, false)) continue;
      if (run) {
        multi = true;
      } else if (small) {  // the entries above the arc move down
        const uint32_t k = (uint32_t)__ffs(held) - 1;
        if (lane > k && lane < row.y) a.darena[row.x + lane - 1] = x;
        if (lane == 0) {
          a.drow[u].y = row.y - 1;
          atomicAdd(&w.s->gc->delta_live[w.dir], ~0ull);
          acct_add(p, 2, 2ull * row.y - 1);
          w.dirtied += gdev::mark_dirty_count(a.dirty, u);
        }
      } else {
        __syncwarp();
        w.remove_one(u, v);
      }
    }
  } else {
    for (uint32_t r0 = 0; r0 < w.F; r0 += w.raw ? kThreads : nthreads()) {
      if (threadIdx.x == 0) sm.nsv = 0;
      __syncthreads();
      const uint32_t i = r0 + (w.raw ? threadIdx.x : dealt_thread());
      bool act = i < w.F && !(w.pending && !(w.ff[i] & kFPending));
      bool queue = false;
      uint32_t u = 0, v = 0;
      uint8_t f = 0;
      long long dlive = 0;
      if (act) {
        w.arc(i, u, v, f);
        uint64_t b, e;
        vxb::base_range(a, u, b, e);
        const uint2 row = a.drow[u];
        SmallRow r = {};
        if (row.y && row.y <= 8u) r.load(a.darena + row.x);  // in flight with the base search
        uint64_t q = ~0ull;
        if (!w.s->classified) {
          const uint64_t at = vxb::lower_bound_masked(a.col, b, e, v);
          const uint32_t c = at < e ? a.col[at] : kTomb;
          bool cur;
          f &= kFAdd;
          if (at < e && (c & kIdMask) == v) {
            f |= kFInBase;
            cur = !(c & kTomb);
            q = at;
          } else {
            cur = row.y <= 8u ? r.holds(row.y, v) : gdev::bsearch_u32(a.darena, row.x, row.x + row.y, v);
          }
          if (cur) f |= kFCur;
          if (cur != ((f & kFAdd) != 0)) f |= kFChanged;
          w.ff[base + i] = f;
          w.fpos[base + i] = q;
        } else {
          q = w.fpos[base + i];
        }
        w.tombs += gdev::tomb_arc(a, u, f, q, 0, w.dirtied);
        if (delta_op(f, false)) {
          if (w.in_run(i, u)) {
            multi = true;
          } else if (row.y > 8u) {
            queue = true;
          } else {
            const uint32_t pos = r.below(row.y, v);
            auto out = [&](uint32_t k) { return k < pos ? r.x[k] : r.x[k < 7 ? k + 1 : 7]; };
            uint4* dst = reinterpret_cast<uint4*>(a.darena + row.x);
            dst[0] = make_uint4(out(0), out(1), out(2), out(3));
            dst[1] = make_uint4(out(4), out(5), out(6), out(7));
            a.drow[u].y = row.y - 1;
            dlive = -1;
            acct_add(p, 2, 2ull * row.y - 1);
            w.dirtied += gdev::mark_dirty_count(a.dirty, u);
          }
        }
      }
      w.candidate(act, u, v, f);
      dlive = vxb::warp_sum(dlive);
      if (lane == 0 && dlive) atomicAdd(&w.s->gc->delta_live[w.dir], (unsigned long long)dlive);
      if (queue) sm.sv[atomicAdd(&sm.nsv, 1u)] = base + i;
      __syncthreads();
      const uint32_t nq = sm.nsv;
      for (uint32_t k = threadIdx.x >> 5; k < nq; k += kThreads / 32) w.remove_one(w.fu[sm.sv[k]], w.fv[sm.sv[k]]);
      __syncthreads();  // the list is rebuilt by the next round
    }
  }
  if (__any_sync(FULL, multi) && lane == 0) atomicOr(&p.c->later, kLaterRuns);
  w.flush();
}

// The second removal pass: delta removals of runs of several arcs, a warp per
// run.  Block-uniform.
__device__ void removal_runs(ArcWork& w, RepairSmem& sm) {
  for (uint32_t r0 = 0; r0 < w.F; r0 += nthreads()) {
    if (threadIdx.x == 0) sm.nsv = 0;
    __syncthreads();
    const uint32_t i = r0 + dealt_thread();
    if (i + 1 < w.F) {
      const uint32_t u = w.fu[i];
      if (w.fu[i + 1] == u && (i == 0 || w.fu[i - 1] != u)) sm.sv[atomicAdd(&sm.nsv, 1u)] = i;
    }
    __syncthreads();
    const uint32_t nq = sm.nsv;
    for (uint32_t k = threadIdx.x >> 5; k < nq; k += kThreads / 32)
      run_remove(*w.a, w.dir, w.fv, w.ff, sm.sv[k], run_end(w.fu, sm.sv[k], w.F), w.fu[sm.sv[k]], w.s->gc,
                 w.p->acct ? w.p->acct + 2 : nullptr);
    __syncthreads();  // the list is rebuilt by the next round
  }
}

// The insertion pass: tombstoned base arcs the batch re-adds revived, delta
// insertions made.  Block-uniform.
__device__ void insertion_pass(ArcWork& w, RepairSmem& sm) {
  const Params& p = *w.p;
  const vxb::DevAdj& a = *w.a;
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t r0 = 0; r0 < w.F; r0 += nthreads()) {
    if (threadIdx.x == 0) sm.nsv = 0;
    __syncthreads();
    const uint32_t i = r0 + dealt_thread();
    bool job = false, queue = false, need_block = false;
    uint32_t u = 0, v = 0;
    uint2 row = make_uint2(0, 0);
    if (i < w.F) {
      u = w.fu[i];
      const uint8_t f = w.ff[i];
      if ((f & kFInBase) && (f & kFChanged) && (f & kFAdd))
        w.tombs += gdev::tomb_arc(a, u, f, w.fpos[i], 1, w.dirtied);
      if (i == 0 || w.fu[i - 1] != u) {
        if (i + 1 < w.F && w.fu[i + 1] == u) {
          queue = true;  // a run of several arcs
        } else if (delta_op(f, true)) {
          v = w.fv[i];
          row = a.drow[u];
          if (row.y < 8u) {
            job = true;
            need_block = a.dcap[u] == 0u;  // no block yet (then the row is empty)
          } else {
            queue = true;
          }
        }
      }
    }
    const uint32_t nm = __ballot_sync(FULL, need_block);
    uint32_t base_off = row.x;
    if (nm) {
      const int leader = __ffs(nm) - 1;
      unsigned long long b0 = 0;
      if ((int)lane == leader) b0 = atomicAdd(&w.s->gc->arena_top[w.dir], 8ull * (unsigned long long)__popc(nm));
      b0 = __shfl_sync(FULL, b0, leader);
      const unsigned long long o = b0 + 8ull * __popc(nm & vxb::lanemask_lt());
      if (need_block) {
        if (o + 8 > w.s->arena_cap[w.dir]) {
          atomicOr(&w.s->gc->err, vxb::kErrArenaOverflow);
          job = false;
        } else {
          base_off = (uint32_t)o;
        }
      }
    }
    long long dlive = 0;
    if (job) {
      SmallRow r = {};
      if (row.y) r.load(a.darena + row.x);
      // output k: x[k] below the new arc's position, the arc at it, x[k - 1] above
      const uint32_t pos = r.below(row.y, v);
      auto out = [&](uint32_t k) { return k < pos ? r.x[k] : (k == pos ? v : r.x[k > 0 ? k - 1 : 0]); };
      uint4* dst = reinterpret_cast<uint4*>(a.darena + base_off);
      dst[0] = make_uint4(out(0), out(1), out(2), out(3));
      dst[1] = make_uint4(out(4), out(5), out(6), out(7));
      dlive = 1;
      acct_add(p, 2, 2ull * row.y + 1);
      a.drow[u] = make_uint2(base_off, row.y + 1);
      if (need_block) a.dcap[u] = 8u;
      w.dirtied += gdev::mark_dirty_count(a.dirty, u);
    }
    dlive = vxb::warp_sum(dlive);
    if (lane == 0 && dlive) atomicAdd(&w.s->gc->delta_live[w.dir], (unsigned long long)dlive);
    if (queue) sm.sv[atomicAdd(&sm.nsv, 1u)] = i;
    __syncthreads();
    const uint32_t nq = sm.nsv;
    for (uint32_t k = threadIdx.x >> 5; k < nq; k += kThreads / 32) {
      const uint32_t st = sm.sv[k], en = run_end(w.fu, st, w.F);
      run_insert(a, w.dir, w.fv, w.ff, w.s->scratch[w.dir], st, en, w.fu[st], w.s->gc, w.s->arena_cap[w.dir],
                 p.acct ? p.acct + 2 : nullptr);
    }
    __syncthreads();  // the list is rebuilt by the next round
  }
  w.flush();
}

// The start of a repair launch: the block's own copy of what its phases change.
__device__ __forceinline__ void start_phases(const Params& p) {
  if (threadIdx.x == 0)
    ph = PhaseParams{p.V, p.dist_len, 0u, p.rq_tail, 0u, p.cascade_bfs, p.fu, p.fv, p.ff, p.F, p.fallback_limit};
  __syncthreads();
}

__device__ void stream_kernel_body(const Params& p, const StreamArgs& s, RepairSmem& sm, LbStage& lb, BlockQueue& bq) {
  BfsCounters* c = p.c;
  const uint32_t sort_err = sort_error(p);
  unsigned long long tmark = globaltimer();
  auto phase = [&](int k) {  // gtid 0 accumulates the time since the previous mark
    if (gtid() == 0) {
      const unsigned long long now = globaltimer();
      c->stream_ns[k] += now - tmark;
      tmark = now;
    }
  };
  if (gtid() == 0) {  // stamps and drain statistics are written by this thread only
    for (int k = 0; k < 6; ++k) c->stream_ns[k] = 0;
    for (int k = 0; k < (int)(sizeof(c->rtrace) / sizeof(c->rtrace[0])); ++k) c->rtrace[k] = 0;
    c->handovers[0] = c->handovers[1] = 0;
  }
  const int ndir = p.g.directed ? 2 : 1;
  start_phases(p);
  for (uint32_t bi = 0; bi < s.nb; ++bi) {
    RawArcs& raw = reinterpret_cast<RawArcs&>(lb);
    uint32_t off = 0, F = 0, Frev = 0;
    if (s.boff) off = s.boff[bi];
    const uint32_t Vpre = bi ? s.vpost[bi - 1] : s.V0, lpre = bi ? s.vpost[bi - 1] : s.len0;
    if (threadIdx.x == 0) {  // the ring's epoch is the first again (reset_ring)
      ph.fu = s.fu[0] + off;
      ph.fv = s.fv[0] + off;
      ph.ff = s.ff[0] + off;
      ph.F = s.raw_n ? p.bar + kRawWord : &s.cnt[0][bi];
      ph.V = Vpre;
      ph.dist_len = lpre;
      ph.touched_base = 0;
      const unsigned long long lim = (unsigned long long)((double)Vpre * s.frac);
      ph.fallback_limit = lim < 1 ? 1 : lim;
    }
    __syncthreads();
    if (s.raw_n) {
      if (canon_raw(s, p.g.directed, raw, p.bar + kRawWord) && threadIdx.x == 0) atomicOr(&c->later, kLaterRows);
    } else {
      F = s.cnt[0][bi];
      if (s.cnt[1]) Frev = *s.cnt[1];
    }
    const uint32_t Vpost = s.vpost ? s.vpost[bi] : s.v_single;
    auto work = [&](int dir) {
      const uint32_t o = dir ? 0u : off;
      return ArcWork{&p, &s, dir ? &p.g.in : &p.g.out, dir, s.fu[dir] + o, s.fv[dir] + o, s.ff[dir] + o, s.fpos[dir] + o,
                     dir ? Frev : F, nullptr, 0u, false, 0ll, 0u};
    };
    stamp(p, 0);
    // A: classification against the pre-batch graph, removals, deletion candidates
    for (int dir = 0; dir < ndir; ++dir) {
      ArcWork w = work(dir);
      if (s.raw_n) {
        w.raw = raw.key + (dir ? raw.n[1] : 0u);
        w.base = raw.base[dir];
        w.F = dir ? raw.n[0] - raw.n[1] : raw.n[1];
      }
      removal_pass(w, sm);
    }
    if (s.digest && bi > 0) digest_pass(p.dist, lpre, &s.digest[bi - 1]);
    if (sort_err) atomicOr(&c->err, sort_err);
    if (!sync_words(p, sm.w)) return;
    phase(0);
    if ((sm.w.later & kLaterRows) && !(canon_grid(p, s, raw, sm.w) && sync_words(p, sm.w))) return;
    if (s.raw_n) {
      F = sm.w.raw_f[0];
      Frev = sm.w.raw_f[1];
    }
    if (sm.w.later & (kLaterArcs | kLaterRows)) {
      for (int dir = 0; dir < ndir; ++dir) {
        ArcWork w = work(dir);
        w.pending = true;
        removal_pass(w, sm);
      }
      if (!sync_words(p, sm.w)) return;
    }
    if (sm.w.later & kLaterRuns) {
      for (int dir = 0; dir < ndir; ++dir) {
        ArcWork w = work(dir);
        removal_runs(w, sm);
      }
      if (!sync_words(p, sm.w)) return;
    }
    phase(1);
    stamp(p, 1);
    // B: the cascade over the graph without the batch's deletions
    const uint32_t ncand = sm.w.candidates;
    if (threadIdx.x == 0) {
      ph.touched_base = ncand;
      ph.cascade_bfs = lpre == Vpre;
    }
    __syncthreads();
    if (gtid() == 0) {
      // last_* counters (bfs.hpp:30-33); the last reader of the previous
      // batch's was this thread, at its end
      c->candidates = ncand;
      c->affected = c->full = 0;
      acct_add(p, 1, ncand + F);  // candidate checks, heads of the canonical arcs
      acct_add(p, 3, F);
      acct_add(p, 4, 1);
    }
    if (ncand) {
      if (!cascade(p, sm, lb, bq, ncand)) return;
      reset_ring(p);
    }
    phase(2);
    stamp(p, 2);
    // C: insertions; new vertices start unreachable and, unless a BFS gives
    // the distances, the affected ones are invalidated
    for (int dir = 0; dir < ndir; ++dir) {
      ArcWork w = work(dir);
      insertion_pass(w, sm);
    }
    for (uint32_t v = lpre + gtid(); v < Vpost; v += nthreads()) p.dist[v] = kUnreachable;
    if (!sm.w.cbig && !sm.w.fallback) invalidate(p, sm.w.affected);
    if (!sync_words(p, sm.w)) return;
    phase(3);
    // D: the post-batch repair (or the fallback full BFS) on the new graph
    if (threadIdx.x == 0) ph.V = ph.dist_len = Vpost;
    __syncthreads();
    repair_post<true>(p, sm, lb, bq);
    phase(4);
    // the repair lists start empty in the next batch (and launch); every block
    // has their lengths in sm.w
    if (gtid() == 0) {
      c->cand_n = c->touched_n = c->a_n = c->fallback = c->later = 0;
      p.bar[kRawWord] = p.bar[kRawWord + 1] = 0u;
    }
    if (bi + 1 == s.nb && !s.digest && !s.bstats) break;
    // every block's counter updates are in before they are recorded and the
    // next batch begins
    if (!sync_grid(p)) return;
    phase(5);
    if (gtid() == 0 && s.bstats) {
      s.bstats[4 * bi + 0] = ld_cg(&c->candidates);
      s.bstats[4 * bi + 1] = ld_cg(&c->affected);
      s.bstats[4 * bi + 2] = ld_cg(&c->full);
      s.bstats[4 * bi + 3] = (uint32_t)__ldcg(&c->reachable);
    }
  }
  if (s.digest && s.nb) digest_pass(p.dist, s.vpost[s.nb - 1], &s.digest[s.nb - 1]);
}

// The full BFS has a kernel of its own (the repair kernels run it too, for the
// fallback and the budget handovers), one block of 1,024 threads per SM: the
// grid barrier's cost grows with the blocks that meet at it, and 32 warps with
// four arcs per lane in flight keep the memory as busy as 48 with one did.
// R-MAT of 30,000 vertices: 75 us with 444 blocks of 512 threads, 56 with 296,
// 45 with 148.  Graphs of fewer than kWideArcs arcs take 512 threads, whose
// block barriers are cheaper (40 us; R-MAT 2^20, 31M arcs: 89 us with 512, 77 with
// 1,024; R-MAT 2^22: 244 and 168), and 64 registers, so that the searches of two
// graphs run side by side: three graphs in turn, us a search, and one alone: R-MAT of
// 24,821 vertices 21 and 41, 500,000 38 and 80, 700 x 700 lattice 350 and 635.  With
// eight arcs per lane and 110 registers one launch had the SMs to itself: 37 and 40,
// 63 and 74, 611 and 619.
template <int kT>
struct FullSmem {
  BlockQueueOf<8192> bq;
  LbStage lb;
  BuStage<kT, kT / 512> bu;
  uint32_t bits[8192];
};

template <int kT>
__global__ void __launch_bounds__(kT, 1024 / kT) bfs_full_kernel(Params p) {
  extern __shared__ __align__(16) unsigned char full_smem[];
  FullSmem<kT>& sm = *reinterpret_cast<FullSmem<kT>*>(full_smem);
  full_bfs<false>(p, sm.bq, sm.lb, sm.bu, sm.bits, 8192u, p.dist, p.trace);
}

__global__ void __launch_bounds__(kThreads, 2) bfs_kernel(const __grid_constant__ Params p, int mode) {
  __shared__ BlockQueue bq;
  __shared__ LbStage lb;
  __shared__ RepairSmem sm;
  start_phases(p);
  if (const uint32_t e = sort_error(p)) atomicOr(&p.c->err, e);
  if (mode == kModePre) repair_pre(p, sm, lb, bq);
  else repair_post<false>(p, sm, lb, bq);
}

// Registers for two blocks per SM: the launches of two graphs (on their own
// streams) then run side by side, which a block with 128 registers a thread
// (no spills, 2% faster alone) does not allow: 10,000-op batches on three R-MAT
// 22 graphs in turn 86 us a batch, 111 us with 128 registers.
// The arguments stay in the kernel's parameter space: as copies for the functions
// that take them by reference they made a stack frame of 1,184 bytes a thread
// instead of 928 (10,000 ops at R-MAT 22, three graphs in turn: 70 us a batch
// instead of 62).
__global__ void __launch_bounds__(kThreads, 2) bfs_stream_kernel(const __grid_constant__ Params p,
                                                                 const __grid_constant__ StreamArgs s) {
  __shared__ BlockQueue bq;
  __shared__ LbStage lb;
  __shared__ RepairSmem sm;
  stream_kernel_body(p, s, sm, lb, bq);
}

// Stream canonicalisation: both arcs of every non-self-loop op keyed by
// (batch, u, v) with the op's stream index as the value; a stable sort then
// leaves each batch's ops for one arc in order, and the last one wins.
__global__ void stream_keys_kernel(const uint32_t* src, const uint32_t* dst, const uint8_t* add,
                                   const uint64_t* boff, uint32_t nb, size_t n, int b, uint64_t* keys,
                                   uint32_t* vals) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = nb;  // the batch t with boff[t] <= i < boff[t + 1]
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (boff[mid] <= i) lo = mid;
      else hi = mid;
    }
    const uint64_t t = (uint64_t)lo << (2 * b);
    const uint32_t u = src[i], v = dst[i];
    const uint32_t val = ((uint32_t)i << 1) | (add[i] ? 1u : 0u);
    const bool ok = u != v;
    keys[2 * i] = ok ? (t | ((uint64_t)u << b) | v) : ~0ull;
    keys[2 * i + 1] = ok ? (t | ((uint64_t)v << b) | u) : ~0ull;
    vals[2 * i] = val;
    vals[2 * i + 1] = val;
  }
}

__global__ void stream_last_kernel(const uint64_t* keys, size_t m, const uint32_t* err, uint32_t* flag) {
  const bool sorted = !(*err & vxb::kErrBarrierTimeout);  // no arcs after a sort whose wait ran out
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < m; i += (size_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    flag[i] = sorted && (k != ~0ull) && (i + 1 == m || keys[i + 1] != k);
  }
}

__global__ void stream_compact_kernel(const uint64_t* keys, const uint32_t* vals, const uint32_t* flag,
                                      const uint32_t* pos, size_t m, int b, uint32_t* fu, uint32_t* fv, uint8_t* ff,
                                      uint32_t* bid) {
  const uint64_t mask = ((uint64_t)1 << b) - 1;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < m; i += (size_t)gridDim.x * blockDim.x) {
    if (!flag[i]) continue;
    const uint32_t q = pos[i];
    const uint64_t k = keys[i];
    fu[q] = (uint32_t)((k >> b) & mask);
    fv[q] = (uint32_t)(k & mask);
    ff[q] = (uint8_t)(vals[i] & 1u);
    bid[q] = (uint32_t)(k >> (2 * b));
  }
}

// boff[t] = first canonical arc of batch t (t <= nb), bcnt[t] = its arc count.
__global__ void stream_bounds_kernel(const uint32_t* bid, const uint32_t* total, uint32_t nb, uint32_t* boff,
                                     uint32_t* bcnt) {
  const uint32_t F = *total;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t <= nb; t += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = F;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (bid[mid] < t) lo = mid + 1;
      else hi = mid;
    }
    boff[t] = lo;
    uint32_t lo2 = lo, hi2 = F;
    while (lo2 < hi2) {
      const uint32_t mid = (lo2 + hi2) >> 1;
      if (bid[mid] <= t) lo2 = mid + 1;
      else hi2 = mid;
    }
    if (t < nb) bcnt[t] = lo2 - lo;
  }
}

__global__ void digest_kernel(const uint32_t* dist, uint32_t n, unsigned long long* out) {
  unsigned long long h = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    h += mix64(((unsigned long long)v << 32) | dist[v]);
  h = vxb::warp_sum(h);
  if ((threadIdx.x & 31) == 0 && h) atomicAdd(out, h);
}


__global__ void reached_arcs_kernel(vxb::DevAdj a, const uint32_t* dist, uint32_t n,
                                    unsigned long long* out) {
  unsigned long long s = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    if (dist[v] == kUnreachable) continue;
    uint64_t b, e;
    vxb::base_range(a, v, b, e);
    // live arcs: base minus tombstones plus delta
    s += (e - b) - a.tcnt[v] + a.drow[v].y;
  }
  s = vxb::warp_sum(s);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(out, s);
}

}  // namespace

// ---------------------------------------------------------------- host --

static int ensure_capacity(Bfs* b, size_t V) {
  if (V <= b->cap && b->dist) return 0;
  size_t c = std::max<size_t>(b->cap ? b->cap : 1024, 1024);
  while (c < V) c *= 2;
  const size_t words = (c + 31) / 32 + 1;
  cudaStream_t s = b->g->stream;
  VX_CUDA_TRY(cudaStreamSynchronize(s));
  // fills and copies go on the graph's (non-blocking) stream, ahead of the
  // kernels that use the new buffers; the old buffers are freed once the
  // stream has finished copying out of them
  std::vector<uint32_t*> old;
  auto realloc_copy = [&](uint32_t** p, size_t n_new, size_t n_old, int fill) -> int {
    uint32_t* q = nullptr;
    if (cudaMalloc(&q, n_new * sizeof(uint32_t)) != cudaSuccess) {
      set_error("BFS allocation of %zu bytes failed", n_new * 4);
      return -4;
    }
    if (cudaMemsetAsync(q, fill, n_new * sizeof(uint32_t), s) != cudaSuccess) return -3;
    if (*p && n_old && cudaMemcpyAsync(q, *p, n_old * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
      return -3;
    if (*p) old.push_back(*p);
    *p = q;
    return 0;
  };
  const size_t oldw = b->cap ? (b->cap + 31) / 32 + 1 : 0;
  int rc = 0;
  rc |= realloc_copy(&b->dist, c, b->cap, 0xFF);
  rc |= realloc_copy(&b->sw, 2 * c, 0, 0);
  rc |= realloc_copy(&b->vis, words, 0, 0);
  rc |= realloc_copy(&b->aff, words, oldw, 0);
  rc |= realloc_copy(&b->inq[0], words, oldw, 0);
  rc |= realloc_copy(&b->inq[1], words, oldw, 0);
  for (int k = 0; k < 3; ++k) {
    rc |= realloc_copy(&b->fb[k], words, 0, 0);
    rc |= realloc_copy(&b->q[k], c, 0, 0);
  }
  rc |= realloc_copy(&b->big, c, 0, 0);
  rc |= realloc_copy(&b->lst_a, c, 0, 0);
  rc |= realloc_copy(&b->lst_t, c, 0, 0);
  rc |= realloc_copy(&b->tent, c, 0, 0);
  rc |= realloc_copy(&b->bul, 2 * list_slots(c), 0, 0);
  const cudaError_t e = cudaStreamSynchronize(s);
  for (uint32_t* p : old) cudaFree(p);
  if (rc) return -4;
  VX_CUDA_TRY(e);
  b->cap = c;
  return 0;
}

// The work ring holds at most one pending item per vertex plus the extra
// chunks of long rows (one per kChunk arcs), so it is sized for capacity +
// arcs / kChunk, with the delta arena counted at its allocated size (so a
// reserved arena needs no growth mid-stream); made with the object and
// checked before every staged batch.
static int ensure_ring(Bfs* b) {
  const Adjacency& a = b->g->adj[0];
  // + the tickets blocks hold past the tail (kClaim each) and slack
  const size_t need = b->cap + (size_t)((a.A + std::max<uint64_t>(a.arena_bound, a.arena_cap)) / kChunk) +
                      (size_t)kThreads * 1024;
  size_t slots = 1;
  while (slots < need) slots <<= 1;
  if (slots <= b->ring_slots) return 0;
  VX_CUDA_TRY(cudaStreamSynchronize(b->g->stream));
  cudaFree(b->ring);
  b->ring = nullptr;
  b->ring_slots = 0;
  if (cudaMalloc(&b->ring, slots * sizeof(unsigned long long)) != cudaSuccess) {
    set_error("BFS work ring allocation of %zu bytes failed", slots * 8);
    return -4;
  }
  // on the graph's stream, so the first launch that drains the ring sees every
  // slot empty (the graph's stream is non-blocking: a legacy-stream memset
  // would not be ordered before it)
  VX_CUDA_TRY(cudaMemsetAsync(b->ring, 0xFF, slots * sizeof(unsigned long long), b->g->stream));
  b->ring_slots = slots;
  return 0;
}

static Params make_params(Bfs* b, uint32_t V, uint32_t dist_len) {
  Graph* g = b->g;
  Params p;
  memset(&p, 0, sizeof(p));
  p.g = g->view();
  p.V = V;
  p.handover = b->tune.handover;
  p.cascade_bfs = dist_len == V;
  p.dist_len = dist_len;
  p.source = b->source;
  p.dist = b->dist;
  p.vis = b->vis;
  for (int k = 0; k < 3; ++k) {
    p.fb[k] = b->fb[k];
    p.q[k] = b->q[k];
  }
  p.big = b->big;
  p.lst_a = b->lst_a;
  p.lst_t = b->lst_t;
  p.tent = b->tent;
  p.bul = b->bul;
  p.bul_half = (uint32_t)list_slots(b->cap);
  p.sw = reinterpret_cast<unsigned long long*>(b->sw);
  p.ring = b->ring;
  p.ring_mask = b->ring_slots ? (uint32_t)(b->ring_slots - 1) : 0u;
  p.rq_head = b->rq;
  p.rq_tail = b->rq + 32;
  p.rq_done = b->rq + 64;
  p.rq_fin = b->rq + 128;
  p.rq_stat = reinterpret_cast<unsigned long long*>(b->rq + 96);
  p.aff = b->aff;
  p.inq[0] = b->inq[0];
  p.inq[1] = b->inq[1];
  p.fu = g->batch.fu;
  p.fv = g->batch.fv;
  p.ff = g->batch.ff;
  p.F = &g->ctr->final_arcs;
  p.c = b->ctr;
  p.graph_err = &g->ctr->err;
  p.total_arcs = g->adj[0].A;  // estimate for the direction switch
  p.alpha = b->tune.alpha;
  p.beta = b->tune.beta;
  p.large_row = b->tune.large_row;
  p.trace = b->trace;
  p.acct = b->acct_on ? b->acct : nullptr;
  p.bar = b->barrier;
  p.deltas = (g->adj[0].arena_bound | g->in().arena_bound) != 0;
  return p;
}

// Every co-resident block of the kernel, once per object.
static int grid_of(const void* kernel, int* grid) {
  if (*grid) return 0;
  int per_sm = 0;
  VX_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0));
  if (per_sm < 1) {
    set_error("BFS kernel cannot be resident on an SM");
    return -3;
  }
  *grid = per_sm * sm_count();
  return 0;
}

// One block per SM, fewer for a graph whose arcs one step of fewer blocks covers
// (kT threads of kVisit arcs): 2,000 vertices 38 us with 148 blocks, 32 with 20.
template <int kT>
static int launch_full_t(Params& p, cudaStream_t s) {
  static std::atomic<int> sms_dev[64];  // SMs of a device whose kernel has its shared memory limit set
  int dev = 0;
  VX_CUDA_TRY(cudaGetDevice(&dev));
  int sms = dev < 64 ? sms_dev[dev].load(std::memory_order_acquire) : 0;
  if (!sms) {
    VX_CUDA_TRY(cudaFuncSetAttribute(bfs_full_kernel<kT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(FullSmem<kT>)));
    VX_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (dev < 64) sms_dev[dev].store(sms, std::memory_order_release);
  }
  const uint64_t want = std::max<uint64_t>(p.V, p.total_arcs) / (kT * kVisit) + 8;
  p.nblocks = (uint32_t)std::min<uint64_t>(want, (uint64_t)sms);
  void* args[] = {&p};
  vxh::count_launch();
  VX_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)bfs_full_kernel<kT>, dim3(p.nblocks), dim3(kT), args,
                                          sizeof(FullSmem<kT>), s));
  return 0;
}

// Launches the full BFS (p.V, p.total_arcs set); p.nblocks is set here.
constexpr uint64_t kWideArcs = 1ull << 24;
static int launch_full(Params& p, cudaStream_t s) {
  return std::max<uint64_t>(p.V, p.total_arcs) >= kWideArcs ? launch_full_t<1024>(p, s) : launch_full_t<512>(p, s);
}

static int launch(Bfs* b, Params& p, int mode) {
  if (mode == kModeFull) return launch_full(p, b->g->stream);
  if (int rc = grid_of((const void*)bfs_kernel, &b->grid)) return rc;
  p.nblocks = (uint32_t)b->grid;
  void* args[] = {&p, &mode};
  vxh::count_launch();
  VX_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)bfs_kernel, dim3(b->grid), dim3(kThreads), args, 0,
                                          b->g->stream));
  return 0;
}

int bfs_create(Bfs** out, Graph* g, uint32_t source, double frac) {
  Bfs* b = new Bfs();
  b->g = g;
  b->source = source;
  b->frac = frac;
  if (cudaMalloc(&b->ctr, sizeof(BfsCounters)) != cudaSuccess ||
      cudaMalloc(&b->trace, 2 * (kTraceLevels + 1) * sizeof(unsigned long long)) != cudaSuccess ||
      cudaMalloc(&b->barrier, vxb::kBarrierWords * sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&b->features, 64 * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&b->rq, 160 * sizeof(uint32_t)) != cudaSuccess ||
      cudaMallocHost(&b->hctr, sizeof(BfsCounters)) != cudaSuccess) {
    set_error("BFS counter allocation failed");
    bfs_destroy(b);
    return -4;
  }
  cudaMemsetAsync(b->ctr, 0, sizeof(BfsCounters), g->stream);
  cudaMemsetAsync(b->barrier, 0, vxb::kBarrierWords * sizeof(uint32_t), g->stream);
  cudaMemsetAsync(b->rq, 0, 160 * sizeof(uint32_t), g->stream);
  memset(b->hctr, 0, sizeof(BfsCounters));
  int rc = bfs_recompute(b);
  if (!rc) rc = ensure_ring(b);  // before the first batch, which would otherwise allocate it
  if (rc) {
    bfs_destroy(b);
    return rc;
  }
  *out = b;
  return 0;
}

void bfs_destroy(Bfs* b) {
  if (!b) return;
  if (b->g && b->g->stream) cudaStreamSynchronize(b->g->stream);
  uint32_t* ptrs[] = {b->dist, b->vis, b->fb[0], b->fb[1], b->fb[2], b->q[0], b->q[1], b->q[2], b->big,
                      b->lst_a, b->lst_t, b->tent, b->bul, b->sw, b->aff, b->inq[0], b->inq[1]};
  for (uint32_t* p : ptrs) cudaFree(p);
  cudaFree(b->ctr);
  cudaFree(b->acct);
  cudaFree(b->trace);
  cudaFree(b->barrier);
  cudaFree(b->features);
  cudaFree(b->rq);
  cudaFree(b->ring);
  b->sb.free_all();
  delete b->vb;
  cudaFreeHost(b->hctr);
  delete b;
}

int bfs_ensure_capacity(Bfs* b, size_t V) { return ensure_capacity(b, V); }

int bfs_recompute(Bfs* b) {
  Graph* g = b->g;
  const size_t V = g->V;
  if (int rc = ensure_capacity(b, std::max<size_t>(V, 1))) return rc;
  b->dist_len = V;
  VX_CUDA_TRY(cudaMemsetAsync(&b->ctr->candidates, 0, 4 * sizeof(uint32_t), g->stream));
  if (V == 0) {
    VX_CUDA_TRY(cudaMemsetAsync(&b->ctr->reachable, 0, 8, g->stream));
    return 0;
  }
  Params p = make_params(b, (uint32_t)V, (uint32_t)V);
  return launch(b, p, kModeFull);
}

// The direction switch and the grid-expanded row length of the full BFS,
// picked by timing: every candidate (alpha, beta, large_row) of a small grid
// runs a full BFS from each of the given roots (CUDA events on the graph's
// stream, one untimed warm-up per candidate), the median over the roots
// decides, and the best candidate stays set on b.  The distances from b's
// own source are recomputed afterwards.
int bfs_autotune(Bfs* b, const uint32_t* roots, size_t k, float* chosen) {
  static const float kAlpha[] = {4.f, 14.f, 40.f, 120.f};
  static const float kBeta[] = {8.f, 24.f, 96.f};
  static const uint32_t kLarge[] = {512u, 1024u, 4096u};
  Graph* g = b->g;
  cudaStream_t s = g->stream;
  const uint32_t source = b->source;
  const BfsTuning keep = b->tune;
  cudaEvent_t e0, e1;
  VX_CUDA_TRY(cudaEventCreate(&e0));
  VX_CUDA_TRY(cudaEventCreate(&e1));
  float best = -1.f;
  BfsTuning pick = keep;
  std::vector<float> ts(k);
  int rc = 0;
  for (float al : kAlpha)
    for (float be : kBeta)
      for (uint32_t lr : kLarge) {
        b->tune.alpha = al;
        b->tune.beta = be;
        b->tune.large_row = lr;
        // each root timed twice, the faster run kept (a single run now and
        // then lands several percent slow); the candidate's score is the
        // mean over the roots
        for (size_t r = 0; r < k && !rc; ++r) {
          b->source = roots[r];
          if (r == 0) rc = bfs_recompute(b);  // warm-up of this candidate
          ts[r] = -1.f;
          for (int rep = 0; rep < 2 && !rc; ++rep) {
            float t = 0.f;
            if (cudaEventRecord(e0, s) != cudaSuccess) rc = -3;
            if (!rc) rc = bfs_recompute(b);
            if (!rc && cudaEventRecord(e1, s) != cudaSuccess) rc = -3;
            if (!rc && cudaEventSynchronize(e1) != cudaSuccess) rc = -3;
            if (!rc && cudaEventElapsedTime(&t, e0, e1) != cudaSuccess) rc = -3;
            if (!rc && (ts[r] < 0.f || t < ts[r])) ts[r] = t;
          }
        }
        if (rc) break;
        float mean = 0.f;
        for (float t : ts) mean += t;
        mean /= (float)k;
        if (best < 0.f || mean < best) {
          best = mean;
          pick = b->tune;
        }
      }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  b->source = source;
  b->tune = rc ? keep : pick;
  if (rc) {
    set_error("autotune: timing failed");
    return rc;
  }
  if (chosen) {
    chosen[0] = pick.alpha;
    chosen[1] = pick.beta;
    chosen[2] = (float)pick.large_row;
    chosen[3] = best;
  }
  return bfs_recompute(b);
}

int bfs_set_accounting(Bfs* b, int on) {
  if (on && !b->acct && cudaMalloc(&b->acct, 8 * sizeof(unsigned long long)) != cudaSuccess) {
    set_error("accounting counter allocation failed");
    return -4;
  }
  if (on) VX_CUDA_TRY(cudaMemsetAsync(b->acct, 0, 8 * sizeof(unsigned long long), b->g->stream));
  b->acct_on = on != 0;
  return 0;
}

int bfs_accounting(Bfs* b, unsigned long long* out5) {
  memset(out5, 0, 5 * sizeof(unsigned long long));
  if (!b->acct) return 0;
  VX_CUDA_TRY(cudaMemcpyAsync(out5, b->acct, 5 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, b->g->stream));
  VX_CUDA_TRY(cudaStreamSynchronize(b->g->stream));
  return 0;
}

static int raw_shift(size_t n) {  // bits of an op's index and its add flag
  int sh = 2;
  while (((size_t)1 << (sh - 1)) < n) ++sh;
  return sh;
}

static int raw_bits(size_t V) {  // bits of a vertex id below max(V, 2)
  int b = 1;
  while (((size_t)1 << b) < V) ++b;
  return b;
}

int bfs_stage(Bfs* b, size_t n, size_t vertex_bound, bool classify) {
  Graph* g = b->g;
  cudaStream_t s = g->stream;
  b->staged_ops = n;
  b->staged_V_pre = g->V;
  b->staged_len_pre = b->dist_len;
  if (n == 0) {  // last_* counters reset on every apply (bfs.hpp:30-33)
    VX_CUDA_TRY(cudaMemsetAsync(&b->ctr->candidates, 0, 4 * sizeof(uint32_t), s));
    return 0;
  }
  // a non-empty batch resets them (and the repair lists) in whichever path
  // consumes it: the fused launch in its first phase, the per-phase and full
  // paths on the host before their kernels
  b->staged_classified = classify;
  b->staged_raw = false;
  if (!classify && n <= kRawOps) {  // keys of two ids, an op's index, its add flag and the direction
    if (int rc = graph_prepare_batch(g, n, vertex_bound)) return rc;
    b->staged_raw = 2 * raw_bits(g->V) + raw_shift(n) <= 62;
  }
  if (!b->staged_raw)
    if (int rc = graph_stage_batch(g, n, vertex_bound, classify)) return rc;
  if (int rc = ensure_capacity(b, std::max<size_t>(g->V, 1))) return rc;
  return ensure_ring(b);
}

static int launch_stream(Bfs* b, Params& p, StreamArgs& sa) {
  if (!b->stream_grid) {
    int per_sm = 0;
    VX_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bfs_stream_kernel, kThreads, 0));
    if (per_sm < 1) {
      set_error("stream kernel cannot be resident on an SM");
      return -3;
    }
    b->stream_grid = per_sm * sm_count();
  }
  // one block per SM by default: against two per SM (every co-resident
  // block) the grid barriers and the work ring's polling are cheaper, and the
  // update step measured 13% faster at R-MAT 22 and R-MAT 20
  const uint32_t want = b->tune.update_blocks ? b->tune.update_blocks : (uint32_t)sm_count();
  p.nblocks = std::min(std::min(want, (uint32_t)b->stream_grid), kRawBlocks);
  p.deltas = 1;  // the launch inserts delta rows itself
  if (b->lists_left) {  // the update launch starts from empty repair lists and leaves them empty
    VX_CUDA_TRY(cudaMemsetAsync(&b->ctr->cand_n, 0, 3 * sizeof(uint32_t), b->g->stream));
    VX_CUDA_TRY(cudaMemsetAsync(&b->ctr->fallback, 0, sizeof(uint32_t), b->g->stream));
    b->lists_left = false;
  }
  void* args[] = {&p, &sa};
  count_launch();
  VX_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)bfs_stream_kernel, dim3(p.nblocks), dim3(kThreads), args,
                                          0, b->g->stream));
  return 0;
}

// The staged batch as a one-batch stream: tombstones, delta removals, the
// cascade, delta insertions and the post-batch repair in one persistent launch
// (a directed graph's two adjacencies one after the other within each pass).  A
// directed 1,000-op batch at 300,000 vertices took some 22 launches and 213 us;
// now one and 73.
static int repair_fused(Bfs* b) {
  Graph* g = b->g;
  const size_t n = b->staged_ops, m = g->directed ? n : 2 * n;
  StreamArgs sa;
  memset(&sa, 0, sizeof(sa));
  sa.fu[0] = g->batch.fu;
  sa.fv[0] = g->batch.fv;
  sa.ff[0] = g->batch.ff;
  sa.fpos[0] = g->batch.fpos;
  sa.cnt[0] = &g->ctr->final_arcs;
  sa.scratch[0] = g->batch.lu;
  sa.gc = g->ctr;
  sa.arena_cap[0] = g->adj[0].arena_cap;
  if (g->directed) {
    sa.fu[1] = g->batch.ru;
    sa.fv[1] = g->batch.rv;
    sa.ff[1] = g->batch.rf;
    sa.fpos[1] = g->batch.rpos;
    sa.cnt[1] = &g->ctr->rev_arcs;
    sa.scratch[1] = g->batch.lv;
    sa.arena_cap[1] = g->adj[1].arena_cap;
  }
  sa.frac = b->frac;
  sa.nb = 1;
  sa.V0 = (uint32_t)b->staged_V_pre;
  sa.len0 = (uint32_t)b->staged_len_pre;
  sa.v_single = (uint32_t)g->V;
  sa.classified = b->staged_classified ? 1u : 0u;
  if (b->staged_raw) {
    sa.over = g->batch.flag;  // the staging's, unused here
    sa.raw_src = g->batch.in_src;
    sa.raw_dst = g->batch.in_dst;
    sa.raw_add = g->batch.in_add;
    sa.raw_n = (uint32_t)n;
    sa.raw_b = (uint32_t)raw_bits(g->V);
    sa.raw_sh = (uint32_t)raw_shift(n);
    sa.raw_bound = (uint32_t)g->V;
    b->staged_raw = false;
  }
  Params p = make_params(b, (uint32_t)g->V, (uint32_t)g->V);
  if (int rc = launch_stream(b, p, sa)) return rc;
  for (int d = 0; d < (g->directed ? 2 : 1); ++d) g->adj[d].arena_bound += 8ull * m + 8;  // what the staging reserved
  ++g->version;
  b->dist_len = std::max<size_t>(b->dist_len, g->V);
  b->staged_ops = 0;
  return 0;
}

int bfs_repair_staged(Bfs* b) {
  Graph* g = b->g;
  cudaStream_t s = g->stream;
  if (b->staged_ops == 0) return 0;
  // a directed batch that was classified when it was staged has no reversed list
  if (b->tune.fused && !(g->directed && b->staged_classified)) return repair_fused(b);
  VX_CUDA_TRY(cudaMemsetAsync(&b->ctr->candidates, 0, 4 * sizeof(uint32_t), s));
  VX_CUDA_TRY(cudaMemsetAsync(&b->ctr->cand_n, 0, 3 * sizeof(uint32_t), s));
  VX_CUDA_TRY(cudaMemsetAsync(b->ctr->rtrace, 0, sizeof(b->ctr->rtrace), s));
  VX_CUDA_TRY(cudaMemsetAsync(b->ctr->handovers, 0, sizeof(b->ctr->handovers), s));
  const size_t V_pre = b->staged_V_pre, len_pre = b->staged_len_pre;
  const size_t V_post = g->V;
  b->lists_left = true;
  // fallback limit: max(1, size_t(double(V) * fraction))  (bfs.hpp:225-226)
  unsigned long long lim = (unsigned long long)((double)V_pre * b->frac);
  if (lim < 1) lim = 1;
  // The fixpoint reads the pre-batch graph without the batch's deletions
  // (exactly the arcs the reference's support count and child propagation
  // exclude), so removals are committed first and insertions after it.
  if (int rc = graph_commit_removals(g)) return rc;
  {
    Params p = make_params(b, (uint32_t)V_pre, (uint32_t)len_pre);
    p.fallback_limit = lim;
    if (len_pre > 0)
      if (int rc = launch(b, p, kModePre)) return rc;
  }
  if (int rc = graph_commit_insertions(g)) return rc;
  if (b->dist_len < V_post) {
    VX_CUDA_TRY(cudaMemsetAsync(b->dist + b->dist_len, 0xFF, (V_post - b->dist_len) * 4, s));
    b->dist_len = V_post;
  }
  b->staged_ops = 0;
  Params p = make_params(b, (uint32_t)V_post, (uint32_t)b->dist_len);
  p.fallback_limit = lim;
  return launch(b, p, kModePost);
}

int bfs_full_staged(Bfs* b) {
  if (b->staged_ops == 0) return 0;
  if (int rc = graph_commit_batch(b->g)) return rc;
  b->staged_ops = 0;
  VX_CUDA_TRY(cudaMemsetAsync(b->ctr->rtrace, 0, sizeof(b->ctr->rtrace), b->g->stream));
  VX_CUDA_TRY(cudaMemsetAsync(b->ctr->handovers, 0, sizeof(b->ctr->handovers), b->g->stream));
  return bfs_recompute(b);
}

int bfs_apply_staged(Bfs* b, size_t n, size_t vertex_bound) {
  // the fused repair classifies the arcs itself; the per-phase path needs them classified
  const bool fused = b->tune.fused;
  if (int rc = bfs_stage(b, n, vertex_bound, !fused)) return rc;
  return bfs_repair_staged(b);
}

int bfs_sync(Bfs* b) {
  cudaStream_t s = b->g->stream;
  VX_CUDA_TRY(cudaMemcpyAsync(b->hctr, b->ctr, sizeof(BfsCounters), cudaMemcpyDeviceToHost, s));
  VX_CUDA_TRY(cudaStreamSynchronize(s));
  if (b->hctr->err) {
    set_error("BFS device error word 0x%x", b->hctr->err);
    return -5;
  }
  return 0;
}

int bfs_reached_arcs(Bfs* b, unsigned long long* arcs) {
  cudaStream_t s = b->g->stream;
  unsigned long long* d = &b->ctr->scratch64;
  VX_CUDA_TRY(cudaMemsetAsync(d, 0, 8, s));
  vxh::count_launch();
  reached_arcs_kernel<<<sm_count() * 8, 256, 0, s>>>(b->g->view().out, b->dist, (uint32_t)b->dist_len, d);
  VX_CUDA_TRY(cudaGetLastError());
  VX_CUDA_TRY(cudaMemcpyAsync(b->g->pinned_scalar, d, 8, cudaMemcpyDeviceToHost, s));
  VX_CUDA_TRY(cudaStreamSynchronize(s));
  *arcs = b->g->pinned_scalar[0];
  return 0;
}

}  // namespace vxh

namespace vxh {
int bfs_level_trace(Bfs* b, unsigned long long* out, size_t cap, size_t* n) {
  if (int rc = bfs_sync(b)) return rc;
  const uint32_t levels = std::min<uint32_t>(b->hctr->levels, kTraceLevels - 1);
  *n = 2 * ((size_t)levels + 1);
  const size_t m = std::min(cap, *n);
  if (out && m) VX_CUDA_TRY(cudaMemcpy(out, b->trace, m * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
  return 0;
}

int bfs_phase_trace(Bfs* b, unsigned long long* out, size_t cap, size_t* n) {
  if (int rc = bfs_sync(b)) return rc;
  constexpr size_t kR = sizeof(b->hctr->rtrace) / sizeof(b->hctr->rtrace[0]);
  constexpr size_t kS = sizeof(b->hctr->stream_ns) / sizeof(b->hctr->stream_ns[0]);
  constexpr size_t kH = sizeof(b->hctr->handovers) / sizeof(b->hctr->handovers[0]);
  *n = kR + kS + kH;
  for (size_t i = 0; i < std::min(cap, kR); ++i) out[i] = b->hctr->rtrace[i];
  for (size_t i = kR; i < std::min(cap, kR + kS); ++i) out[i] = b->hctr->stream_ns[i - kR];
  for (size_t i = kR + kS; i < std::min(cap, kR + kS + kH); ++i) out[i] = b->hctr->handovers[i - kR - kS];
  return 0;
}

// ------------------------------------------------------- batched stream --

void StreamBufs::free_all() {
  void* ptrs[] = {src, dst, add, off, keys, keys_alt, vals, vals_alt, flag, pos, fu, fv, bid, ff, fpos,
                  boff, bcnt, vpost, total, scratch, digest, bstats};
  for (void* q : ptrs) cudaFree(q);
  *this = StreamBufs();
}

int StreamBufs::ensure(size_t n, size_t nb, size_t maxf) {
  if (n <= ops_cap && nb <= nb_cap && maxf <= maxf_cap) return 0;
  const size_t N = std::max(n, ops_cap), B = std::max(nb, nb_cap), MF = std::max(maxf, maxf_cap);
  free_all();
  const size_t m = 2 * std::max<size_t>(N, 1);
  bool ok = true;
  auto al = [&](auto** q, size_t count, size_t size) {
    if (ok && cudaMalloc((void**)q, std::max<size_t>(count, 1) * size) != cudaSuccess) ok = false;
  };
  al(&src, N, 4);
  al(&dst, N, 4);
  al(&add, N, 1);
  al(&off, B + 1, 8);
  al(&keys, m, 8);
  al(&keys_alt, m, 8);
  al(&vals, m, 4);
  al(&vals_alt, m, 4);
  al(&flag, m, 4);
  al(&pos, m, 4);
  al(&fu, m, 4);
  al(&fv, m, 4);
  al(&bid, m, 4);
  al(&ff, m, 1);
  al(&fpos, m, 8);
  al(&boff, B + 1, 4);
  al(&bcnt, B, 4);
  al(&vpost, B, 4);
  al(&total, 1, 4);
  al(&scratch, MF, 4);
  al(&digest, B, 8);
  al(&bstats, 4 * B, 4);
  if (!ok) {
    free_all();
    set_error("stream buffer allocation failed");
    return -4;
  }
  ops_cap = N;
  nb_cap = B;
  maxf_cap = MF;
  return 0;
}

int bfs_apply_stream(Bfs* b, const uint32_t* hs, const uint32_t* hd, const uint8_t* ha, const uint64_t* hoff,
                     size_t nb, uint64_t* digests, uint32_t* stats, size_t* applied) {
  Graph* g = b->g;
  cudaStream_t st = g->stream;
  *applied = 0;
  if (nb == 0) return 0;
  if (hoff[0] != 0) {
    set_error("batch offsets must start at 0");
    return -1;
  }
  const size_t n = hoff[nb];
  const size_t Vbefore = g->V;
  // vertex count after every batch (the graph grows to max id + 1 over the
  // non-self-loop ops, dynamic_graph.hpp:717-733) and the arena bound
  std::vector<uint32_t> vpost(nb);
  size_t V = g->V, maxf = 1;
  uint64_t bound = 0;
  size_t nonempty = 0;
  for (size_t t = 0; t < nb; ++t) {
    if (hoff[t + 1] < hoff[t]) {
      set_error("batch offsets must not decrease");
      return -1;
    }
    for (uint64_t i = hoff[t]; i < hoff[t + 1]; ++i)
      if (hs[i] != hd[i]) V = std::max<size_t>(V, (size_t)std::max(hs[i], hd[i]) + 1);
    if (V > vxb::kMaxVertices) {
      set_error("vertex id beyond the supported maximum (2^31 - 1)");
      return -2;
    }
    vpost[t] = (uint32_t)V;
    const size_t m = 2 * (size_t)(hoff[t + 1] - hoff[t]);
    if (m) {
      bound += 8ull * m + 8;
      ++nonempty;
    }
    maxf = std::max(maxf, m);
  }
  int bbits = 1;
  while (bbits < 32 && ((size_t)1 << bbits) < std::max<size_t>(V, 2)) ++bbits;
  int tbits = 1;
  while (tbits < 40 && ((size_t)1 << tbits) < nb) ++tbits;
  const uint32_t window = std::min<uint32_t>(b->tune.stream_window, kMaxVersions);
  if (!stats && window && !g->directed && nb >= 2 && 2 * bbits + 8 <= 64 && n < (1ull << 31)) {
    // every batch but the last in version-parallel windows
    StreamBufs& S = b->sb;
    if (int rc = S.ensure(n, nb, maxf)) return rc;
    VX_CUDA_TRY(cudaMemcpyAsync(S.src, hs, n * 4, cudaMemcpyHostToDevice, st));
    VX_CUDA_TRY(cudaMemcpyAsync(S.dst, hd, n * 4, cudaMemcpyHostToDevice, st));
    VX_CUDA_TRY(cudaMemcpyAsync(S.add, ha, n, cudaMemcpyHostToDevice, st));
    // every window's buffers up front, so that no window allocates
    size_t wops = 0;
    for (size_t t0 = 0; t0 + 1 < nb; t0 += window)
      wops = std::max<size_t>(wops, hoff[std::min<size_t>(t0 + window, nb - 1)] - hoff[t0]);
    if (int rc = stream_versions_reserve(b, wops, std::max<size_t>(b->dist_len, vpost[nb - 2]),
                                         std::min<size_t>(window, nb - 1)))
      return rc;
    for (size_t t0 = 0; t0 + 1 < nb; t0 += window) {
      const size_t t1 = std::min<size_t>(t0 + window, nb - 1);
      if (int rc = stream_versions(b, S.src, S.dst, S.add, hoff, vpost.data(), t0, t1, digests)) return rc;
      *applied = t1;
    }
    const uint64_t tail[2] = {0, hoff[nb] - hoff[nb - 1]};
    const uint64_t lo = hoff[nb - 1];
    size_t last = 0;
    if (int rc = bfs_apply_stream(b, hs + lo, hd + lo, ha + lo, tail, 1, digests ? digests + nb - 1 : nullptr,
                                  nullptr, &last))
      return rc;
    *applied += last;
    return 0;
  }
  // the persistent path covers undirected graphs whose (batch, u, v) keys fit
  // 64 bits and whose arena takes the whole stream; the caller loops otherwise
  if (g->directed || 2 * bbits + tbits > 64 || n >= (1ull << 31)) return 0;
  int fits = 0;
  if (int rc = graph_reserve_stream(g, bound, &fits)) return rc;
  if (!fits) return 0;
  if (int rc = graph_grow(g, V)) return rc;
  const uint32_t len0 = (uint32_t)b->dist_len;
  if (int rc = ensure_capacity(b, std::max<size_t>(V, 1))) return rc;
  Adjacency& a = g->adj[0];
  a.arena_bound += bound;
  if (int rc = ensure_ring(b)) return rc;
  StreamBufs& S = b->sb;
  if (int rc = S.ensure(n, nb, maxf)) return rc;
  VX_CUDA_TRY(cudaMemcpyAsync(S.src, hs, n * 4, cudaMemcpyHostToDevice, st));
  VX_CUDA_TRY(cudaMemcpyAsync(S.dst, hd, n * 4, cudaMemcpyHostToDevice, st));
  VX_CUDA_TRY(cudaMemcpyAsync(S.add, ha, n, cudaMemcpyHostToDevice, st));
  VX_CUDA_TRY(cudaMemcpyAsync(S.off, hoff, (nb + 1) * 8, cudaMemcpyHostToDevice, st));
  VX_CUDA_TRY(cudaMemcpyAsync(S.vpost, vpost.data(), nb * 4, cudaMemcpyHostToDevice, st));
  const size_t m = 2 * n;
  const unsigned grid_n = (unsigned)std::max<size_t>(1, std::min<size_t>((n + 255) / 256, (size_t)sm_count() * 32));
  const unsigned grid_m = (unsigned)std::max<size_t>(1, std::min<size_t>((m + 255) / 256, (size_t)sm_count() * 32));
  count_launch();
  stream_keys_kernel<<<grid_n, 256, 0, st>>>(S.src, S.dst, S.add, S.off, (uint32_t)nb, n, bbits, S.keys, S.vals);
  VX_CUDA_TRY(cudaGetLastError());
  bool in_alt = false;
  if (int rc = radix_sort_u64(S.keys, S.keys_alt, S.vals, S.vals_alt, m, 2 * bbits + tbits, &in_alt, g->scratch, g->sort_wait(), st))
    return rc;
  uint64_t* keys = in_alt ? S.keys_alt : S.keys;
  uint32_t* vals = in_alt ? S.vals_alt : S.vals;
  count_launch();
  stream_last_kernel<<<grid_m, 256, 0, st>>>(keys, m, &g->ctr->err, S.flag);
  if (int rc = scan_exclusive_u32(S.flag, S.pos, m, S.total, g->scratch, st)) return rc;
  count_launch();
  stream_compact_kernel<<<grid_m, 256, 0, st>>>(keys, vals, S.flag, S.pos, m, bbits, S.fu, S.fv, S.ff, S.bid);
  count_launch();
  stream_bounds_kernel<<<(unsigned)((nb + 256) / 256), 256, 0, st>>>(S.bid, S.total, (uint32_t)nb, S.boff, S.bcnt);
  VX_CUDA_TRY(cudaGetLastError());
  if (digests) VX_CUDA_TRY(cudaMemsetAsync(S.digest, 0, nb * 8, st));
  StreamArgs sa;
  memset(&sa, 0, sizeof(sa));
  sa.fu[0] = S.fu;
  sa.fv[0] = S.fv;
  sa.ff[0] = S.ff;
  sa.fpos[0] = S.fpos;
  sa.boff = S.boff;
  sa.cnt[0] = S.bcnt;
  sa.vpost = S.vpost;
  sa.scratch[0] = S.scratch;
  sa.digest = digests ? S.digest : nullptr;
  sa.bstats = stats ? S.bstats : nullptr;
  sa.gc = g->ctr;
  sa.arena_cap[0] = a.arena_cap;
  sa.frac = b->frac;
  sa.nb = (uint32_t)nb;
  sa.V0 = (uint32_t)Vbefore;
  sa.len0 = len0;
  Params p = make_params(b, (uint32_t)V, (uint32_t)V);
  if (int rc = launch_stream(b, p, sa)) return rc;
  g->version += nonempty;
  b->dist_len = V;
  b->staged_ops = 0;
  if (digests) VX_CUDA_TRY(cudaMemcpyAsync(digests, S.digest, nb * 8, cudaMemcpyDeviceToHost, st));
  if (stats) VX_CUDA_TRY(cudaMemcpyAsync(stats, S.bstats, nb * 16, cudaMemcpyDeviceToHost, st));
  *applied = nb;
  return digests || stats ? bfs_sync(b) : 0;
}

int bfs_digest(Bfs* b, uint64_t* out) {
  cudaStream_t st = b->g->stream;
  unsigned long long* d = &b->ctr->scratch64;
  VX_CUDA_TRY(cudaMemsetAsync(d, 0, 8, st));
  if (b->dist_len) {
    count_launch();
    digest_kernel<<<sm_count() * 8, 256, 0, st>>>(b->dist, (uint32_t)b->dist_len, d);
    VX_CUDA_TRY(cudaGetLastError());
  }
  VX_CUDA_TRY(cudaMemcpyAsync(b->g->pinned_scalar, d, 8, cudaMemcpyDeviceToHost, st));
  VX_CUDA_TRY(cudaStreamSynchronize(st));
  *out = b->g->pinned_scalar[0];
  return 0;
}
}  // namespace vxh

// ------------------------------------------------ allocation-free full BFS --
//
// Some callers cannot call cudaMalloc: a host framework that owns the whole
// device memory through its own pool (and forbids raw driver allocations),
// or a latency-critical serving loop that must never block on the driver's
// allocator after start-up.  vx_bfs_csr_static serves them: it runs the same
// direction-optimising BFS kernel as recompute() on a CSR the caller already
// holds in device memory, writing distances into the caller's buffer, and
// keeps every other buffer (visited and frontier bitmaps, frontier queues,
// counters, barrier words) in one file-scope
// device array.  It allocates nothing.
//
// Limits and sharing: at most kStaticMaxVertices vertices; every GPU that
// loads this library holds the array (about 6.5 MB) until the process exits;
// all calls share it and it keeps the last call's contents, so calls that
// overlap on the GPU (different streams, different threads) race -- issue
// them one at a time per device.  The first call on a device looks up the
// array's device address for that device; make that first call before any
// stream capture.
namespace vxh {
namespace {

constexpr uint32_t kStaticMaxVertices = 1u << 18;  // 262,144
constexpr uint32_t kStaticWords = kStaticMaxVertices / 32 + 1;

struct StaticBfsScratch {
  uint32_t vis[kStaticWords];
  uint32_t fb[3][kStaticWords];
  uint32_t q[3][kStaticMaxVertices];
  uint32_t big[kStaticMaxVertices];
  uint32_t bul[2 * list_slots(kStaticMaxVertices)];  // the bottom-up candidate lists
  BfsCounters ctr;
  uint32_t bar[vxb::kBarrierWords];
};

}  // namespace
}  // namespace vxh

static __device__ __align__(256) unsigned char vx_static_bfs_scratch[sizeof(vxh::StaticBfsScratch)];

namespace {
constexpr int kStaticMaxDevices = 64;
// device address of the array, per device; two host threads making their
// first call on one device at once both look it up and store the same value
std::atomic<void*> g_static_scratch_addr[kStaticMaxDevices];
}  // namespace

extern "C" int vx_bfs_csr_static(const uint64_t* d_out_offsets, const uint32_t* d_out_cols,
                                 const uint64_t* d_in_offsets, const uint32_t* d_in_cols, uint32_t vertices,
                                 uint64_t arcs, uint32_t source, uint32_t* d_dist, void* stream,
                                 uint64_t* reachable) {
  using vxh::StaticBfsScratch;
  if (!d_out_offsets || !d_out_cols || !d_in_offsets || !d_in_cols || !d_dist) {
    vxh::set_error("vx_bfs_csr_static: null argument");
    return -1;
  }
  if (vertices == 0 || vertices > vxh::kStaticMaxVertices) {
    vxh::set_error("vx_bfs_csr_static: %u vertices; the static scratch holds 1..%u", vertices,
                   vxh::kStaticMaxVertices);
    return -2;
  }
  int dev = 0;
  VX_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kStaticMaxDevices) {
    vxh::set_error("vx_bfs_csr_static: device %d beyond the supported %d", dev, kStaticMaxDevices);
    return -2;
  }
  void* addr = g_static_scratch_addr[dev].load(std::memory_order_acquire);
  if (!addr) {
    // one-time set-up on this device (the device is current here)
    const cudaError_t e = cudaGetSymbolAddress(&addr, vx_static_bfs_scratch);
    if (e != cudaSuccess || !addr) {
      vxh::set_error("vx_bfs_csr_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return -3;
    }
    g_static_scratch_addr[dev].store(addr, std::memory_order_release);
  }
  StaticBfsScratch* sc = static_cast<StaticBfsScratch*>(addr);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // what must start at zero: counters, barrier words (a plain CSR has no delta rows to read)
  VX_CUDA_TRY(cudaMemsetAsync(&sc->ctr, 0, sizeof(vxh::BfsCounters), s));
  VX_CUDA_TRY(cudaMemsetAsync(sc->bar, 0, sizeof(sc->bar), s));
  vxh::Params p;
  memset(&p, 0, sizeof(p));
  auto adj = [&](const uint64_t* off, const uint32_t* col) {
    vxb::DevAdj a;
    memset(&a, 0, sizeof(a));
    a.off = off;
    a.col = const_cast<uint32_t*>(col);
    a.Vb = vertices;
    return a;
  };
  p.g.out = adj(d_out_offsets, d_out_cols);
  p.g.in = adj(d_in_offsets, d_in_cols);
  p.g.V = vertices;
  p.g.directed = d_in_offsets != d_out_offsets || d_in_cols != d_out_cols;
  p.V = vertices;
  p.dist_len = vertices;
  p.source = source;
  p.dist = d_dist;
  p.vis = sc->vis;
  for (int k = 0; k < 3; ++k) {
    p.fb[k] = sc->fb[k];
    p.q[k] = sc->q[k];
  }
  p.big = sc->big;
  p.bul = sc->bul;
  p.bul_half = (uint32_t)vxh::list_slots(vxh::kStaticMaxVertices);
  p.c = &sc->ctr;
  p.total_arcs = arcs;
  p.alpha = 14.0f;
  p.beta = 24.0f;
  p.large_row = 1024;
  p.bar = sc->bar;
  if (int rc = vxh::launch_full(p, s)) return rc;
  uint32_t err = 0;
  unsigned long long reach = 0;
  VX_CUDA_TRY(cudaMemcpyAsync(&err, &sc->ctr.err, sizeof(err), cudaMemcpyDeviceToHost, s));
  VX_CUDA_TRY(cudaMemcpyAsync(&reach, &sc->ctr.reachable, sizeof(reach), cudaMemcpyDeviceToHost, s));
  VX_CUDA_TRY(cudaStreamSynchronize(s));
  if (err) {
    vxh::set_error("vx_bfs_csr_static: device error word 0x%x", err);
    return -5;
  }
  if (reachable) *reachable = reach;
  return 0;
}
