// Device building blocks shared by the single-root and multi-root BFS
// kernels: grid-stride indices, row expansion (flattened small rows,
// warp-walked medium rows), a block-aggregated frontier queue, timers.
#pragma once

#include <cstdint>

#include "vx_common.cuh"

namespace vxh {
namespace frontier {

using vxb::DevAdj;
using vxb::kIdMask;
using vxb::kTomb;
using vxb::kUnreachable;

__device__ __forceinline__ uint32_t ld_cg(const uint32_t* p) { return __ldcg(p); }

__device__ __forceinline__ uint32_t gtid() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint32_t nthreads() { return gridDim.x * blockDim.x; }
__device__ __forceinline__ uint32_t gwarp() { return gtid() >> 5; }
__device__ __forceinline__ uint32_t nwarps() { return nthreads() >> 5; }

__device__ __forceinline__ bool test_bit(const uint32_t* bm, uint32_t v) { return (bm[v >> 5] >> (v & 31)) & 1u; }

__device__ __forceinline__ uint32_t degree_of(const DevAdj& a, uint32_t u) {
  uint64_t b, e;
  vxb::base_range(a, u, b, e);
  return (uint32_t)(e - b) + a.drow[u].y;
}

// The W per-vertex words at base (W = 1, 2, 4 or 8 consecutive words, base
// aligned to 4 * W bytes), one vector load per 16 bytes.
template <uint32_t W>
__device__ __forceinline__ void load_words(const uint32_t* base, uint32_t* out) {
  if constexpr (W == 1) {
    out[0] = base[0];
  } else if constexpr (W == 2) {
    const uint2 t = *reinterpret_cast<const uint2*>(base);
    out[0] = t.x;
    out[1] = t.y;
  } else {
#pragma unroll
    for (uint32_t h = 0; h < W / 4; ++h) {
      const uint4 t = reinterpret_cast<const uint4*>(base)[h];
      out[4 * h] = t.x;
      out[4 * h + 1] = t.y;
      out[4 * h + 2] = t.z;
      out[4 * h + 3] = t.w;
    }
  }
}

// The listed rows (lengths len[0, n)) of which this warp holds a slice, when
// every row is cut into slices of `slice` arcs and the slices of all rows, in
// list order, are dealt to the warps in turn: f(r, len_r, first slice) for
// each, warp-uniformly; the warp's further slices of the row follow nwarps()
// apart.  The lengths are read 32 at a time, so a warp passes the rows it has
// no slice of without a round trip per row.  (With the slices of row r dealt
// from warp r on, the few hub rows of a small frontier all lay on the same
// warps: 55 rows with 478,438 arcs 286 us, so 21 us.)
template <class F>
__device__ __forceinline__ void for_my_rows(const uint32_t* len, uint32_t n, uint32_t slice, F&& f) {
  const uint32_t lane = threadIdx.x & 31, nw = nwarps(), gw = gwarp();
  uint32_t first = 0;  // slices of the rows before r0, mod the warp count
  for (uint32_t r0 = 0; r0 < n; r0 += 32) {
    const uint32_t r = r0 + lane;
    const uint32_t l = r < n ? __ldcg(&len[r]) : 0u;
    const uint32_t sl = (l + slice - 1) / slice;
    uint32_t incl = sl;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= d) incl += t;
    }
    const uint32_t s0 = (gw + nw - (first + incl - sl) % nw) % nw;
    first = (first + __shfl_sync(0xFFFFFFFFu, incl, 31)) % nw;
    uint32_t mine = __ballot_sync(0xFFFFFFFFu, s0 < sl);
    while (mine) {
      const uint32_t k = __ffs(mine) - 1;
      mine &= mine - 1;
      f(r0 + k, __shfl_sync(0xFFFFFFFFu, l, k), __shfl_sync(0xFFFFFFFFu, s0, k));
    }
  }
}

// --------------------------------------------------- row expansion core --

constexpr uint32_t FULL = 0xFFFFFFFFu;

// The 32-vertex groups that a warp takes of a pull level: the first by its number,
// further ones from one counter (zero before the level), one at a time where its last
// group was a heavy one (arcs to read past the rows' heads, or much to write), else
// kClaimGroups.  Claims serialise on the counter, which shows where a level does little
// beside them: one root in a star of 2^20 vertices, two pull levels, 136 us a run with
// single claims, 112 so, 104 with claims of four.  Those leave the grid waiting for a
// warp with several heavy groups: 64 roots in a graph of 2^20 vertices and 2^21 edges
// 574, 593 and 702 us.
constexpr uint32_t kClaimGroups = 2;
struct GroupClaims {
  // warp-uniform; numbered across the blocks first, as a skewed graph's heavy groups
  // may lie side by side
  uint32_t cur = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, end = cur + 1;
  bool heavy = false;  // the last group was (set by the caller)
  // The next group, or one at or past the level's last when there are no more; whole warp.
  __device__ __forceinline__ uint32_t next(uint32_t* counter) {
    if (cur == end) {
      const uint32_t n = heavy ? 1u : kClaimGroups;
      uint32_t c = 0;
      if ((threadIdx.x & 31) == 0) c = nwarps() + atomicAdd(counter, n);
      cur = __shfl_sync(FULL, c, 0);
      end = cur + n;
    }
    return cur++;
  }
};

// The whole warp walks one row (all lanes pass the same u); f as above.
template <class F>
__device__ __forceinline__ void warp_row(const DevAdj& a, uint32_t u, F& f) {
  const int lane = threadIdx.x & 31;
  uint64_t b, e;
  vxb::base_range(a, u, b, e);
  for (uint64_t j0 = b; j0 < e; j0 += 32) {
    const uint64_t j = j0 + lane;
    const uint32_t x = j < e ? a.col[j] : kTomb;
    f(!(x & kTomb), x & kIdMask, u);
  }
  const uint2 dr = a.drow[u];
  for (uint32_t j0 = dr.x; j0 < dr.x + dr.y; j0 += 32) {
    const uint32_t j = j0 + lane;
    const bool ok = j < dr.x + dr.y;
    f(ok, ok ? a.darena[j] : 0u, u);
  }
}

__device__ __forceinline__ uint64_t globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Block-aggregated frontier queue: warps reserve slots in shared memory
// (shared atomics); the block flushes with one global atomic per phase.  Warps
// that find the buffer full append straight to the global queue.
constexpr uint32_t kBlockQueueCap = 2048;
template <uint32_t kCap>
struct BlockQueueOf {
  uint32_t cnt;
  uint32_t gbase;
  uint32_t items[kCap];
};
using BlockQueue = BlockQueueOf<kBlockQueueCap>;

// gbase0: the global counter's value that corresponds to gq[0] (a counter
// that is not reset between uses, as the bottom-up candidate lists use).
template <uint32_t kCap>
__device__ __forceinline__ void bq_push(BlockQueueOf<kCap>& bq, bool pred, uint32_t v, uint32_t* gcnt, uint32_t* gq,
                                        uint32_t gbase0 = 0u) {
  const uint32_t mask = __ballot_sync(FULL, pred);
  if (!mask) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  const uint32_t n = __popc(mask);
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(&bq.cnt, n);
  base = __shfl_sync(FULL, base, leader);
  const uint32_t r = __popc(mask & vxb::lanemask_lt());
  const uint32_t spill = base + n > kCap ? base + n - max(base, kCap) : 0u;
  uint32_t gb = 0;
  if (spill && lane == leader) gb = atomicAdd(gcnt, spill);
  gb = __shfl_sync(FULL, gb, leader);
  if (pred) {
    const uint32_t slot = base + r;
    if (slot < kCap) bq.items[slot] = v;
    else gq[(gb - gbase0) + (slot - max(base, kCap))] = v;
  }
}

// The lanes' entries v[j] where bit `lane` of mask[j] is set (masks are
// warp-uniform), one reservation for all of them.
template <int N, uint32_t kCap>
__device__ __forceinline__ void bq_push_n(BlockQueueOf<kCap>& bq, const uint32_t (&mask)[N], const uint32_t (&v)[N],
                                          uint32_t* gcnt, uint32_t* gq) {
  uint32_t n = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) n += __popc(mask[j]);
  if (!n) return;
  const int lane = threadIdx.x & 31;
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(&bq.cnt, n);
  base = __shfl_sync(FULL, base, 0);
  const uint32_t first = max(base, kCap);  // slots from here on overflow to the global queue
  uint32_t gb = 0;
  if (base + n > first) {
    if (lane == 0) gb = atomicAdd(gcnt, base + n - first);
    gb = __shfl_sync(FULL, gb, 0);
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if ((mask[j] >> lane) & 1u) {
      const uint32_t slot = base + __popc(mask[j] & vxb::lanemask_lt());
      if (slot < kCap) bq.items[slot] = v[j];
      else gq[gb + (slot - first)] = v[j];
    }
    base += __popc(mask[j]);
  }
}

// Block-uniform: moves the buffered entries to the global queue.
template <uint32_t kCap>
__device__ __forceinline__ void bq_flush(BlockQueueOf<kCap>& bq, uint32_t* gcnt, uint32_t* gq, uint32_t gbase0 = 0u) {
  __syncthreads();
  const uint32_t n = min(bq.cnt, kCap);
  if (threadIdx.x == 0) bq.gbase = n ? atomicAdd(gcnt, n) : 0u;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) gq[(bq.gbase - gbase0) + i] = bq.items[i];
  __syncthreads();
  if (threadIdx.x == 0) bq.cnt = 0;
  __syncthreads();
}

}  // namespace frontier
}  // namespace vxh
