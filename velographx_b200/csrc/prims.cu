// Stable LSD radix sort and exclusive scans (see prims.cuh).
//
// Radix sort: 8-bit digits.  n <= kSmallN runs as one CTA that keeps the whole
// array in shared memory for every pass.  Larger inputs read the keys once for
// the digit counts of all passes, then run one kernel per pass: a tile ranks
// its items, publishes its digit counts, adds up those of the tiles before it
// (the decoupled look-back of Merrill and Garland, "Single-pass parallel prefix
// scan with decoupled look-back", 2016) and writes its items in digit order, so
// that each digit's run of the tile goes out coalesced.  Stability inside a
// tile comes from ranking items in position order: warp w owns consecutive
// positions, and lanes inside a warp are ranked with __match_any_sync.
#include <algorithm>

#include "prims.cuh"
#include "vx_common.cuh"

namespace vxh {

namespace {

constexpr int kDigits = 256;

// ------------------------------------------------------------------ scan --

constexpr int kScanBlock = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanBlock * kScanItems;

template <typename T>
__device__ T block_exclusive_scan(T v, T* warp_tot, T* block_total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    T w = lane < (kScanBlock / 32) ? warp_tot[lane] : T(0);
    T wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < (kScanBlock / 32)) warp_tot[lane] = wi - w;
    if (lane == (kScanBlock / 32) - 1) *block_total = wi;
  }
  __syncthreads();
  return incl - v + warp_tot[warp];
}

template <typename In, typename Out>
__global__ void __launch_bounds__(kScanBlock) scan_reduce_kernel(const In* in, size_t n, Out* partial) {
  __shared__ Out red[kScanBlock / 32];
  const size_t base = (size_t)blockIdx.x * kScanTile;
  Out s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const size_t idx = base + (size_t)i * kScanBlock + threadIdx.x;
    if (idx < n) s += (Out)in[idx];
  }
  s = vxb::warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    Out t = 0;
    for (int w = 0; w < kScanBlock / 32; ++w) t += red[w];
    partial[blockIdx.x] = t;
  }
}

// Exclusive scan of one tile plus an optional per-tile offset.
template <typename In, typename Out>
__global__ void __launch_bounds__(kScanBlock) scan_tile_kernel(const In* in, Out* out, size_t n,
                                                               const Out* tile_offset, Out* total) {
  __shared__ Out buf[kScanTile];
  __shared__ Out warp_tot[32];
  __shared__ Out btot;
  const size_t base = (size_t)blockIdx.x * kScanTile;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const int j = i * kScanBlock + threadIdx.x;
    const size_t idx = base + j;
    buf[j] = idx < n ? (Out)in[idx] : Out(0);
  }
  __syncthreads();
  Out local[kScanItems];
  Out s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    local[i] = buf[threadIdx.x * kScanItems + i];
    s += local[i];
  }
  const Out off = tile_offset ? tile_offset[blockIdx.x] : Out(0);
  Out run = block_exclusive_scan<Out>(s, warp_tot, &btot) + off;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    buf[threadIdx.x * kScanItems + i] = run;
    run += local[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const int j = i * kScanBlock + threadIdx.x;
    const size_t idx = base + j;
    if (idx < n) out[idx] = buf[j];
  }
  if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = off + btot;
}

size_t scan_levels_bytes(size_t n, size_t elem) {
  size_t bytes = 0;
  while (n > (size_t)kScanTile) {
    n = (n + kScanTile - 1) / kScanTile;
    bytes += ((n * elem + 255) / 256) * 256;
  }
  return bytes + 256;
}

template <typename In, typename Out>
int scan_impl(const In* in, Out* out, size_t n, Out* total, char* scratch, cudaStream_t s) {
  if (n == 0) {
    if (total) VX_CUDA_TRY(cudaMemsetAsync(total, 0, sizeof(Out), s));
    return 0;
  }
  const size_t nblk = (n + kScanTile - 1) / kScanTile;
  if (nblk == 1) {
    vxh::count_launch();
    scan_tile_kernel<In, Out><<<1, kScanBlock, 0, s>>>(in, out, n, nullptr, total);
    VX_CUDA_TRY(cudaGetLastError());
    return 0;
  }
  Out* partial = reinterpret_cast<Out*>(scratch);
  char* rest = scratch + ((nblk * sizeof(Out) + 255) / 256) * 256;
  vxh::count_launch();
  scan_reduce_kernel<In, Out><<<(unsigned)nblk, kScanBlock, 0, s>>>(in, n, partial);
  VX_CUDA_TRY(cudaGetLastError());
  int rc = scan_impl<Out, Out>(partial, partial, nblk, nullptr, rest, s);
  if (rc) return rc;
  vxh::count_launch();
  scan_tile_kernel<In, Out><<<(unsigned)nblk, kScanBlock, 0, s>>>(in, out, n, partial, total);
  VX_CUDA_TRY(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------------ radix sort --

constexpr int kSmallBlock = 1024;
constexpr int kSmallItems = 8;
constexpr size_t kSmallN = (size_t)kSmallBlock * kSmallItems;
constexpr int kBigBlock = 256;
constexpr int kBigItems = 16;
constexpr int kBigTile = kBigBlock * kBigItems;

__device__ __forceinline__ uint32_t digit_of(uint64_t k, int shift) {
  return (uint32_t)(k >> shift) & 0xFFu;
}

// Stable block-wide digit ranking with warp-private histograms.
//
// Warp w owns the ITEMS*32 consecutive tile positions starting at
// w*ITEMS*32; round r of the warp holds positions w*ITEMS*32 + r*32 + lane.
// Each warp ranks its own items in position order (match_any peers + a
// private 256-bin histogram, no block barrier), then one pass over the
// histograms gives every warp its per-digit offset.  The returned rank of an
// item is its position among equal digits of the tile (earlier warps, earlier
// rounds, lower lanes first), and digit_total[d] the tile's count of digit d.
template <int BLOCK, int ITEMS>
__device__ void rank_tile(const uint32_t (&d)[ITEMS], uint32_t (&rank)[ITEMS], uint32_t* warp_hist /*[W][256]*/,
                          uint32_t* digit_total /*[256]*/) {
  constexpr int W = BLOCK / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* h = warp_hist + warp * kDigits;
  for (int i = lane; i < kDigits; i += 32) h[i] = 0;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d[r]);
    const uint32_t base = h[d[r]];
    __syncwarp();
    if (lane == __ffs(peers) - 1) h[d[r]] = base + __popc(peers);
    __syncwarp();
    rank[r] = base + __popc(peers & vxb::lanemask_lt());
  }
  __syncthreads();
  for (int dd = threadIdx.x; dd < kDigits; dd += BLOCK) {
    uint32_t s = 0;
#pragma unroll 4
    for (int w = 0; w < W; ++w) {
      const uint32_t c = warp_hist[w * kDigits + dd];
      warp_hist[w * kDigits + dd] = s;
      s += c;
    }
    digit_total[dd] = s;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) rank[r] += h[d[r]];
}

// Whole sort inside one CTA.  Shared layout: keys[kSmallN] u64, vals[kSmallN]
// u32, warp_hist[32*256], digit_total[256], digit_base[256].
__global__ void __launch_bounds__(kSmallBlock) small_sort_kernel(uint64_t* keys, uint32_t* vals, size_t n,
                                                                  int passes) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t* sk = reinterpret_cast<uint64_t*>(smem);
  uint32_t* sv = reinterpret_cast<uint32_t*>(sk + kSmallN);
  uint32_t* warp_hist = sv + kSmallN;
  uint32_t* total = warp_hist + (kSmallBlock / 32) * kDigits;
  uint32_t* dbase = total + kDigits;
  for (size_t i = threadIdx.x; i < kSmallN; i += kSmallBlock) {
    sk[i] = i < n ? keys[i] : ~0ull;
    if (vals) sv[i] = i < n ? vals[i] : 0u;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pos0 = warp * kSmallItems * 32 + lane;
  for (int p = 0; p < passes; ++p) {
    const int shift = p * 8;
    uint64_t k[kSmallItems];
    uint32_t v[kSmallItems], d[kSmallItems], rank[kSmallItems];
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
      k[r] = sk[pos0 + r * 32];
      v[r] = vals ? sv[pos0 + r * 32] : 0u;
      d[r] = digit_of(k[r], shift);
    }
    rank_tile<kSmallBlock, kSmallItems>(d, rank, warp_hist, total);
    if (threadIdx.x < 32) {
      // exclusive scan of the 256 digit totals by one warp (8 per lane)
      uint32_t loc[8], run = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        loc[j] = total[threadIdx.x * 8 + j];
        run += loc[j];
      }
      uint32_t incl = run;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (threadIdx.x >= o) incl += y;
      }
      uint32_t ex = incl - run;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        dbase[threadIdx.x * 8 + j] = ex;
        ex += loc[j];
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
      const uint32_t dst = dbase[d[r]] + rank[r];
      sk[dst] = k[r];
      if (vals) sv[dst] = v[r];
    }
    __syncthreads();
  }
  for (size_t i = threadIdx.x; i < n; i += kSmallBlock) {
    keys[i] = sk[i];
    if (vals) vals[i] = sv[i];
  }
}

constexpr size_t kSmallSmem =
    kSmallN * 8 + kSmallN * 4 + (kSmallBlock / 32) * kDigits * 4 + kDigits * 4 * 2;
static_assert(kSmallSmem <= 227 * 1024, "small sort exceeds shared memory");

// Digit counts of every pass, counts[pass][digit]: one read of the keys.  Four
// copies of each counter by lane: the upper digits of a skewed graph's ids are
// mostly equal, and equal addresses of a warp are added one after another.
constexpr int kCopies = 4;
__global__ void __launch_bounds__(kBigBlock) radix_count_kernel(const uint64_t* keys, size_t n, int passes,
                                                                unsigned long long* counts) {
  __shared__ uint32_t h[8 * kDigits * kCopies];
  for (int i = threadIdx.x; i < passes * kDigits * kCopies; i += kBigBlock) h[i] = 0;
  __syncthreads();
  const uint32_t copy = threadIdx.x % kCopies;
  const size_t step = (size_t)gridDim.x * kBigBlock;
  size_t i = (size_t)blockIdx.x * kBigBlock + threadIdx.x;
  for (; i + 3 * step < n; i += 4 * step) {
    uint64_t k[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) k[j] = keys[i + j * step];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      for (int p = 0; p < passes; ++p) atomicAdd(&h[(p * kDigits + digit_of(k[j], 8 * p)) * kCopies + copy], 1u);
  }
  for (; i < n; i += step) {
    const uint64_t k = keys[i];
    for (int p = 0; p < passes; ++p) atomicAdd(&h[(p * kDigits + digit_of(k, 8 * p)) * kCopies + copy], 1u);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < passes * kDigits; j += kBigBlock) {
    uint32_t c = 0;
#pragma unroll
    for (int q = 0; q < kCopies; ++q) c += h[j * kCopies + q];
    if (c) atomicAdd(&counts[j], (unsigned long long)c);
  }
}

// counts[pass][digit] -> first position of the digit; one block per pass.
__global__ void __launch_bounds__(kDigits) radix_bases_kernel(unsigned long long* counts) {
  __shared__ unsigned long long warp_tot[32], total;
  unsigned long long* c = counts + (size_t)blockIdx.x * kDigits;
  static_assert(kDigits == kScanBlock, "one digit per thread of the block scan");
  const unsigned long long v = c[threadIdx.x];
  c[threadIdx.x] = block_exclusive_scan<unsigned long long>(v, warp_tot, &total);
}

// A tile's word for one digit: its count, or the count of it and all tiles
// before it, once published.
constexpr unsigned long long kTileSum = 1ull << 62, kTilePrefix = 2ull << 62, kTileMask = (1ull << 62) - 1;
constexpr uint32_t kLookBack = 8;  // words of earlier tiles in flight per look

// One pass.  Tiles take their numbers from a ticket, so every tile before a
// running one is running or done, and the look-back ends.  33.5M keys: 358 us a
// pass against 548 for the counts, scans and an unstaged scatter of a pass before
// (537 MB would take 82: with 444 tiles in flight the look-back is the chain);
// 200,000 keys with values: 15 us against 33.  4, 16 or 32 words in flight: no
// faster (the words themselves are L2 traffic).
__global__ void __launch_bounds__(kBigBlock, 3) radix_pass_kernel(const uint64_t* keys, const uint32_t* vals,
                                                               uint64_t* keys_out, uint32_t* vals_out, size_t n,
                                                               int shift, const unsigned long long* bases,
                                                               unsigned long long* state, uint32_t* ticket,
                                                               SortWait wait) {
  __shared__ __align__(16) uint64_t stage[kBigTile];
  __shared__ uint32_t warp_hist[(kBigBlock / 32) * kDigits];
  __shared__ uint32_t total[kDigits];
  __shared__ uint32_t first[kDigits];           // the digit's first place in the tile
  __shared__ unsigned long long gbase[kDigits];  // its first place in the output, less that
  __shared__ uint32_t warp_tot[32], tsum, tile_s;
  static_assert(kDigits == kBigBlock, "a thread per digit");
  const uint32_t t = threadIdx.x;
  if (t == 0) tile_s = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint32_t tile = tile_s;
  const int lane = t & 31, warp = t >> 5;
  const size_t lo = (size_t)tile * kBigTile;
  const uint32_t m = (uint32_t)(n - lo < (size_t)kBigTile ? n - lo : (size_t)kBigTile);
  const uint32_t pos0 = warp * kBigItems * 32 + lane;
  uint64_t k[kBigItems];
  uint32_t d[kBigItems], rank[kBigItems];
#pragma unroll
  for (int r = 0; r < kBigItems; ++r) k[r] = pos0 + r * 32 < m ? keys[lo + pos0 + r * 32] : ~0ull;
#pragma unroll
  for (int r = 0; r < kBigItems; ++r) d[r] = pos0 + r * 32 < m ? digit_of(k[r], shift) : kDigits - 1u;
  rank_tile<kBigBlock, kBigItems>(d, rank, warp_hist, total);  // padding ranks behind every item of its digit
  const uint32_t mine = total[t] - (t == kDigits - 1 ? kBigTile - m : 0u);
  unsigned long long* word = state + (size_t)tile * kDigits + t;
  if (tile > 0) __stcg(word, kTileSum | mine);
  else __stcg(word, kTilePrefix | mine);
  first[t] = block_exclusive_scan<uint32_t>(total[t], warp_tot, &tsum);
  __syncthreads();
  // the keys wait in shared memory, so the look-back has their registers
#pragma unroll
  for (int r = 0; r < kBigItems; ++r) {
    rank[r] += first[d[r]];
    stage[rank[r]] = k[r];
  }
  unsigned long long before = 0;
  if (tile > 0) {
    uint32_t idle = 0;  // looks since the last word that was there
    for (int64_t j = (int64_t)tile - 1; j >= 0;) {
      if (idle++ == wait.looks) {
        atomicOr(wait.err, vxb::kErrBarrierTimeout);
        break;
      }
      unsigned long long w[kLookBack];
#pragma unroll
      for (uint32_t q = 0; q < kLookBack; ++q)
        w[q] = j >= (int64_t)q ? __ldcg(state + (size_t)(j - q) * kDigits + t) : kTilePrefix;
      bool done = false, stuck = false;
#pragma unroll
      for (uint32_t q = 0; q < kLookBack; ++q) {
        if (done || stuck) continue;
        stuck = (w[q] & ~kTileMask) == 0ull;
        if (stuck) continue;
        before += w[q] & kTileMask;
        done = (w[q] & kTilePrefix) != 0ull;
        --j;
        idle = 0;
      }
      if (done) break;
    }
    __stcg(word, kTilePrefix | (before + mine));
  }
  gbase[t] = bases[t] + before - first[t];
  __syncthreads();
  uint32_t dst[kBigItems];  // counts of arcs fit 32 bits throughout
#pragma unroll
  for (int r = 0; r < kBigItems; ++r) {
    const uint32_t i = r * kBigBlock + t;
    if (i < m) {
      const uint64_t key = stage[i];
      dst[r] = (uint32_t)(gbase[digit_of(key, shift)] + i);
      if (dst[r] < n) keys_out[dst[r]] = key;  // out of range only after a wait gave up
    }
  }
  if (!vals) return;
  __syncthreads();
  uint32_t* vstage = reinterpret_cast<uint32_t*>(stage);
#pragma unroll
  for (int r = 0; r < kBigItems; ++r)
    if (pos0 + r * 32 < m) vstage[rank[r]] = vals[lo + pos0 + r * 32];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kBigItems; ++r) {
    const uint32_t i = r * kBigBlock + t;
    if (i < m && dst[r] < n) vals_out[dst[r]] = vstage[i];
  }
}

}  // namespace

int Scratch::ensure(size_t bytes) {
  if (bytes <= cap) return 0;
  release();
  size_t c = bytes < (1u << 20) ? (1u << 20) : bytes + bytes / 4;
  if (cudaMalloc(&ptr, c) != cudaSuccess) {
    ptr = nullptr;
    cap = 0;
    set_error("scratch allocation of %zu bytes failed", c);
    return -4;
  }
  cap = c;
  return 0;
}

void Scratch::release() {
  if (ptr) cudaFree(ptr);
  ptr = nullptr;
  cap = 0;
}

int sm_count() {
  static int cached = 0;
  if (!cached) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev);
    if (cached <= 0) cached = 148;
  }
  return cached;
}

size_t scan_scratch_bytes(size_t n) { return scan_levels_bytes(n, 8) + 512; }

int scan_exclusive_u32_to_u64(const uint32_t* in, uint64_t* out, size_t n, uint64_t* total_dev,
                              Scratch& scratch, cudaStream_t s) {
  if (int rc = scratch.ensure(scan_scratch_bytes(n))) return rc;
  return scan_impl<uint32_t, uint64_t>(in, out, n, total_dev, static_cast<char*>(scratch.ptr), s);
}

int scan_exclusive_u32(const uint32_t* in, uint32_t* out, size_t n, uint32_t* total_dev, Scratch& scratch,
                       cudaStream_t s) {
  if (int rc = scratch.ensure(scan_scratch_bytes(n))) return rc;
  return scan_impl<uint32_t, uint32_t>(in, out, n, total_dev, static_cast<char*>(scratch.ptr), s);
}

// [8][256] digit counts, one ticket per pass, then one state word per tile and
// digit for each pass (cleared together).
constexpr size_t kSortHead = 8 * kDigits * 8 + 256;

size_t radix_sort_scratch_bytes(size_t n) {
  const size_t tiles = (n + kBigTile - 1) / kBigTile;
  return kSortHead + tiles * kDigits * 8 + 512;
}

int radix_sort_u64(uint64_t* keys, uint64_t* keys_alt, uint32_t* vals, uint32_t* vals_alt, size_t n,
                   int key_bits, bool* in_alt, Scratch& scratch, const SortWait& wait, cudaStream_t s) {
  *in_alt = false;
  if (n <= 1) return 0;
  if (key_bits < 1) key_bits = 1;
  if (key_bits > 64) key_bits = 64;
  const int passes = (key_bits + 7) / 8;
  if (n <= kSmallN) {
    static bool attr_set = false;
    if (!attr_set) {
      VX_CUDA_TRY(cudaFuncSetAttribute(small_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kSmallSmem));
      attr_set = true;
    }
    vxh::count_launch();
    small_sort_kernel<<<1, kSmallBlock, kSmallSmem, s>>>(keys, vals, n, passes);
    VX_CUDA_TRY(cudaGetLastError());
    return 0;
  }
  if (int rc = scratch.ensure(radix_sort_scratch_bytes(n))) return rc;
  const uint32_t tiles = (uint32_t)((n + kBigTile - 1) / kBigTile);
  unsigned long long* counts = static_cast<unsigned long long*>(scratch.ptr);
  uint32_t* tickets = reinterpret_cast<uint32_t*>(counts + 8 * kDigits);
  unsigned long long* state = reinterpret_cast<unsigned long long*>(static_cast<char*>(scratch.ptr) + kSortHead);
  VX_CUDA_TRY(cudaMemsetAsync(scratch.ptr, 0, kSortHead, s));
  vxh::count_launch();
  radix_count_kernel<<<std::min<uint32_t>(tiles, (uint32_t)sm_count() * 4), kBigBlock, 0, s>>>(keys, n, passes, counts);
  vxh::count_launch();
  radix_bases_kernel<<<passes, kDigits, 0, s>>>(counts);
  VX_CUDA_TRY(cudaGetLastError());
  uint64_t *ki = keys, *ko = keys_alt;
  uint32_t *vi = vals, *vo = vals_alt;
  for (int p = 0; p < passes; ++p) {
    const int shift = p * 8;
    VX_CUDA_TRY(cudaMemsetAsync(state, 0, (size_t)tiles * kDigits * 8, s));
    vxh::count_launch();
    radix_pass_kernel<<<tiles, kBigBlock, 0, s>>>(ki, vi, ko, vo, n, shift, counts + p * kDigits, state, tickets + p,
                                                  wait);
    VX_CUDA_TRY(cudaGetLastError());
    uint64_t* tk = ki;
    ki = ko;
    ko = tk;
    uint32_t* tv = vi;
    vi = vo;
    vo = tv;
  }
  *in_alt = (passes & 1) != 0;
  return 0;
}

}  // namespace vxh
