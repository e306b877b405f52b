// pbf_sort.cu — integer pipeline of the neighbour search: single-pass
// decoupled look-back exclusive scan, counting-sort scatter, stable
// within-cell order by particle id, the stable LSD radix sort of the
// stand-alone search, the state moved along with the order, id-order export
// and the per-step metrics reduction.
//
// Reference counterparts (relative to the reference root):
//   ExclusiveScan.execute + scanShader.ts  src/simulator/neighbor/exclusiveScan.ts:134-166,
//                                          src/simulator/neighbor/scanShader.ts:16-107
//   ParticleInsert / CountingSort          src/simulator/neighbor/neighborShader.ts:24-60
// The reference's within-cell order is the order its atomicAdd calls happened
// to return; here it is defined as particle-id order (the sequential
// semantics), which the sort below reproduces exactly whatever order the
// warp-aggregated atomics ran in.
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/pbf_gb300.h"
#include "pbf_device.cuh"
#include "pbf_kernels.h"

namespace pbf {

namespace {
constexpr uint32_t kFull = 0xffffffffu;
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048 elements per tile
static_assert(kScanTile == (int)kScanTileElements, "scan tile size");
constexpr uint32_t kFlagAggregate = 1u, kFlagPrefix = 2u;
constexpr uint32_t kSpinLimit = 1u << 22;             // ~ tens of ms at worst, then give up

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long pack(uint32_t flag, uint32_t value) {
  return ((unsigned long long)flag << 32) | value;
}

// Block-wide exclusive scan of one value per thread; returns the block total in *total.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* total, uint32_t* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    uint32_t w = (lane < nw) ? warp_sums[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(kFull, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) warp_sums[lane] = w;  // inclusive warp prefix
  }
  __syncthreads();
  uint32_t warp_excl = (warp == 0) ? 0u : warp_sums[warp - 1];
  *total = warp_sums[(blockDim.x >> 5) - 1];
  return warp_excl + x - v;
}

// Single-pass scan: tiles take ids from a counter in launch order, publish
// their aggregate, look back over predecessors (bounded waits) and publish
// the inclusive prefix.  Status words pack (flag << 32 | value).  Along the
// way X.zero (n entries) is cleared, X.in_copy receives the first in_copy_n
// inputs and X.out_copy the result, each where given.
__global__ void __launch_bounds__(kScanThreads) k_scan(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                       size_t n, unsigned long long* status, uint32_t* counter,
                                                       uint32_t* err, ScanExtra X) {
  chain_begin(in);
  __shared__ uint32_t s_items[kScanTile + kScanTile / 32];
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_prefix;
  if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const size_t base = (size_t)tile * kScanTile;
  // striped coalesced load, padded transpose to blocked order
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int li = k * kScanThreads + threadIdx.x;
    size_t gi = base + li;
    const uint32_t v = (gi < n) ? __ldg(in + gi) : 0u;
    s_items[li + (li >> 5)] = v;
    if (X.zero && gi < n) X.zero[gi] = 0u;
    if (X.in_copy && gi < X.in_copy_n) X.in_copy[gi] = v;
  }
  __syncthreads();
  uint32_t items[kScanItems];
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int li = threadIdx.x * kScanItems + k;
    items[k] = s_items[li + (li >> 5)];
    sum += items[k];
  }
  uint32_t total;
  uint32_t texcl = block_exclusive(sum, &total, s_warp);
  // look-back
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    uint32_t prefix = 0;
    if (tile == 0) {
      if (lane == 0) st_release_u64(status + 0, pack(kFlagPrefix, total));
    } else {
      if (lane == 0) st_release_u64(status + tile, pack(kFlagAggregate, total));
      long pred = (long)tile - 1;
      bool done = false;
      while (!done) {
        long idx = pred - lane;
        unsigned long long w = pack(kFlagPrefix, 0);  // lanes past tile 0 read as an empty prefix
        uint32_t spins = 0;
        if (idx >= 0) {
          w = ld_acquire_u64(status + idx);
          while ((uint32_t)(w >> 32) == 0u) {
            if (++spins > kSpinLimit) {
              atomicOr(err, (uint32_t)PBF_DEVERR_SCAN_TIMEOUT);
              w = pack(kFlagPrefix, 0);
              break;
            }
            __nanosleep(32);
            w = ld_acquire_u64(status + idx);
          }
        }
        uint32_t flag = (uint32_t)(w >> 32), val = (uint32_t)w;
        uint32_t pmask = __ballot_sync(kFull, flag == kFlagPrefix);
        // lanes up to (and including) the nearest prefix contribute
        int stop = pmask ? (__ffs(pmask) - 1) : 31;
        uint32_t contrib = (lane <= stop) ? val : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(kFull, contrib, o);
        prefix += contrib;
        if (pmask) done = true;
        pred -= 32;
      }
      if (lane == 0) st_release_u64(status + tile, pack(kFlagPrefix, prefix + total));
    }
    if (lane == 0) s_prefix = prefix;
  }
  __syncthreads();
  uint32_t run = s_prefix + texcl;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int li = threadIdx.x * kScanItems + k;
    s_items[li + (li >> 5)] = run;
    run += items[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int li = k * kScanThreads + threadIdx.x;
    size_t gi = base + li;
    if (gi < n) {
      out[gi] = s_items[li + (li >> 5)];
      if (X.out_copy) X.out_copy[gi] = s_items[li + (li >> 5)];
    }
  }
}

// ---- counting-sort scatter (CountingSort, neighborShader.ts:49-60) -----------------
__global__ void __launch_bounds__(256) k_scatter(uint32_t n, const uint32_t* __restrict__ key,
                                                 const uint32_t* __restrict__ rank, const uint32_t* __restrict__ cell_start,
                                                 const uint32_t* __restrict__ ids, uint32_t* __restrict__ perm_raw,
                                                 uint32_t* __restrict__ id_raw) {
  chain_begin(key, rank, cell_start, ids);
  uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  uint32_t k = key[s];
  uint32_t dst = __ldg(cell_start + k) + rank[s];
  perm_raw[dst] = s;
  id_raw[dst] = ids ? __ldg(ids + s) : s;
}

// ---- stable within-cell order and the state in the new order ------------------------
// Moves the state of input slot s (particle id) to sorted slot d.
template <bool kCb>
__device__ __forceinline__ void place_state(const GatherArgs& G, uint32_t d, uint32_t s, uint32_t id) {
  G.pos_out[d] = __ldg(G.pos_in + s);
  const float4 x = __ldg(G.xs_in + s);
  G.xs_out[d] = x;
  G.id_out[d] = id;
  if constexpr (kCb) {
    G.xs0_out[d] = x;
    G.skey_out[d] = __ldg(G.key + s);
  }
  if (G.f_in) G.f_out[d] = __ldg(G.f_in + s);
}

// One thread per sorted position q: the entry scattered there ranks itself
// by particle id among its cell's entries and moves to cell_start + rank,
// with its state (the cell is a few consecutive slots, so the stores of a warp
// stay together; a gather of its own would read the order back).  The work
// follows the particles (sum over cells of count^2), not the cell count, so
// empty cells cost nothing.  Cells above kRankMax entries go to the block
// radix path (the thread at the cell's first position lists it).
constexpr uint32_t kRankMax = 1024;

template <bool kCb>
__global__ void __launch_bounds__(256) k_cellfix(uint32_t n, const uint32_t* __restrict__ key,
                                                 const uint32_t* __restrict__ cell_count,
                                                 const uint32_t* __restrict__ cell_start,
                                                 const uint32_t* __restrict__ perm_raw,
                                                 const uint32_t* __restrict__ id_raw, uint32_t* __restrict__ perm,
                                                 uint32_t* big_list, uint32_t* big_count, GatherArgs G) {
  chain_begin(key, cell_count, cell_start, perm_raw, id_raw, G.pos_in, G.xs_in, G.key, G.f_in);
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const uint32_t s = perm_raw[q], my = id_raw[q];
  const uint32_t c = __ldg(key + s);
  const uint32_t cnt = __ldg(cell_count + c), st = __ldg(cell_start + c);
  if (cnt > kRankMax) {
    if (q == st) big_list[atomicAdd(big_count, 1u)] = c;
    return;
  }
  uint32_t r = 0;
  if (cnt > 1)
    for (uint32_t m = 0; m < cnt; ++m) r += (__ldg(id_raw + st + m) < my) ? 1u : 0u;
  perm[st + r] = s;
  place_state<kCb>(G, st + r, s, my);
}

// Block LSD radix sort (8-bit digits) of one very full cell by particle id;
// stable because tiles are processed in order and ranks within a tile follow
// thread order.
constexpr int kRadixThreads = 256;
template <bool kCb>
__global__ void __launch_bounds__(kRadixThreads) k_bigcell(const uint32_t* __restrict__ big_list,
                                                           const uint32_t* __restrict__ big_count,
                                                           const uint32_t* __restrict__ cell_count,
                                                           const uint32_t* __restrict__ cell_start,
                                                           uint32_t* __restrict__ perm_raw, uint32_t* __restrict__ id_raw,
                                                           uint32_t* __restrict__ perm, uint32_t* __restrict__ tmp_slot,
                                                           uint32_t* __restrict__ tmp_id, int passes, GatherArgs G) {
  chain_begin(big_list, big_count, cell_count, cell_start, G.pos_in, G.xs_in, G.key, G.f_in);
  __shared__ uint32_t s_base[256];
  __shared__ uint32_t s_wcount[kRadixThreads / 32][256];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t nb = *big_count;
  for (uint32_t bi = blockIdx.x; bi < nb; bi += gridDim.x) {
    const uint32_t c = big_list[bi];
    const uint32_t cnt = cell_count[c], st = cell_start[c];
    // ping-pong between the cell's own segments of (perm_raw, id_raw) and (tmp_slot, tmp_id);
    // the last pass writes the slots straight into perm.
    uint32_t* src_slot = perm_raw + st;
    uint32_t* src_id = id_raw + st;
    for (int pass = 0; pass < passes; ++pass) {
      const int shift = 8 * pass;
      const bool even = (pass & 1) == 0;
      uint32_t* dst_slot = (even ? tmp_slot : perm_raw) + st;
      uint32_t* dst_id = (even ? tmp_id : id_raw) + st;
      if (pass == passes - 1) dst_slot = perm + st;
      // histogram
      for (int d = tid; d < 256; d += kRadixThreads) s_base[d] = 0;
      __syncthreads();
      for (uint32_t e = tid; e < cnt; e += kRadixThreads) atomicAdd(&s_base[(src_id[e] >> shift) & 255u], 1u);
      __syncthreads();
      if (tid == 0) {
        uint32_t run = 0;
        for (int d = 0; d < 256; ++d) {
          uint32_t v = s_base[d];
          s_base[d] = run;
          run += v;
        }
      }
      __syncthreads();
      for (uint32_t t0 = 0; t0 < cnt; t0 += kRadixThreads) {
        for (int q = tid; q < (kRadixThreads / 32) * 256; q += kRadixThreads) (&s_wcount[0][0])[q] = 0;
        __syncthreads();
        uint32_t e = t0 + tid;
        bool valid = e < cnt;
        uint32_t d = valid ? ((src_id[e] >> shift) & 255u) : 256u;
        uint32_t peers = __match_any_sync(kFull, d);
        uint32_t lrank = __popc(peers & ((1u << lane) - 1u));
        if (valid && lrank == 0) s_wcount[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
          uint32_t r = s_base[d] + lrank;
          for (int w = 0; w < warp; ++w) r += s_wcount[w][d];
          dst_slot[r] = src_slot[e];
          dst_id[r] = src_id[e];
        }
        __syncthreads();
        for (int dd = tid; dd < 256; dd += kRadixThreads) {
          uint32_t add = 0;
          for (int w = 0; w < kRadixThreads / 32; ++w) add += s_wcount[w][dd];
          s_base[dd] += add;
        }
        __syncthreads();
      }
      src_slot = dst_slot;
      src_id = dst_id;
      __syncthreads();
    }
    for (uint32_t e = tid; e < cnt; e += kRadixThreads) place_state<kCb>(G, st + e, src_slot[e], src_id[e]);
    __syncthreads();
  }
}

// ---- stable LSD radix sort by cell key of points in particle-id order ---------------
// The stand-alone search receives its points in id order, so a stable sort
// of the ids by cell key yields the order with every cell's particles in id
// order: no within-cell pass, and skewed cell occupancy costs nothing extra.
// Each pass over a digit is reduce-then-scan: every tile of 3072 records
// counts its digits (written digit-major, count[d * tiles + tile]); one
// exclusive scan of that matrix gives each (digit, tile) run its global
// place; then every tile ranks its records by digit in shared memory (stable
// in input order) and writes each digit's run there.  Reads and writes are
// coalesced, and no tile waits on another.  The first pass's counts come from
// the kernel that computes the keys.  Up to kFewTiles tiles the scan is a
// launch for a few thousand words: every tile then adds up the counts it needs
// itself, and the previous pass counts the next one's digits where it writes
// its records (their place says their tile), so a pass is one kernel.
constexpr int kOsThreads = 256;
constexpr int kOsItems = 12;
constexpr int kOsTile = kOsThreads * kOsItems;  // 3072 records per tile
constexpr int kOsWarps = kOsThreads / 32;
constexpr int kOsMaxRadix = 256;

// Lanes of the warp holding the same digit (valid lanes only): one ballot per
// digit bit.
template <int kWidth>
__device__ __forceinline__ unsigned digit_peers(uint32_t d, bool valid) {
  unsigned peers = __ballot_sync(kFull, valid);
#pragma unroll
  for (int b = 0; b < kWidth; ++b) {
    const unsigned m = __ballot_sync(kFull, (d >> b) & 1u);
    peers &= ((d >> b) & 1u) ? m : ~m;
  }
  return peers;
}

// Adds 1 to count[key] for each valid lane (the first ones of the warp): one
// addition per run of equal keys.
__device__ __forceinline__ void add_runs(uint32_t* count, uint32_t key, uint32_t lane, bool valid) {
  const uint32_t up = __shfl_up_sync(kFull, key, 1);
  const bool start = valid && (lane == 0u || up != key);
  const unsigned starts = __ballot_sync(kFull, start);
  const unsigned valid_mask = __ballot_sync(kFull, valid);
  if (start) {
    const unsigned later = starts & ~((2u << lane) - 1u);
    const uint32_t end = later ? (uint32_t)(__ffs(later) - 1) : (uint32_t)(32 - __clz(valid_mask));
    atomicAdd(count + key, end - lane);
  }
}

// Up to this many tiles (98,304 points) the passes work from the counts
// themselves.  A tile reads tiles x 2^width words for it; at 32 tiles that is
// less than a launch of the scan, at 64 about the same.
constexpr uint32_t kFewTiles = 32;
// ... and from this many on a warp adds its records to the next pass's counts
// in runs.  Records of a crowd have the same next digit in the same tile, and
// additions to one word wait for each other: 98,304 points in one cell of 100^3
// 151 us without runs, 53 with (110 with three launches a pass), 73,728 126 and
// 51 (101).  Runs cost an even cloud 1 us: 5,003 points 22.5 and 23.5 us, 85,000
// 28.5 and 30.0.
constexpr uint32_t kRunTiles = 20;

// Cell key of every point (ParticleInsert) and the first pass's digit counts
// of each tile (per-warp counters in shared memory, summed at the end).  The
// grid may be larger than the tiles: every CTA clears its share of the
// scratch of the kernels that follow.
template <int kWidth>
__global__ void __launch_bounds__(kOsThreads) k_keys_digits(GridParams g, const float4* __restrict__ pos, uint32_t n,
                                                            uint32_t* __restrict__ key, uint32_t* __restrict__ count,
                                                            uint32_t tiles, ClearRanges clear) {
  constexpr uint32_t kRadix = 1u << kWidth, kMask = kRadix - 1u;
  __shared__ uint32_t s_cnt[kOsWarps][kRadix];
  chain_begin(pos);
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  for (uint32_t d = tid; d < kOsWarps * kRadix; d += kOsThreads) (&s_cnt[0][0])[d] = 0u;
#pragma unroll
  for (int r = 0; r < ClearRanges::kRanges; ++r)
    for (size_t i = (size_t)blockIdx.x * kOsThreads + tid; i < clear.words[r]; i += (size_t)gridDim.x * kOsThreads)
      clear.p[r][i] = 0u;
  if (blockIdx.x >= tiles) return;
  const uint32_t t0 = blockIdx.x * (uint32_t)kOsTile;
  uint32_t d[kOsItems];
#pragma unroll
  for (int i = 0; i < kOsItems; ++i) {
    const uint32_t idx = t0 + (uint32_t)i * kOsThreads + tid;
    d[i] = kRadix;
    if (idx < n) {
      const float4 x = __ldg(pos + idx);
      const int cx = cell_axis(x.x, g.origin[0], g.inv_cell[0], g.dim[0]);
      const int cy = cell_axis(x.y, g.origin[1], g.inv_cell[1], g.dim[1]);
      const int cz = cell_axis(x.z, g.origin[2], g.inv_cell[2], g.dim[2]);
      const uint32_t k = cell_key(cx, cy, cz, g);
      key[idx] = k;
      d[i] = k & kMask;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kOsItems; ++i)
    if (d[i] < kRadix) atomicAdd(&s_cnt[warp][d[i]], 1u);
  __syncthreads();
  for (uint32_t dd = tid; dd < kRadix; dd += kOsThreads) {
    uint32_t c = 0;
#pragma unroll
    for (int w = 0; w < kOsWarps; ++w) c += s_cnt[w][dd];
    count[(size_t)dd * tiles + blockIdx.x] = c;
  }
}

// Digit counts of one tile, digit-major (per-warp counters in shared memory,
// summed at the end).
template <int kWidth>
__global__ void __launch_bounds__(kOsThreads) k_tile_digits(uint32_t n, const uint32_t* __restrict__ kin,
                                                            uint32_t* __restrict__ count, uint32_t tiles, int shift) {
  chain_begin(kin);
  constexpr uint32_t kRadix = 1u << kWidth, kMask = kRadix - 1u;
  __shared__ uint32_t s_cnt[kOsWarps][kRadix];
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  for (uint32_t d = tid; d < kOsWarps * kRadix; d += kOsThreads) (&s_cnt[0][0])[d] = 0u;
  const uint32_t t0 = blockIdx.x * (uint32_t)kOsTile;
  uint32_t d[kOsItems];
#pragma unroll
  for (int i = 0; i < kOsItems; ++i) {
    const uint32_t idx = t0 + (uint32_t)i * kOsThreads + tid;
    d[i] = idx < n ? (__ldg(kin + idx) >> shift) & kMask : kRadix;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kOsItems; ++i)
    if (d[i] < kRadix) atomicAdd(&s_cnt[warp][d[i]], 1u);
  __syncthreads();
  for (uint32_t dd = tid; dd < kRadix; dd += kOsThreads) {
    uint32_t c = 0;
#pragma unroll
    for (int w = 0; w < kOsWarps; ++w) c += s_cnt[w][dd];
    count[(size_t)dd * tiles + blockIdx.x] = c;
  }
}

// One pass over the digit (key >> shift) & (2^kWidth - 1): place[d * tiles +
// tile] is where the tile's run of digit d starts.  vin == nullptr: the values
// are the input positions (particle ids).  cell_count (the last pass only):
// the written keys are in final order, so each run of equal keys a warp
// writes is added to its cell's count once; vout2 (optional) receives the
// values too.  kFew: place holds the tiles' digit counts instead (at most
// kFewTiles tiles), and next_count (optional, cleared) receives those of the
// next pass, added up in runs with kRuns.
template <int kWidth, bool kFew, bool kRuns>
__global__ void __launch_bounds__(kOsThreads, 4) k_radix_pass(uint32_t n, const uint32_t* __restrict__ kin,
                                                              const uint32_t* __restrict__ vin,
                                                              uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                              const uint32_t* __restrict__ place, uint32_t tiles,
                                                              int shift, uint32_t* cell_count,
                                                              uint32_t* __restrict__ vout2, uint32_t* next_count) {
  constexpr uint32_t kRadix = 1u << kWidth, kMask = kRadix - 1u;
  __shared__ uint32_t s_key[kOsTile];
  __shared__ uint32_t s_val[kOsTile];
  __shared__ uint32_t s_wcnt[kOsWarps][kRadix];  // per-warp digit counts, then offsets over warps
  __shared__ uint32_t s_loc[kRadix];             // digit counts of the tile, then their exclusive scan
  __shared__ uint32_t s_glob[kRadix];            // global place of the tile's first record of each digit
  chain_begin(kin, vin, place);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t tile = blockIdx.x;
  for (uint32_t i = tid; i < kOsWarps * kRadix; i += kOsThreads) (&s_wcnt[0][0])[i] = 0u;
  if constexpr (kFew) {
    // the digit's records in all tiles, and in the tiles before this one
    __shared__ uint32_t s_warp[32];
    uint32_t all = 0u, before = 0u, total;
    if (tid < kRadix)
      for (uint32_t t = 0; t < tiles; ++t) {
        const uint32_t c = __ldg(place + (size_t)tid * tiles + t);
        all += c;
        before += t < tile ? c : 0u;
      }
    const uint32_t base = block_exclusive(all, &total, s_warp);
    if (tid < kRadix) s_glob[tid] = base + before;
  } else {
    for (uint32_t d = tid; d < kRadix; d += kOsThreads) s_glob[d] = __ldg(place + (size_t)d * tiles + tile);
  }
  const uint32_t t0 = tile * (uint32_t)kOsTile;
  // warp w holds records t0 + 512 w .. + 511; round i is records 32 i .. 32 i + 31 of it
  const uint32_t w0 = t0 + warp * (32u * kOsItems) + lane;
  uint32_t k[kOsItems], v[kOsItems], r[kOsItems];
#pragma unroll
  for (int i = 0; i < kOsItems; ++i) {
    const uint32_t idx = w0 + 32u * i;
    const bool valid = idx < n;
    k[i] = valid ? __ldg(kin + idx) : 0xffffffffu;
    v[i] = valid ? (vin ? __ldg(vin + idx) : idx) : 0u;
  }
  __syncthreads();
  // stable ranks within the warp, round by round in input order: the lowest
  // lane of each digit group adds the group to the warp's counter and passes
  // the old count on (shared-memory atomics keep the rounds in order)
  uint32_t* wc = s_wcnt[warp];
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < kOsItems; ++i) {
    const bool valid = w0 + 32u * i < n;
    const uint32_t d = (k[i] >> shift) & kMask;
    const unsigned peers = digit_peers<kWidth>(d, valid);
    const int leader = __ffs(peers) - 1;
    uint32_t before = 0u;
    if (valid && (int)lane == leader) before = atomicAdd(wc + d, (uint32_t)__popc(peers));
    before = __shfl_sync(kFull, before, leader & 31);
    r[i] = before + (uint32_t)__popc(peers & lt);
  }
  __syncthreads();
  // per digit: offsets over the warps and the tile's count
  if (tid < kRadix) {
    uint32_t cnt = 0;
#pragma unroll
    for (int w = 0; w < kOsWarps; ++w) {
      const uint32_t c = s_wcnt[w][tid];
      s_wcnt[w][tid] = cnt;
      cnt += c;
    }
    s_loc[tid] = cnt;
  }
  __syncthreads();
  // exclusive scan of the tile's digit counts (warp 0)
  if (warp == 0) {
    constexpr uint32_t kPer = (kRadix + 31u) / 32u;
    uint32_t loc[kPer];
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
      const uint32_t d = lane * kPer + j;
      loc[j] = d < kRadix ? s_loc[d] : 0u;
      sum += loc[j];
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, x, o);
      if ((int)lane >= o) x += y;
    }
    uint32_t run = x - sum;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
      const uint32_t d = lane * kPer + j;
      if (d < kRadix) s_loc[d] = run;
      run += loc[j];
    }
  }
  __syncthreads();
  // records to their tile-sorted place in shared memory
#pragma unroll
  for (int i = 0; i < kOsItems; ++i) {
    if (w0 + 32u * i < n) {
      const uint32_t d = (k[i] >> shift) & kMask;
      const uint32_t lp = s_loc[d] + s_wcnt[warp][d] + r[i];
      s_key[lp] = k[i];
      s_val[lp] = v[i];
    }
  }
  __syncthreads();
  // each digit's run to its global place: consecutive j, consecutive addresses
  const uint32_t in_tile = (n - t0) < (uint32_t)kOsTile ? (n - t0) : (uint32_t)kOsTile;
#pragma unroll 4
  for (uint32_t j0 = 0; j0 < in_tile; j0 += kOsThreads) {
    const uint32_t j = j0 + tid;
    const bool valid = j < in_tile;
    const uint32_t kk = valid ? s_key[j] : 0xffffffffu;
    uint32_t next = 0u;  // where the next pass counts the record
    if (valid) {
      const uint32_t d = (kk >> shift) & kMask;
      const uint32_t p = s_glob[d] + (j - s_loc[d]);
      if (p < n) {
        const uint32_t v = s_val[j];
        kout[p] = kk;
        vout[p] = v;
        if (vout2) vout2[p] = v;
        if constexpr (kRuns)
          next = ((kk >> (shift + kWidth)) & kMask) * tiles + p / (uint32_t)kOsTile;
        else if constexpr (kFew)
          if (next_count) atomicAdd(next_count + (size_t)((kk >> (shift + kWidth)) & kMask) * tiles + p / kOsTile, 1u);
      }
    }
    if constexpr (kRuns)
      if (next_count) add_runs(next_count, next, lane, valid);
    if (cell_count) add_runs(cell_count, kk, lane, valid);
  }
}

// particleSortIndex: the place of each particle within its cell, by particle
// id.  Four sorted positions a thread (vector loads keep more reads in flight
// ahead of the scattered stores).
__global__ void __launch_bounds__(256) k_rank_sorted(uint32_t n, const uint32_t* __restrict__ skey,
                                                     const uint32_t* __restrict__ order,
                                                     const uint32_t* __restrict__ cell_start,
                                                     uint32_t* __restrict__ rank_out) {
  chain_begin(skey, order, cell_start);
  const uint32_t q0 = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
  if (q0 >= n) return;
  if (q0 + 4u <= n) {
    const uint4 k = __ldg(reinterpret_cast<const uint4*>(skey + q0));
    const uint4 o = __ldg(reinterpret_cast<const uint4*>(order + q0));
    const uint32_t s0 = __ldg(cell_start + k.x), s1 = __ldg(cell_start + k.y), s2 = __ldg(cell_start + k.z),
                   s3 = __ldg(cell_start + k.w);
    rank_out[o.x] = q0 - s0;
    rank_out[o.y] = q0 + 1u - s1;
    rank_out[o.z] = q0 + 2u - s2;
    rank_out[o.w] = q0 + 3u - s3;
  } else {
    for (uint32_t q = q0; q < n; ++q) rank_out[order[q]] = q - __ldg(cell_start + skey[q]);
  }
}

__global__ void k_scatter_f4(uint32_t n, const uint32_t* __restrict__ id, const float4* __restrict__ src,
                             float4* __restrict__ dst) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  dst[id[t]] = src[t];
}
__global__ void k_scatter_w(uint32_t n, const uint32_t* __restrict__ id, const float4* __restrict__ src,
                            float* __restrict__ dst) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  dst[id[t]] = src[t].w;
}
__global__ void k_scatter_u32(uint32_t n, const uint32_t* __restrict__ id, const uint32_t* __restrict__ src,
                              uint32_t* __restrict__ dst) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  dst[id[t]] = src[t];
}
// ---- neighbour lists in the reference layout (stand-alone search) -------------------
// NeighborCount + NeighborList (neighborShader.ts:101-246) in two traversals
// of the 27 cells.  The positions go into sorted order once, each with its
// particle id in w, so the traversals read neighbouring candidates and the
// list kernel has a neighbour's id at hand.
__global__ void __launch_bounds__(256) k_ns_sorted(uint32_t n, const uint32_t* __restrict__ order,
                                                   const float4* __restrict__ pos, float4* __restrict__ sorted,
                                                   uint32_t* __restrict__ scan, uint32_t scan_words,
                                                   unsigned long long* total) {
  chain_begin(order, pos);
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  for (uint32_t i = t; i < scan_words; i += gridDim.x * blockDim.x) scan[i] = 0u;  // of the scan between the traversals
  if (t == 0u) *total = 0ull;
  if (t >= n) return;
  const uint32_t o = min(order[t], n - 1u);  // (after a sort whose scan gave up, an entry may be unwritten)
  float4 x = __ldg(pos + o);
  x.w = __uint_as_float(o);
  sorted[t] = x;
}

// each(in, id): every candidate in order, in: whether it is a neighbour.  Four
// loads in flight; the last, partial group of a run is taken one by one.
template <class Each>
__device__ __forceinline__ void test_cells27(const GridParams& g, const uint32_t* __restrict__ cell_start,
                                             const float4* __restrict__ sorted, f3 xi, float h2, Each&& each) {
  const int cx = cell_axis(xi.x, g.origin[0], g.inv_cell[0], g.dim[0]);
  const int cy = cell_axis(xi.y, g.origin[1], g.inv_cell[1], g.dim[1]);
  const int cz = cell_axis(xi.z, g.origin[2], g.inv_cell[2], g.dim[2]);
  for (int dx = -1; dx <= 1; ++dx)
    for (int dy = -1; dy <= 1; ++dy) {
      const Run r = run_of(g, cell_start, cx, cy, cz, dx, dy);
      uint32_t u = r.b;
      for (; u + 4u <= r.e; u += 4u) {
        float4 c[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) c[m] = __ldg(sorted + u + m);
#pragma unroll
        for (int m = 0; m < 4; ++m) each(dist2_rn(xyz(c[m]) - xi) <= h2, __float_as_uint(c[m].w));
      }
      for (; u < r.e; ++u) {
        const float4 c = __ldg(sorted + u);
        each(dist2_rn(xyz(c) - xi) <= h2, __float_as_uint(c.w));
      }
    }
}

// Counts by particle id; entry n receives 0, so a scan of n + 1 ends in the
// total modulo 2^32.  *total is the whole sum: 65,536 points within a radius
// of each other already have 2^32 neighbours.
__global__ void __launch_bounds__(128) k_ns_count(uint32_t n, GridParams g, float h2,
                                                  const float4* __restrict__ sorted,
                                                  const uint32_t* __restrict__ cell_start,
                                                  uint32_t* __restrict__ count, unsigned long long* total) {
  chain_begin(sorted, cell_start);
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t == n) count[n] = 0u;
  uint32_t c = 0;
  if (t < n) {
    const float4 x = sorted[t];
    test_cells27(g, cell_start, sorted, xyz(x), h2, [&](bool in, uint32_t) { c += in ? 1u : 0u; });
    count[__float_as_uint(x.w)] = c;
  }
  const uint32_t lo = __reduce_add_sync(kFull, c & 0xffffu), hi = __reduce_add_sync(kFull, c >> 16);
  if ((threadIdx.x & 31u) == 0u && t < n) atomicAdd(total, ((unsigned long long)hi << 16) + lo);
}

// The lists, written only if they all fit (*total <= capacity).  A thread
// writes its particle's run as it finds it: the id arrives with the candidate.
// Each run is tested against the capacity all the same: offsets are too small
// after a scan that gave up.
__global__ void __launch_bounds__(128) k_ns_list(uint32_t n, GridParams g, float h2,
                                                 const float4* __restrict__ sorted,
                                                 const uint32_t* __restrict__ cell_start,
                                                 const uint32_t* __restrict__ count,
                                                 const uint32_t* __restrict__ offset, uint32_t* __restrict__ list,
                                                 uint32_t capacity, const unsigned long long* __restrict__ total) {
  chain_begin(sorted, cell_start, count, offset, total);
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n || *total > capacity) return;
  const float4 x = sorted[t];
  const uint32_t id = __float_as_uint(x.w), first = __ldg(offset + id);
  if ((uint64_t)first + __ldg(count + id) > capacity) return;
  uint32_t* out = list + first;
  test_cells27(g, cell_start, sorted, xyz(x), h2, [&](bool in, uint32_t j) {
    if (in) *out++ = j;
  });
}

// ---- metrics --------------------------------------------------------------------------
__device__ __forceinline__ void atomic_max_pos_float(float* addr, float v) {
  // v >= 0: the int ordering of non-negative floats matches their value ordering
  atomicMax(reinterpret_cast<int*>(addr), __float_as_int(v));
}
__global__ void __launch_bounds__(256) k_metrics(SimParams p, FieldParams f, const float* __restrict__ sdf,
                                                 const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                 const uint32_t* __restrict__ nbr_count, uint32_t n, float* accum_f,
                                                 double* accum_d, uint32_t* accum_u) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  float comp = 0.f, aerr = 0.f;
  double ke = 0.0, serr = 0.0, scomp = 0.0;
  uint32_t bad = 0, pen = 0, nb = 0;
  if (t < n) {
    if (nbr_count) nb = nbr_count[t];
    float4 x = pos[t];
    float4 v = vel[t];
    bool fin = isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(v.x) && isfinite(v.y) && isfinite(v.z);
    if (!fin) {
      bad = 1;
    } else {
      float e = x.w / p.rho0 - 1.0f;
      comp = fmaxf(0.0f, e);
      aerr = fabsf(e);
      serr = aerr;
      scomp = comp;
      ke = 0.5 * (double)p.m * ((double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z);
      if (f.loaded && sdf) {
        CellLoc L = field_locate(f, mk(x.x, x.y, x.z));
        uint32_t idx[32];
        cell_nodes(f, L.i, L.j, L.k, false, idx);
        float N[32];
        f3 dN[32];
        float val[32];
        shape32(L.s, N, dN);
        for (int q = 0; q < 32; ++q) val[q] = sdf[idx[q]];
        if (sum32(N, val) < 0.0f) pen = 1;
      }
    }
  }
  // warp reduce then one atomic per warp
  for (int o = 16; o > 0; o >>= 1) {
    comp = fmaxf(comp, __shfl_xor_sync(kFull, comp, o));
    aerr = fmaxf(aerr, __shfl_xor_sync(kFull, aerr, o));
    ke += __shfl_xor_sync(kFull, ke, o);
    serr += __shfl_xor_sync(kFull, serr, o);
    scomp += __shfl_xor_sync(kFull, scomp, o);
    bad += __shfl_xor_sync(kFull, bad, o);
    pen += __shfl_xor_sync(kFull, pen, o);
    nb += __shfl_xor_sync(kFull, nb, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomic_max_pos_float(accum_f + 0, comp);
    atomic_max_pos_float(accum_f + 1, aerr);
    atomicAdd(accum_d + 0, serr);
    atomicAdd(accum_d + 1, ke);
    atomicAdd(accum_d + 2, scomp);
    atomicAdd(accum_u + 0, bad);
    atomicAdd(accum_u + 1, pen);
    atomicAdd(accum_u + 2, nb);
  }
}

inline unsigned blocks_for(size_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

RadixPlan radix_plan(uint32_t cells, size_t n) {
  RadixPlan r;
  uint32_t bits = 1;
  while (bits < 32 && (1ull << bits) < (uint64_t)cells) ++bits;
  r.passes = (int)((bits + 7) / 8);
  r.width = (int)((bits + (uint32_t)r.passes - 1) / (uint32_t)r.passes);
  r.tiles = (n + kOsTile - 1) / kOsTile;
  return r;
}

namespace {
size_t round256(size_t b) { return (b + 255) / 256 * 256; }
}  // namespace

// Scratch for up to n points: the digit-major count matrix, its scan and one
// scan scratch per pass; or, for so few points that the tiles are few, one
// count matrix per pass.
constexpr int kMaxPasses = 4;
size_t radix_scratch_bytes(size_t n) {
  size_t tiles = (n + kOsTile - 1) / kOsTile;
  if (tiles == 0) tiles = 1;
  const size_t m = tiles * kOsMaxRadix;
  const size_t many = 2 * round256(m * sizeof(uint32_t)) + kMaxPasses * round256(scan_scratch_bytes(m));
  const size_t few = kMaxPasses * std::min(tiles, (size_t)kFewTiles) * kOsMaxRadix * sizeof(uint32_t);
  return tiles > kFewTiles ? std::max(many, few) : few;
}

namespace {
template <int W>
cudaError_t radix_sort(const GridParams& g, const float4* pos, uint32_t n, const RadixPlan& plan, uint32_t* keys,
                       uint32_t* skeys, uint32_t* order, uint32_t* order2, uint32_t* const tmp_k[2],
                       uint32_t* const tmp_v[2], char* sc, uint32_t* err, cudaStream_t st, cudaEvent_t after_keys,
                       uint32_t* cell_count, uint32_t* scan_scratch) {
  constexpr uint32_t kRadix = 1u << W;
  const uint32_t tiles = (uint32_t)plan.tiles;
  const bool few = tiles <= kFewTiles, early = n <= kEarlyMax;
  const size_t m = plan.tiles * kRadix;
  uint32_t* count = reinterpret_cast<uint32_t*>(sc);
  uint32_t* place = reinterpret_cast<uint32_t*>(sc + round256(m * sizeof(uint32_t)));
  char* scans = sc + 2 * round256(m * sizeof(uint32_t));
  const size_t scan_bytes = round256(scan_scratch_bytes(m));
  ClearRanges clear{};
  clear.p[0] = cell_count;
  clear.words[0] = (size_t)g.cells + 1;
  clear.p[1] = scan_scratch;
  clear.words[1] = scan_scratch_bytes((size_t)g.cells + 1) / sizeof(uint32_t);
  // few: the later passes' counts are added up in place; else the scans' scratch
  clear.p[2] = few ? count + m : reinterpret_cast<uint32_t*>(scans);
  clear.words[2] = few ? (size_t)(plan.passes - 1) * m : (size_t)plan.passes * scan_bytes / sizeof(uint32_t);
  // enough CTAs that clearing the cells does not hang on a few of them
  const size_t clearing = std::min<size_t>((clear.words[0] + 4095) / 4096, 152u * 8u);
  cudaError_t e = launch_chain(early, k_keys_digits<W>, (unsigned)std::max<size_t>(tiles, clearing), kOsThreads, 0, st, g,
                               pos, n, keys, count, tiles, clear);
  if (e != cudaSuccess) return e;
  if (after_keys && (e = cudaEventRecord(after_keys, st)) != cudaSuccess) return e;
  for (int p = 0; p < plan.passes; ++p) {
    const bool last = p == plan.passes - 1;
    const uint32_t* kin = p == 0 ? keys : tmp_k[(p - 1) & 1];
    const uint32_t* vin = p == 0 ? nullptr : tmp_v[(p - 1) & 1];
    uint32_t* kout = last ? skeys : tmp_k[p & 1];
    uint32_t* vout = last ? order : tmp_v[p & 1];
    uint32_t* cc = last ? cell_count : nullptr;
    uint32_t* v2 = last ? order2 : nullptr;
    const int shift = p * W;
    if (few) {
      uint32_t* c = count + (size_t)p * m;
      e = launch_chain(early, tiles > kRunTiles ? k_radix_pass<W, true, true> : k_radix_pass<W, true, false>, tiles,
                       kOsThreads, 0, st, n, kin, vin, kout, vout, c, tiles, shift, cc, v2, last ? nullptr : c + m);
    } else {
      if (p > 0) {
        e = launch_chain(early, k_tile_digits<W>, tiles, kOsThreads, 0, st, n, kin, count, tiles, shift);
        if (e != cudaSuccess) return e;
      }
      e = launch_exclusive_scan_cleared(count, place, m, scans + (size_t)p * scan_bytes, err, st, ScanExtra{}, early);
      if (e != cudaSuccess) return e;
      e = launch_chain(early, k_radix_pass<W, false, false>, tiles, kOsThreads, 0, st, n, kin, vin, kout, vout, place,
                       tiles, shift, cc, v2, nullptr);
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
}  // namespace

cudaError_t launch_radix_sort_idorder(GridParams g, const float4* pos, uint32_t n, uint32_t* keys, uint32_t* skeys,
                                      uint32_t* order, uint32_t* order2, uint32_t* const tmp_k[2],
                                      uint32_t* const tmp_v[2], void* scratch, uint32_t* err, cudaStream_t st,
                                      cudaEvent_t after_keys, uint32_t* cell_count, void* scan_scratch) {
  const RadixPlan plan = radix_plan(g.cells, n);
  switch (plan.width) {
#define PBF_RADIX_WIDTH(W)                                                                                        \
  case W:                                                                                                         \
    return radix_sort<W>(g, pos, n, plan, keys, skeys, order, order2, tmp_k, tmp_v, reinterpret_cast<char*>(scratch), \
                         err, st, after_keys, cell_count, reinterpret_cast<uint32_t*>(scan_scratch));
    PBF_RADIX_WIDTH(1)
    PBF_RADIX_WIDTH(2)
    PBF_RADIX_WIDTH(3)
    PBF_RADIX_WIDTH(4)
    PBF_RADIX_WIDTH(5)
    PBF_RADIX_WIDTH(6)
    PBF_RADIX_WIDTH(7)
    PBF_RADIX_WIDTH(8)
#undef PBF_RADIX_WIDTH
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t launch_rank_sorted(uint32_t n, const uint32_t* skeys, const uint32_t* order, const uint32_t* cell_start,
                               uint32_t* rank_out, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const uint32_t threads = (n + 3u) / 4u;
  return launch_chain(n <= kEarlyMax, k_rank_sorted, (threads + 255u) / 256u, 256, 0, st, n, skeys, order, cell_start,
                      rank_out);
}

size_t scan_scratch_bytes(size_t n) {
  size_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles == 0) tiles = 1;
  return 256 + tiles * sizeof(unsigned long long);
}

cudaError_t launch_exclusive_scan(const uint32_t* in, uint32_t* out, size_t n, void* scratch, uint32_t* err,
                                  cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(scratch, 0, scan_scratch_bytes(n), st);
  return e != cudaSuccess ? e : launch_exclusive_scan_cleared(in, out, n, scratch, err, st, ScanExtra{}, false);
}

cudaError_t launch_exclusive_scan_cleared(const uint32_t* in, uint32_t* out, size_t n, void* scratch, uint32_t* err,
                                          cudaStream_t st, const ScanExtra& X, bool early) {
  if (n == 0) return cudaSuccess;
  const size_t tiles = (n + kScanTile - 1) / kScanTile;
  uint32_t* counter = reinterpret_cast<uint32_t*>(scratch);
  unsigned long long* status = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(scratch) + 256);
  return launch_chain(early, k_scan, (unsigned)tiles, kScanThreads, 0, st, in, out, n, status, counter, err, X);
}

// Self-test of the look-back's bounded wait: one CTA of a two-tile scan,
// started as tile 1 (the tile counter is preset), so tile 0's status word,
// which nothing writes, is what it waits for.  The wait gives up after
// kSpinLimit polls, flags PBF_DEVERR_SCAN_TIMEOUT in *err and the kernel
// completes.  Every access stays inside the two tiles' buffers.
cudaError_t launch_scan_timeout_selftest(uint32_t* err, cudaStream_t st) {
  const size_t n = 2 * (size_t)kScanTile;
  uint32_t *in = nullptr, *out = nullptr;
  void* scratch = nullptr;
  cudaError_t e = cudaMallocAsync(&in, n * sizeof(uint32_t), st);
  if (e == cudaSuccess) e = cudaMallocAsync(&out, n * sizeof(uint32_t), st);
  if (e == cudaSuccess) e = cudaMallocAsync(&scratch, scan_scratch_bytes(n), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(in, 0, n * sizeof(uint32_t), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(scratch, 0, scan_scratch_bytes(n), st);
  const uint32_t one = 1u;
  uint32_t* counter = reinterpret_cast<uint32_t*>(scratch);
  if (e == cudaSuccess) e = cudaMemcpyAsync(counter, &one, sizeof(one), cudaMemcpyHostToDevice, st);
  unsigned long long* status = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(scratch) + 256);
  if (e == cudaSuccess) {
    k_scan<<<1, kScanThreads, 0, st>>>(in, out, n, status, counter, err, ScanExtra{});
    e = cudaGetLastError();
  }
  // the host value copied above must outlive the copy
  cudaError_t e2 = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = e2;
  cudaFreeAsync(in, st);
  cudaFreeAsync(out, st);
  cudaFreeAsync(scratch, st);
  e2 = cudaStreamSynchronize(st);
  return e == cudaSuccess ? e2 : e;
}

cudaError_t launch_sort_by_cell(GridParams g, uint32_t n, const uint32_t* ids, SortBuffers& b, uint32_t id_bits,
                                const GatherArgs& G, cudaStream_t st) {
  const bool early = n <= kEarlyMax;
  cudaError_t e = launch_exclusive_scan_cleared(b.cell_count, b.cell_start, (size_t)g.cells + 1, b.scan_scratch,
                                                      b.err, st, ScanExtra{b.count_next}, early);
  if (e != cudaSuccess) return e;
  if (n == 0) return cudaSuccess;
  e = launch_chain(early, k_scatter, blocks_for(n, 256), 256, 0, st, n, b.key, b.rank, b.cell_start, ids, b.perm_raw,
                   b.id_raw);
  if (e != cudaSuccess) return e;
  int passes = (int)((id_bits + 7) / 8);
  if (passes < 1) passes = 1;
  e = launch_chain(early, G.skey_out ? k_cellfix<true> : k_cellfix<false>, blocks_for(n, 256), 256, 0, st, n, b.key,
                   b.cell_count, b.cell_start, b.perm_raw, b.id_raw, b.perm, b.big_list, b.big_count, G);
  if (e != cudaSuccess) return e;
  return launch_chain(early, G.skey_out ? k_bigcell<true> : k_bigcell<false>, 152, kRadixThreads, 0, st, b.big_list,
                      b.big_count, b.cell_count, b.cell_start, b.perm_raw, b.id_raw, b.perm, b.tmp_a, b.tmp_b, passes,
                      G);
}

cudaError_t launch_scatter_by_id(uint32_t n, const uint32_t* id, const float4* src, float4* dst, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_scatter_f4<<<blocks_for(n, 256), 256, 0, st>>>(n, id, src, dst);
  return cudaGetLastError();
}
cudaError_t launch_scatter_w_by_id(uint32_t n, const uint32_t* id, const float4* src, float* dst, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_scatter_w<<<blocks_for(n, 256), 256, 0, st>>>(n, id, src, dst);
  return cudaGetLastError();
}
cudaError_t launch_scatter_by_id_u32(uint32_t n, const uint32_t* id, const uint32_t* src, uint32_t* dst,
                                     cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_scatter_u32<<<blocks_for(n, 256), 256, 0, st>>>(n, id, src, dst);
  return cudaGetLastError();
}
cudaError_t launch_ns_count(uint32_t n, const GridParams& g, float h2, const uint32_t* order, const float4* pos,
                            const uint32_t* cell_start, float4* sorted, uint32_t* count, uint32_t* offset,
                            unsigned long long* total, void* scan, uint32_t* err, cudaStream_t st) {
  const bool early = n <= kEarlyMax;
  const size_t m = (size_t)n + 1;
  cudaError_t e = launch_chain(early, k_ns_sorted, blocks_for(m, 256), 256, 0, st, n, order, pos, sorted,
                               reinterpret_cast<uint32_t*>(scan), (uint32_t)(scan_scratch_bytes(m) / sizeof(uint32_t)),
                               total);
  if (e != cudaSuccess) return e;
  e = launch_chain(early, k_ns_count, blocks_for(m, 128), 128, 0, st, n, g, h2, sorted, cell_start, count, total);
  if (e != cudaSuccess) return e;
  return launch_exclusive_scan_cleared(count, offset, m, scan, err, st, ScanExtra{}, early);
}
cudaError_t launch_ns_list(uint32_t n, const GridParams& g, float h2, const float4* sorted, const uint32_t* cell_start,
                           const uint32_t* count, const uint32_t* offset, const unsigned long long* total,
                           uint32_t* list, uint32_t capacity, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  return launch_chain(n <= kEarlyMax, k_ns_list, blocks_for(n, 128), 128, 0, st, n, g, h2, sorted, cell_start, count,
                      offset, list, capacity, total);
}
cudaError_t launch_metrics(SimParams p, FieldParams f, const float* sdf, const float4* pos, const float4* vel,
                           const uint32_t* nbr_count, uint32_t n, float* accum_f, double* accum_d, uint32_t* accum_u,
                           cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_metrics<<<blocks_for(n, 256), 256, 0, st>>>(p, f, sdf, pos, vel, nbr_count, n, accum_f, accum_d, accum_u);
  return cudaGetLastError();
}

}  // namespace pbf
