// Device primitives of the frontier dedupe: exclusive scan and a stable LSD radix sort of (u64 key, u32 value)
// pairs over a chosen bit range, 8-bit digits, one launch per digit pass (see radix_sort); small sorts count each pair's
// place in one launch. All launches go to the caller's stream.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "cz_place.h"

namespace cz {
namespace {   // each translation unit that sorts gets its own copy of these kernels

constexpr int SORT_THREADS = 256;
constexpr int SORT_ITEMS = 16;
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;   // keys per tile
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_CHUNK = SCAN_THREADS * SCAN_ITEMS;

// ---------------- exclusive scan of u32 ----------------
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}
// block-wide exclusive scan of one value per thread (blockDim.x == SCAN_THREADS); returns the block total too
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t &total) {
  __shared__ uint32_t ws[SCAN_THREADS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t inc = warp_incl_scan(v, lane);
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  if (w == 0) {
    const uint32_t x = lane < SCAN_THREADS / 32 ? ws[lane] : 0;
    const uint32_t xi = warp_incl_scan(x, lane);
    if (lane < SCAN_THREADS / 32) ws[lane] = xi - x;
  }
  __syncthreads();
  const uint32_t r = ws[w] + inc - v;
  total = 0;
  __shared__ uint32_t tot;
  if (threadIdx.x == SCAN_THREADS - 1) tot = r + v;
  __syncthreads();
  total = tot;
  __syncthreads();
  return r;
}

__global__ void k_scan_partials(const uint32_t *in, size_t n, uint32_t *partials) {
  const size_t base = (size_t)blockIdx.x * SCAN_CHUNK;
  uint32_t s = 0;
  for (int i = 0; i < SCAN_ITEMS; i++) {
    const size_t j = base + (size_t)i * SCAN_THREADS + threadIdx.x;
    if (j < n) s += in[j];
  }
  uint32_t total;
  (void)block_excl_scan(s, total);
  if (threadIdx.x == 0) partials[blockIdx.x] = total;
}
// one block: exclusive scan of the partials in place, grand total to *total
__global__ void k_scan_single(uint32_t *p, size_t np, uint32_t *total) {
  uint32_t carry = 0;
  for (size_t b = 0; b < np; b += SCAN_THREADS) {
    const size_t j = b + threadIdx.x;
    const uint32_t v = j < np ? p[j] : 0;
    uint32_t t;
    const uint32_t e = block_excl_scan(v, t);
    if (j < np) p[j] = carry + e;
    carry += t;
  }
  if (threadIdx.x == 0 && total) *total = carry;
}
__global__ void k_scan_apply(const uint32_t *in, size_t n, const uint32_t *partials, uint32_t *out) {
  const size_t base = (size_t)blockIdx.x * SCAN_CHUNK;
  // each thread owns SCAN_ITEMS consecutive values
  uint32_t v[SCAN_ITEMS], s = 0;
  for (int i = 0; i < SCAN_ITEMS; i++) {
    const size_t j = base + (size_t)threadIdx.x * SCAN_ITEMS + i;
    v[i] = j < n ? in[j] : 0;
    s += v[i];
  }
  uint32_t total;
  uint32_t e = block_excl_scan(s, total) + partials[blockIdx.x];
  for (int i = 0; i < SCAN_ITEMS; i++) {
    const size_t j = base + (size_t)threadIdx.x * SCAN_ITEMS + i;
    if (j < n) out[j] = e;
    e += v[i];
  }
}

// partials: >= ceil(n / SCAN_CHUNK) + 1 words; in may equal out
inline void exclusive_scan(const uint32_t *in, uint32_t *out, size_t n, uint32_t *partials, uint32_t *total,
                           cudaStream_t s) {
  const size_t nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
  if (nb == 0) { if (total) cudaMemsetAsync(total, 0, 4, s); return; }
  k_scan_partials<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, n, partials);
  k_scan_single<<<1, SCAN_THREADS, 0, s>>>(partials, nb, total);
  k_scan_apply<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, n, partials, out);
}
inline size_t scan_partials_words(size_t n) { return (n + SCAN_CHUNK - 1) / SCAN_CHUNK + 1; }

// ---------------- radix sort ----------------
// Stable LSD radix sort of (u64 key, u32 value) pairs by bits [lo, hi) of the key, 8-bit digits, one launch per
// digit pass:
//  * k_sort_upsweep reads the keys once and counts every pass's digits (global histograms);
//  * k_sort_onesweep, per pass, takes tiles of OS_TILE keys in the order of an atomic ticket. A tile counts its
//    digits, publishes them, and finds the keys of earlier tiles per digit by looking back over their published
//    words (decoupled look-back: an earlier tile's word is either its own count or, once its look-back is done, the
//    inclusive prefix; walking back stops at the first prefix). Its keys are ranked stably without block barriers
//    between rounds: each warp holds a contiguous eighth of the tile and ranks its keys among its own (a ballot per bit,
//    one counter update per digit group), a scan over the warps' counts per digit joins the eighths, and the keys are
//    placed in shared memory in digit order and written out so that neighbouring threads write neighbouring
//    addresses.
// A tile waits only for tiles with smaller tickets, whose blocks are already running, so the waits end; every wait
// is still bounded (OS_SPIN_MAX polls). Should one give up, the tile counts the earlier tiles' digits itself from
// the input (slow, still exact) and the sort records it (sort_failed), so a result is never wrong and nothing hangs.
// Status words: tag (pass + 1, 4 bits) | state (2 bits: 1 count, 2 prefix) | value (58 bits); the scratch is
// cleared once per sort, and the tag tells one pass's words from the previous pass's.
constexpr int OS_THREADS = 256;
constexpr int OS_ITEMS = 8;
constexpr int OS_TILE = OS_THREADS * OS_ITEMS;     // keys per tile
constexpr int OS_MAXPASS = 8;
constexpr long long OS_SPIN_MAX = 1LL << 26;
constexpr size_t OS_HEAD_WORDS = 256 * OS_MAXPASS + 16;   // digit counts per pass, tickets per pass, error flag
constexpr unsigned long long OS_VALUE = (1ULL << 58) - 1;
constexpr size_t OS_SCAN_MIN = (size_t)1 << 22;     // sorts of at least this many keys take the scan path

inline size_t sort_tiles(size_t n) { return (n + OS_TILE - 1) / OS_TILE; }
// 32-bit words of sort scratch for n keys (header + one 64-bit status word per tile and digit)
inline size_t sort_hist_words(size_t n) { return OS_HEAD_WORDS + 2 * 256 * (sort_tiles(n) + 1); }

__global__ void __launch_bounds__(256) k_sort_upsweep(const uint64_t *keys, size_t n, int lo, int npass,
                                                       uint32_t *counts) {
  __shared__ uint32_t h[OS_MAXPASS][256];
  for (int p = 0; p < npass; p++) h[p][threadIdx.x] = 0;
  __syncthreads();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    for (int p = 0; p < npass; p++) atomicAdd(&h[p][(k >> (lo + 8 * p)) & 255], 1u);
  }
  __syncthreads();
  for (int p = 0; p < npass; p++)
    if (h[p][threadIdx.x]) atomicAdd(&counts[p * 256 + threadIdx.x], h[p][threadIdx.x]);
}

// per-tile digit counts of one pass, digit-major (hist[d * ntiles + tile]), tiles of OS_TILE keys
__global__ void __launch_bounds__(256) k_sort_tilehist(const uint64_t *keys, size_t n, int shift, uint32_t *hist,
                                                       uint32_t ntiles) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const size_t base = (size_t)blockIdx.x * OS_TILE;
  uint64_t k[OS_TILE / 256];                        // all loads before the first count: 75 -> 46 us a pass, 30 M pairs
#pragma unroll
  for (int r = 0; r < OS_TILE / 256; r++) {
    const size_t j = base + 256 * r + threadIdx.x;
    k[r] = j < n ? keys[j] : 0;
  }
#pragma unroll
  for (int r = 0; r < OS_TILE / 256; r++)
    if (base + 256 * r + threadIdx.x < n) atomicAdd(&h[(k[r] >> shift) & 255], 1u);
  __syncthreads();
  hist[(size_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

__device__ __forceinline__ unsigned long long os_load(const unsigned long long *p) {
  return *(const volatile unsigned long long *)p;
}
__device__ __forceinline__ void os_store(unsigned long long *p, unsigned long long v) {
  *(volatile unsigned long long *)p = v;
}
// exclusive scan of one u32 per thread over the 256 threads of the block
__device__ __forceinline__ uint32_t os_block_scan(uint32_t v, uint32_t *ws) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t inc = warp_incl_scan(v, lane);
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  if (w == 0) {
    const uint32_t x = lane < OS_THREADS / 32 ? ws[lane] : 0;
    const uint32_t xi = warp_incl_scan(x, lane);
    if (lane < OS_THREADS / 32) ws[lane] = xi - x;
  }
  __syncthreads();
  const uint32_t r = ws[w] + inc - v;
  __syncthreads();
  return r;
}

template <bool LOOKBACK>
__global__ void __launch_bounds__(OS_THREADS, 4) k_sort_onesweep(const uint64_t *kin, const uint32_t *vin, uint64_t *kout,
                                                               uint32_t *vout, size_t n, int shift, int pass,
                                                               uint32_t *head, unsigned long long *status,
                                                               unsigned *err, const uint32_t *offs, uint32_t ntiles) {
  constexpr int NW = OS_THREADS / 32;
  __shared__ uint64_t sk[OS_TILE];
  __shared__ uint32_t sv[OS_TILE];
  __shared__ uint32_t lex[256], run[256], wcnt[NW][256], ws[NW];
  __shared__ unsigned long long gbase[256];
  __shared__ unsigned ticket;
  __shared__ int fallback;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint32_t *counts = head + pass * 256;
  unsigned *tickets = head + 256 * OS_MAXPASS;
  if (tid == 0) { ticket = LOOKBACK ? atomicAdd(&tickets[pass], 1u) : blockIdx.x; fallback = 0; }
  for (int x = 0; x < NW; x++) wcnt[x][tid] = 0;
  __syncthreads();
  const size_t tile = ticket, start = tile * OS_TILE;
  const unsigned long long tag = (unsigned long long)(pass + 1) << 60;
  // warp w holds tile positions [w * 32 * OS_ITEMS, (w + 1) * 32 * OS_ITEMS), round r lane l the position
  // w * 32 * OS_ITEMS + 32 r + l: input order is (warp, round, lane)
  uint64_t key[OS_ITEMS];
  uint32_t val[OS_ITEMS], wr[OS_ITEMS];
  int dig[OS_ITEMS];
#pragma unroll
  for (int r = 0; r < OS_ITEMS; r++) {
    const size_t i = start + (size_t)w * 32 * OS_ITEMS + 32 * r + lane;
    dig[r] = 256;
    if (i < n) {
      key[r] = kin[i];
      val[r] = vin[i];
      dig[r] = (int)((key[r] >> shift) & 255);
    }
  }
  // each warp's digit counts and every key's rank among its warp's keys of the same digit (earlier rounds, then
  // lower lanes): one leader per digit group updates the warp's counter, so no atomics and no block barrier. The lanes
  // of one digit are found by a ballot per digit bit (and one for the tile's end): __match_any_sync, whose cost grows
  // with the distinct digits of a warp, held the kernel (30 M pairs, four passes: 1037 us with it, 885 with ballots;
  // the same counters by shared atomics 1353, tiles of 512 threads 1214)
  const unsigned lt = (1u << lane) - 1;
#pragma unroll
  for (int r = 0; r < OS_ITEMS; r++) {
    const int d = dig[r];
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 9; b++) {
      const bool on = (d >> b) & 1;
      const unsigned m = __ballot_sync(0xffffffffu, on);
      peers &= on ? m : ~m;
    }
    const int leader = __ffs(peers) - 1;
    uint32_t old = 0;
    if (d < 256 && lane == leader) { old = wcnt[w][d]; wcnt[w][d] = old + (uint32_t)__popc(peers); }
    old = __shfl_sync(0xffffffffu, old, leader);
    wr[r] = old + (uint32_t)__popc(peers & lt);
    __syncwarp();
  }
  __syncthreads();
  // per digit tid: the warps' counts become exclusive prefixes (earlier warps' keys of the digit); the tile's count
  uint32_t mine = 0;
#pragma unroll
  for (int x = 0; x < NW; x++) {
    const uint32_t t = wcnt[x][tid];
    wcnt[x][tid] = mine;
    mine += t;
  }
  if constexpr (LOOKBACK) {
    // this tile's count of digit tid: publish it, then add up the earlier tiles' counts by looking back
    unsigned long long *st = status + tile * 256 + tid;
    unsigned long long before = 0;
    bool ok = true;
    if (tile == 0) {
      os_store(st, tag | (2ULL << 58) | mine);
    } else {
      os_store(st, tag | (1ULL << 58) | mine);
      for (long long j = (long long)tile - 1; j >= 0 && ok; j--) {
        const unsigned long long *q = status + (size_t)j * 256 + tid;
        unsigned long long v = os_load(q);
        long long spins = 0;
        while ((v >> 60) != (tag >> 60) && ++spins < OS_SPIN_MAX) {
          __nanosleep(64);
          v = os_load(q);
        }
        if ((v >> 60) != (tag >> 60)) { ok = false; break; }
        before += v & OS_VALUE;
        if (((v >> 58) & 3) == 2) break;
      }
    }
    if (!ok) { atomicOr(err, 1u); fallback = 1; }
    __syncthreads();
    if (fallback) {                               // a wait gave up: count the earlier tiles' digits directly
      run[tid] = 0;
      __syncthreads();
      for (size_t i = tid; i < start; i += OS_THREADS) atomicAdd(&run[(kin[i] >> shift) & 255], 1u);
      __syncthreads();
      before = run[tid];
      __syncthreads();
    }
    if (tile != 0) os_store(st, tag | (2ULL << 58) | ((before + mine) & OS_VALUE));
    // output base of digit tid for this tile: keys of smaller digits (all tiles) + this digit's in earlier tiles
    const uint32_t dex = os_block_scan(counts[tid], ws);
    gbase[tid] = (unsigned long long)dex + before;
  } else {
    gbase[tid] = offs[(size_t)tid * ntiles + tile];   // the scanned digit-major tile histograms
  }
  lex[tid] = os_block_scan(mine, ws);             // keys of smaller digits in this tile
  __syncthreads();
  // each key to its place in the tile's digit order: smaller digits, earlier warps' keys of its digit, its rank
#pragma unroll
  for (int r = 0; r < OS_ITEMS; r++) {
    const int d = dig[r];
    if (d < 256) {
      const uint32_t pos = lex[d] + wcnt[w][d] + wr[r];
      sk[pos] = key[r];
      sv[pos] = val[r];
    }
  }
  __syncthreads();
  const int tn = (int)(n - start < (size_t)OS_TILE ? n - start : (size_t)OS_TILE);
  for (int i = tid; i < tn; i += OS_THREADS) {
    const uint64_t k = sk[i];
    const int d = (int)((k >> shift) & 255);
    const unsigned long long pos = gbase[d] + (unsigned long long)(i - (int)lex[d]);
    if (pos < n) {                                // always, for a consistent input (nothing else writes the keys)
      kout[pos] = k;
      vout[pos] = sv[i];
    } else {
      atomicOr(err, 2u);
    }
  }
}

// Small sorts in one launch: a pair's place is the number of smaller keys plus the number of equal keys before it,
// counted directly. A block places 32 pairs (one per lane); its warps share the keys, read tile by tile into shared
// memory, and a key is compared with 32 at once from a broadcast. n^2 / 32 compares, but no passes, no scratch and one
// launch where the digit passes need 1 + passes and a memset. On the B200 (us; counting / digit passes):
//   pairs   8 bits       16 bits      32 bits      64 bits
//   1000    11 / 16      11 / 22      11 / 34      12 / 59
//   4096    16 / 17.5    16 / 26      16 / 42      16 / 75
//   6000    20 / 18      20 / 26      20 / 42      24 / 75
//   8192    24.5 / 18    24.5 / 26    24.5 / 42    29 / 75
// so one pass is counted up to 4096 pairs, and two or more, which meet counting at about 8400, up to 8192.
// Keys that change while they are sorted (a caller's, not ordered before the call) can give two pairs one place, or one the
// place n, which is not written. Where the caller's flags are given, the places' marks are summed: see SortFlags.
constexpr size_t sort_count_max(int bits) { return bits <= 8 ? 4096 : 8192; }   // pairs sorted by counting
constexpr int SC_THREADS = 256, SC_TILE = 1024;
template <typename K>     // uint32_t when hi - lo <= 32, else uint64_t: the digits compared
__global__ void __launch_bounds__(SC_THREADS) k_sort_count(const uint64_t *kin, const uint32_t *vin, uint64_t *kout, uint32_t *vout,
                                                           int n, int lo, uint64_t mask, unsigned long long *places) {
  constexpr int NW = SC_THREADS / 32, PER = SC_TILE / NW;
  __shared__ K tile[SC_TILE];
  __shared__ int part[NW][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i0 = blockIdx.x * 32, i = i0 + lane;
  const uint64_t key = i < n ? kin[i] : 0;
  const K mine = (K)((key >> lo) & mask);
  int cnt = 0;
  for (int t0 = 0; t0 < n; t0 += SC_TILE) {
    const int tn = min(SC_TILE, n - t0);
    __syncthreads();
    for (int x = threadIdx.x; x < tn; x += SC_THREADS) tile[x] = (K)((kin[t0 + x] >> lo) & mask);
    __syncthreads();
    const int a = w * PER, b = min(a + PER, tn);
    if (t0 + b <= i0) {                                          // all before the block's pairs: equal keys count
#pragma unroll 8
      for (int x = a; x < b; x++) cnt += tile[x] <= mine;
    } else if (t0 + a >= i0 + 32) {                              // all behind them
#pragma unroll 8
      for (int x = a; x < b; x++) cnt += tile[x] < mine;
    } else {
      for (int x = a; x < b; x++) cnt += tile[x] < mine || (tile[x] == mine && t0 + x < i);
    }
  }
  part[w][lane] = cnt;
  __syncthreads();
  if (w == 0) {
    unsigned pos = 0;
#pragma unroll
    for (int x = 0; x < NW; x++) pos += (unsigned)part[x][lane];
    if (i < n && pos < (unsigned)n) {
      kout[pos] = key;
      vout[pos] = vin[i];
    }
    if (places) {
      uint64_t d = i < n ? place_mark(pos) - place_mark((uint32_t)i) : 0;
#pragma unroll
      for (int m = 16; m; m >>= 1) d += __shfl_xor_sync(0xffffffffu, d, m);
      if (lane == 0 && d) atomicAdd(places, (unsigned long long)d);
    }
  }
}

// what a sort tells of itself: both words are 0 before it and after a good one, so nothing clears them between sorts
struct SortFlags {
  uint32_t err, pad;              // digit passes: bit 0, a look-back wait gave up; bit 1, a position outside the array
  unsigned long long places;      // counting sort: the sum of its places' marks, 0 for a permutation
};
struct SortScratch {
  uint32_t *hist = nullptr;       // sort scratch: sort_hist_words(n) words
  uint32_t *partials = nullptr;   // scan partials: scan_partials_words(sort_hist_words(n)) words (large sorts)
  size_t cap_hist = 0, cap_part = 0;
  SortFlags *flags = nullptr;     // for sort_failed (nullptr: not read)
};

// sorts (k0, v0) by bits [lo, hi) of the key (hi - lo a multiple of 8, at most 64), stable; uses (k1, v1) as the
// other buffer. Returns true when the result ended in (k1, v1). Counts launches into *launches.
inline bool radix_sort(uint64_t *k0, uint32_t *v0, uint64_t *k1, uint32_t *v1, size_t n, int lo, int hi,
                       const SortScratch &sc, cudaStream_t s, int *launches) {
  if (n <= 1 || hi <= lo) return false;
  if (n <= sort_count_max(hi - lo)) {
    unsigned long long *places = sc.flags ? &sc.flags->places : nullptr;
    const unsigned nb = (unsigned)((n + 31) / 32);
    if (hi - lo <= 32)
      k_sort_count<uint32_t><<<nb, SC_THREADS, 0, s>>>(k0, v0, k1, v1, (int)n, lo, hi - lo == 32 ? 0xffffffffULL : (1ULL << (hi - lo)) - 1, places);
    else
      k_sort_count<uint64_t><<<nb, SC_THREADS, 0, s>>>(k0, v0, k1, v1, (int)n, lo, hi - lo == 64 ? ~0ULL : (1ULL << (hi - lo)) - 1, places);
    if (launches) (*launches)++;
    return true;
  }
  const int npass = (hi - lo + 7) / 8;
  const size_t ntiles = sort_tiles(n);
  const bool scan = n >= OS_SCAN_MIN && sc.partials && sc.cap_part >= scan_partials_words(256 * ntiles);
  cudaMemsetAsync(sc.hist, 0, (OS_HEAD_WORDS + (scan ? 0 : 2 * 256 * ntiles)) * 4, s);
  unsigned long long *status = (unsigned long long *)(sc.hist + OS_HEAD_WORDS);
  uint32_t *offs = sc.hist + OS_HEAD_WORDS;                  // scan path: the digit-major tile histograms
  unsigned *err = sc.flags ? &sc.flags->err : sc.hist + 256 * OS_MAXPASS + OS_MAXPASS;
  if (!scan) {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const unsigned ub = (unsigned)std::max<size_t>(1, std::min<size_t>((n + 255) / 256, (size_t)nsm * 8));
    k_sort_upsweep<<<ub, 256, 0, s>>>(k0, n, lo, npass, sc.hist);
  }
  bool flip = false;
  for (int p = 0; p < npass; p++) {
    const uint64_t *ki = flip ? k1 : k0;
    const uint32_t *vi = flip ? v1 : v0;
    uint64_t *ko = flip ? k0 : k1;
    uint32_t *vo = flip ? v0 : v1;
    if (scan) {
      k_sort_tilehist<<<(unsigned)ntiles, 256, 0, s>>>(ki, n, lo + 8 * p, offs, (uint32_t)ntiles);
      exclusive_scan(offs, offs, 256 * ntiles, sc.partials, nullptr, s);
      k_sort_onesweep<false><<<(unsigned)ntiles, OS_THREADS, 0, s>>>(ki, vi, ko, vo, n, lo + 8 * p, p, sc.hist, status,
                                                                   err, offs, (uint32_t)ntiles);
    } else {
      k_sort_onesweep<true><<<(unsigned)ntiles, OS_THREADS, 0, s>>>(ki, vi, ko, vo, n, lo + 8 * p, p, sc.hist, status,
                                                                  err, nullptr, 0);
    }
    flip = !flip;
  }
  if (launches) *launches += scan ? 5 * npass : 1 + npass;
  return flip;
}
// the last sort's flags (synchronises the stream; the scratch has them): bit 0, a look-back wait gave up (the result is
// exact all the same: the tile counted its predecessors' digits itself); bit 1, a scatter position fell outside the
// array, or a small sort's places are no permutation (the keys changed while the sort ran; the result is not to be used)
inline uint32_t sort_failed(const SortScratch &sc, cudaStream_t s) {
  SortFlags f{0, 0, 0};
  cudaMemcpyAsync(&f, sc.flags, sizeof f, cudaMemcpyDeviceToHost, s);
  cudaStreamSynchronize(s);
  if (f.err || f.places) cudaMemsetAsync(sc.flags, 0, sizeof f, s);
  return f.err | (f.places ? 2u : 0u);
}

}  // namespace
}  // namespace cz
