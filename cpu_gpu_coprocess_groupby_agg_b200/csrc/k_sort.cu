// Key-ordered output: a call's groups sorted by key, with every aggregate
// column permuted alike.
//
// The reference leaves each partition's groups in hash-table order
// (groupby_agg_intra_partition.cu:245-276 copies collect_kv_in_ht's output as
// it comes); key order is an option of this library, for callers that join or
// merge the groups downstream.
//
// A sample sort (splitters from a sorted sample, buckets that fit shared
// memory; Frazer and McKellar, 1970).  Keys of groups are distinct, so buckets
// are even whatever the keys' distribution.
//   k_sort_split    per segment: up to 8192 sampled keys sorted in shared
//                   memory, 2^bits - 1 splitters
//   k_sort_hist     keys of every bucket counted (a binary search per key)
//   k_sort_plan     bucket bounds, write cursors, tiles of the next level
//   k_part_scatter  (k_part.cu) keys and aggregate columns moved to their buckets
//   k_sort_buckets  a CTA orders one bucket in shared memory and writes its keys
//                   and aggregates to their final place
// One level for up to 2^19 groups, two levels above.  Jobs of up to one bucket
// are all sorted in place by one launch (k_sort_small).
//
// Bytes per group of b bytes: 2 (b + key) per level and 2 b for the buckets,
// against 2 (key + 4) for each of up to 8 passes plus the random gather of a
// least-significant-digit sort over (key, index) pairs.  Measured (us, that
// sort / this one): 16.8M int64 groups with 2 aggregates 2714 / 1130, 9.9M with
// 1 aggregate 1390 / 695, 48 queries of up to 2^17 groups (the whole batch
// call) 5410 / 1590.  The bucket kernel (2.3 TB/s on the 16.8M groups) is bound
// by its barriers and shared-memory round trips at 3 CTAs of 512 threads per
// SM (2 CTAs: 500 against 350 us), the count by the binary search's
// shared-memory reads.
//
// Jobs beyond the two levels, and a job with a bucket that outgrows shared
// memory (the sample missed the keys' distribution), take the
// least-significant-digit sort.  Its pass structure is the single-sweep radix
// sort published by Adinets and Merrill ("Onesweep", 2022): one upfront read
// of the keys counts every digit position, and each pass is then one kernel
// that ranks its tile and finds its global offsets by a decoupled look-back
// over earlier tiles, per digit.
//   k_sort_prep     counts of every 8-bit digit of the order-normalised key
//                   (sign bit flipped for signed keys), all positions at once
//   k_sort_mask     the digit positions whose keys do not all share one digit;
//                   only those passes run
//   k_sort_pass     one per pass: a CTA takes the next 4096-key tile from a
//                   counter, each warp ranks its 512 keys in order, 32 at a
//                   time (peers of equal digit from 8 ballots; their leader adds
//                   them to the warp's digit counter in shared memory), the tile
//                   publishes its digit counts and looks back over earlier tiles
//                   for their running totals (bounded spin; a timeout raises
//                   GBA_FLAG_WAIT_TIMEOUT), the tile is staged in shared memory
//                   in digit order and written out as contiguous runs; order
//                   inside a digit is the input order, so the sort is stable
//   k_sort_gather   every aggregate column permuted by the sorted group index
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "gba_internal.cuh"
#include "part_kernels.h"
#include "sort_kernels.h"

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortSteps = 16;                        // 32-key steps per warp
constexpr int kWarpSpan = 32 * kSortSteps;            // a warp's keys in a tile
constexpr int kSortTile = kSortThreads * kSortSteps;  // 4096 keys per tile
constexpr unsigned long long kAggregate = 1ull << 62;  // look-back word: this tile's count
constexpr unsigned long long kPrefix = 2ull << 62;     // look-back word: running total through this tile
constexpr unsigned long long kValue = (1ull << 62) - 1;
constexpr unsigned kSpinLimit = 1u << 24;   // look-back rounds without progress before giving up
constexpr int kLookWindow = 8;              // predecessor tiles read per look-back round

template <bool K64>
__device__ __forceinline__ unsigned long long load_raw(const void* keys, int64_t i) {
  if (K64) return __ldg(static_cast<const unsigned long long*>(keys) + i);
  return __ldg(static_cast<const unsigned*>(keys) + i);
}

template <bool K64>
__device__ __forceinline__ void store_raw(void* keys, int64_t i, unsigned long long k) {
  if (K64) static_cast<unsigned long long*>(keys)[i] = k;
  else static_cast<unsigned*>(keys)[i] = unsigned(k);
}

__device__ __forceinline__ unsigned digit_of(unsigned long long raw, unsigned long long flip, int shift) {
  return unsigned((raw ^ flip) >> shift) & 255u;
}

// hist[p * 256 + d]: keys whose digit p is d.  A warp whose 32 keys share a
// digit adds 32 once (the common case at the top of a narrow key range).
template <bool K64>
__global__ void __launch_bounds__(kSortThreads) k_sort_prep(const void* keys, int64_t g, unsigned long long flip,
                                                            unsigned* hist) {
  constexpr int P = K64 ? 8 : 4;
  __shared__ unsigned h[P * 256];
  for (int i = threadIdx.x; i < P * 256; i += kSortThreads) h[i] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t stride = int64_t(gridDim.x) * kSortThreads;
  for (int64_t base = int64_t(blockIdx.x) * kSortThreads; base < g; base += stride) {
    const int64_t i = base + threadIdx.x;
    const bool ok = i < g;
    const unsigned long long k = ok ? load_raw<K64>(keys, i) ^ flip : 0ull;
    const unsigned active = __ballot_sync(~0u, ok);
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const unsigned d = unsigned(k >> (8 * p)) & 255u;
      const unsigned d0 = __shfl_sync(~0u, d, 0);  // lane 0 is active whenever any lane is
      if (__all_sync(~0u, !ok || d == d0)) {
        if (lane == 0) atomicAdd(&h[p * 256 + d], unsigned(__popc(active)));
      } else if (ok) {
        atomicAdd(&h[p * 256 + d], 1u);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < P * 256; i += kSortThreads)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

// mask[j] bit p: pass p of job j moves keys (its digit is not the same for all)
__global__ void __launch_bounds__(kSortThreads) k_sort_mask(const unsigned* hists, const int64_t* gs, int npos,
                                                            unsigned* mask) {
  __shared__ unsigned m;
  if (threadIdx.x == 0) m = 0;
  __syncthreads();
  const unsigned* h = hists + size_t(blockIdx.x) * 8 * 256;
  const unsigned g = unsigned(gs[blockIdx.x]);
  for (int p = 0; p < 8; ++p)
    if (p < npos && h[p * 256 + threadIdx.x] == g) atomicOr(&m, 1u << p);  // one digit holds every key
  __syncthreads();
  if (threadIdx.x == 0) mask[blockIdx.x] = ~m & ((1u << npos) - 1u);
}

// The lanes whose 8-bit digit equals this lane's, among the lanes with ok set:
// one ballot per digit bit (the same mask __match_any_sync gives, from plain
// votes).
__device__ __forceinline__ unsigned digit_peers(unsigned d, bool ok) {
  unsigned m = __ballot_sync(~0u, ok);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const unsigned v = __ballot_sync(~0u, (d >> b) & 1u);
    m &= (d >> b) & 1u ? v : ~v;
  }
  return m;
}

// exclusive prefix over the block's 256 threads (one value each)
__device__ __forceinline__ unsigned long long block_excl256(unsigned long long v, unsigned long long* warp_tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(~0u, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  unsigned long long before = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w)
    if (w < warp) before += warp_tot[w];
  __syncthreads();
  return before + x - v;
}

struct PassArgs {
  const void* keys_in;
  const unsigned* idx_in;   // null: the key's index is its position (first pass)
  void* keys_out;
  unsigned* idx_out;
  int64_t g;
  unsigned long long flip;
  int shift;
  const unsigned* hist;     // this pass's 256 digit counts over all keys
  unsigned long long* look; // [tile][256] look-back words, zeroed
  unsigned* tile_ctr;       // zeroed
  unsigned* flags;
};

template <bool K64>
__global__ void __launch_bounds__(kSortThreads, 3) k_sort_pass(PassArgs a) {
  using KeyT = typename std::conditional<K64, unsigned long long, unsigned>::type;
  extern __shared__ __align__(16) unsigned char stage[];
  KeyT* skeys = reinterpret_cast<KeyT*>(stage);
  unsigned* sidx = reinterpret_cast<unsigned*>(stage + sizeof(KeyT) * kSortTile);
  __shared__ unsigned wcnt[kSortWarps][256];
  __shared__ unsigned dstart[256];
  __shared__ unsigned long long gbase[256];
  __shared__ unsigned long long warp_tot[kSortWarps];
  __shared__ unsigned s_tile;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t == 0) s_tile = atomicAdd(a.tile_ctr, 1u);
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) wcnt[w][t] = 0;
  __syncthreads();
  const int64_t tile = s_tile;
  const int64_t tile0 = tile * kSortTile;
  const int tile_n = a.g - tile0 < kSortTile ? int(a.g - tile0) : kSortTile;

  // rank every key among the tile's keys of the same digit, in input order
  const unsigned lt = (1u << lane) - 1u;
  const int64_t base = tile0 + int64_t(warp) * kWarpSpan + lane;
  KeyT key[kSortSteps];
  unsigned idx[kSortSteps], rank[kSortSteps];
#pragma unroll
  for (int step = 0; step < kSortSteps; ++step) {
    const int64_t i = base + step * 32;
    const bool ok = i < a.g;
    key[step] = ok ? KeyT(load_raw<K64>(a.keys_in, i)) : KeyT(0);
    idx[step] = ok ? (a.idx_in ? __ldg(a.idx_in + i) : unsigned(i)) : 0u;
  }
#pragma unroll
  for (int step = 0; step < kSortSteps; ++step) {
    const bool ok = base + step * 32 < a.g;
    const unsigned d = ok ? digit_of(key[step], a.flip, a.shift) : 0u;
    const unsigned peers = digit_peers(d, ok);
    const int leader = __ffs(peers) - 1;
    // the leader's atomic returns the count before this step; steps do not
    // wait on one another (the warp's counter row is touched by it alone)
    unsigned before = 0;
    if (ok && lane == leader) before = atomicAdd(&wcnt[warp][d], unsigned(__popc(peers)));
    before = __shfl_sync(~0u, before, leader);
    rank[step] = before + unsigned(__popc(peers & lt));
  }
  __syncthreads();

  // thread t owns digit t: warp prefix, tile count, publish, look back
  unsigned total = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    const unsigned c = wcnt[w][t];
    wcnt[w][t] = total;
    total += c;
  }
  unsigned long long* look = a.look + size_t(tile) * 256 + t;
  if (tile == 0) atomicExch(look, kPrefix | total);
  else atomicExch(look, kAggregate | total);
  const unsigned long long gstart = block_excl256(a.hist[t], warp_tot);
  dstart[t] = unsigned(block_excl256(total, warp_tot));
  unsigned long long excl = 0;
  if (tile > 0) {
    // walk back kLookWindow tiles per round of independent loads (the tiles of
    // the first wave all publish at once; one dependent load per tile would
    // make their walks serial)
    int64_t j = tile - 1;
    unsigned spins = 0;
    while (true) {
      unsigned long long w[kLookWindow];
#pragma unroll
      for (int u = 0; u < kLookWindow; ++u)
        w[u] = j - u >= 0 ? *reinterpret_cast<const volatile unsigned long long*>(a.look + size_t(j - u) * 256 + t)
                          : kPrefix;  // before tile 0: a running total of zero
      int used = 0;
      bool done = false;
#pragma unroll
      for (int u = 0; u < kLookWindow; ++u) {
        if (done || used < u) continue;        // stopped earlier in this window
        const unsigned long long f = w[u] & ~kValue;
        if (f == 0ull) continue;               // tile j - u has not published yet
        excl += w[u] & kValue;
        done = f == kPrefix;
        used = u + 1;
      }
      if (done) break;
      if (used == 0 && ++spins > kSpinLimit) {
        atomicOr(a.flags, GBA_FLAG_WAIT_TIMEOUT);
        break;
      }
      j -= used;
    }
    atomicExch(look, kPrefix | (excl + total));
  }
  gbase[t] = gstart + excl;
  __syncthreads();

  // stage the tile in digit order, then write each digit's run contiguously
#pragma unroll
  for (int step = 0; step < kSortSteps; ++step) {
    if (base + step * 32 >= a.g) continue;
    const unsigned d = digit_of(key[step], a.flip, a.shift);
    const unsigned pos = dstart[d] + wcnt[warp][d] + rank[step];
    skeys[pos] = KeyT(key[step]);
    sidx[pos] = idx[step];
  }
  __syncthreads();
  for (int i = t; i < tile_n; i += kSortThreads) {
    const unsigned long long k = skeys[i];
    const unsigned d = digit_of(k, a.flip, a.shift);
    const unsigned long long gpos = gbase[d] + unsigned(i - int(dstart[d]));
    if (gpos >= (unsigned long long)a.g) continue;  // only after a timed-out look-back
    store_raw<K64>(a.keys_out, int64_t(gpos), k);
    a.idx_out[gpos] = sidx[i];
  }
}

// ---- sample sort ------------------------------------------------------------------
constexpr int kBucketCap = 4096, kBucketThreads = 512, kBucketBins = 12;  // one bucket in shared memory
constexpr int kSampleCap = 8192, kSampleThreads = 1024, kSampleBins = 13;
constexpr int kLevelBits = 8;        // splitter bits per level at most
constexpr int kSamplePer = 64;       // sampled keys per bucket (32 at 8 bits)
constexpr int kBucketTarget = 2048;  // keys per bucket aimed at (at most; half of it at least)
constexpr int kBinMost = 16;         // keys per bin up to which a bin is ordered by comparing all of it

constexpr size_t order_smem(int cap, int bins) { return size_t(cap) * 8 + ((size_t(1) << bins) + 4) * 4 + size_t(cap) * 4; }

// Orders n <= CAP keys sk[0..n) of the CTA: order[r] = index of the r-th
// smallest.  The keys are counted into 2^BINS bins over their range (a power of
// two wide each), then each key counts the smaller keys of its bin.  Keys
// bunched in few bins take a bitonic sort of their indices instead.  Syncs
// before it returns.
template <int CAP, int THREADS, int BINS>
struct CtaOrder {
  unsigned long long* sk;
  unsigned* cnt;          // 2^BINS + 1
  unsigned short* bk;     // CAP
  unsigned short* order;  // CAP

  __device__ __forceinline__ CtaOrder(unsigned char* sm) {
    sk = reinterpret_cast<unsigned long long*>(sm);
    cnt = reinterpret_cast<unsigned*>(sk + CAP);
    bk = reinterpret_cast<unsigned short*>(cnt + (1 << BINS) + 4);
    order = bk + CAP;
  }
  __device__ __forceinline__ bool less(unsigned a, unsigned b) const {  // 0xffff: past the end
    if (a == 0xffffu || b == 0xffffu) return a != 0xffffu;
    const unsigned long long x = sk[a], y = sk[b];
    return x < y || (x == y && a < b);
  }
  // order[0..m) (m a power of two) sorted by key, the indices past the end last
  __device__ __forceinline__ void bitonic(int m) const {
    for (int size = 2; size <= m; size <<= 1)
      for (int step = size >> 1; step; step >>= 1) {
        for (int t = threadIdx.x; t < m / 2; t += THREADS) {
          const int i = 2 * t - (t & (step - 1)), j = i + step;
          const unsigned a = order[i], b = order[j];
          if (less(b, a) == ((i & size) == 0)) {
            order[i] = (unsigned short)b;
            order[j] = (unsigned short)a;
          }
        }
        __syncthreads();
      }
  }
  // Keys bunched in few bins: kSplit - 1 splitters from a sorted sample make
  // the bins instead (a sample sort inside shared memory; few keys are sorted
  // by the bitonic network outright).
  __device__ __forceinline__ void bunched(int n) const {
    constexpr int kSplit = 512, kSplitBits = 9;
    const int tid = threadIdx.x;
    __syncthreads();
    if (n <= 2 * kSplit) {
      int m = 1;
      while (m < n) m <<= 1;
      for (int i = tid; i < m; i += THREADS) order[i] = i < n ? (unsigned short)i : (unsigned short)0xffffu;
      __syncthreads();
      bitonic(m);
      return;
    }
    unsigned long long* split = reinterpret_cast<unsigned long long*>(cnt + kSplit + 16);
    for (int i = tid; i < kSplit; i += THREADS) order[i] = (unsigned short)((long long)n * i / kSplit);
    for (int i = tid; i <= kSplit; i += THREADS) cnt[i] = 0;
    __syncthreads();
    bitonic(kSplit);
    for (int i = tid; i < kSplit; i += THREADS) split[i] = i + 1 < kSplit ? sk[order[i + 1]] : ~0ull;
    __syncthreads();
    unsigned at[CAP / THREADS];  // bin << 16 | rank in the bin
#pragma unroll
    for (int u = 0; u < CAP / THREADS; ++u) {
      const int i = u * THREADS + tid;
      at[u] = 0;
      if (i < n) {
        const unsigned d = gba_range_digit(split, kSplitBits, sk[i]);
        at[u] = d << 16 | atomicAdd(&cnt[d], 1u);
      }
    }
    __syncthreads();
    if (tid < 32) {  // counts to starts, by one warp
      unsigned c[kSplit / 32], sum = 0;
#pragma unroll
      for (int u = 0; u < kSplit / 32; ++u) {
        c[u] = cnt[tid * (kSplit / 32) + u];
        sum += c[u];
      }
      unsigned x = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(~0u, x, o);
        if (tid >= o) x += y;
      }
      unsigned s = x - sum;
#pragma unroll
      for (int u = 0; u < kSplit / 32; ++u) {
        cnt[tid * (kSplit / 32) + u] = s;
        s += c[u];
      }
      if (tid == 31) cnt[kSplit] = s;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < CAP / THREADS; ++u) {
      const int i = u * THREADS + tid;
      if (i < n) bk[cnt[at[u] >> 16] + (at[u] & 0xffffu)] = (unsigned short)i;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < CAP / THREADS; ++u) {
      const int i = u * THREADS + tid;
      if (i < n) place(i, cnt[at[u] >> 16], cnt[(at[u] >> 16) + 1]);
    }
    __syncthreads();
  }
  // key i's place among the keys of its bin, bk[b..e)
  __device__ __forceinline__ void place(int i, unsigned b, unsigned e) const {
    const unsigned long long k = sk[i];
    unsigned r = b;
    for (unsigned j = b; j < e; ++j) {
      const unsigned o = bk[j];
      const unsigned long long ko = sk[o];
      r += ko < k || (ko == k && int(o) < i);
    }
    order[r] = (unsigned short)i;
  }
  __device__ __forceinline__ void run(int n) const {
    constexpr int kPer = CAP / THREADS;
    constexpr int kBinsPer = (1 << BINS) / THREADS;
    __shared__ unsigned long long s_lo[THREADS / 32], s_hi[THREADS / 32];
    __shared__ unsigned s_w[THREADS / 32];
    __shared__ unsigned s_most;
    const int tid = threadIdx.x;
    const unsigned lane = lane_id(), warp = tid >> 5;
    unsigned long long lo = ~0ull, hi = 0ull;
    for (int i = tid; i < n; i += THREADS) {
      const unsigned long long k = sk[i];
      lo = k < lo ? k : lo;
      hi = k > hi ? k : hi;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const unsigned long long a = __shfl_xor_sync(~0u, lo, o), b = __shfl_xor_sync(~0u, hi, o);
      lo = a < lo ? a : lo;
      hi = b > hi ? b : hi;
    }
    if (lane == 0) {
      s_lo[warp] = lo;
      s_hi[warp] = hi;
    }
    if (tid == 0) s_most = 0;
    for (int i = tid; i <= (1 << BINS); i += THREADS) cnt[i] = 0;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
      lo = s_lo[w] < lo ? s_lo[w] : lo;
      hi = s_hi[w] > hi ? s_hi[w] : hi;
    }
    const int len = n > 0 ? 64 - __clzll((long long)(hi - lo)) : 0;
    const int sh = len > BINS ? len - BINS : 0;
    unsigned rank[kPer], most = 0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = u * THREADS + tid;
      rank[u] = 0;
      if (i < n) rank[u] = atomicAdd(&cnt[unsigned((sk[i] - lo) >> sh)], 1u);
      most = rank[u] > most ? rank[u] : most;
    }
    most = __reduce_max_sync(~0u, most);
    if (lane == 0 && most) atomicMax(&s_most, most);
    __syncthreads();
    if (s_most >= kBinMost) {
      bunched(n);
      return;
    }
    // counts to starts
    unsigned c[kBinsPer], sum = 0;
#pragma unroll
    for (int u = 0; u < kBinsPer; ++u) {
      c[u] = cnt[tid * kBinsPer + u];
      sum += c[u];
    }
    unsigned x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(~0u, x, o);
      if (lane >= unsigned(o)) x += y;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    unsigned run_at = x - sum;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) run_at += w < int(warp) ? s_w[w] : 0u;
#pragma unroll
    for (int u = 0; u < kBinsPer; ++u) {
      cnt[tid * kBinsPer + u] = run_at;
      run_at += c[u];
    }
    if (tid == THREADS - 1) cnt[1 << BINS] = run_at;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = u * THREADS + tid;
      if (i < n) bk[cnt[unsigned((sk[i] - lo) >> sh)] + rank[u]] = (unsigned short)i;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = u * THREADS + tid;
      if (i >= n) continue;
      const unsigned bin = unsigned((sk[i] - lo) >> sh);
      place(i, cnt[bin], cnt[bin + 1]);
    }
    __syncthreads();
  }
};

__device__ __forceinline__ unsigned long long sort_key(const void* keys, int key64, int64_t i, unsigned long long flip) {
  return (key64 ? __ldg(static_cast<const unsigned long long*>(keys) + i)
                : (unsigned long long)__ldg(static_cast<const unsigned*>(keys) + i)) ^
         flip;
}

// splitters of segment blockIdx.x (rows [offs[x], offs[x + 1]), or [0, n) when
// offs is null) from an evenly spaced sample of its keys
__global__ void __launch_bounds__(kSampleThreads) k_sort_split(const void* keys, int key64, unsigned long long flip,
                                                               int64_t n, const unsigned long long* offs, int bits,
                                                               unsigned long long* split) {
  extern __shared__ __align__(16) unsigned char sm[];
  const CtaOrder<kSampleCap, kSampleThreads, kSampleBins> s(sm);
  const int64_t b = offs ? int64_t(offs[blockIdx.x]) : 0, e = offs ? int64_t(offs[blockIdx.x + 1]) : n;
  const int64_t rows = e - b;
  const int want = kSamplePer << bits < kSampleCap ? kSamplePer << bits : kSampleCap;
  const int m = int(rows < want ? rows : want);
  for (int i = threadIdx.x; i < m; i += kSampleThreads) s.sk[i] = sort_key(keys, key64, b + rows * i / m, flip);
  __syncthreads();
  s.run(m);
  const int nb = 1 << bits;
  for (int i = threadIdx.x; i < nb; i += kSampleThreads)
    split[(size_t(blockIdx.x) << bits) + i] =
        m > 0 && i < nb - 1 ? s.sk[s.order[(i + 1) * m >> bits]] : ~0ull;
}

struct SortHistArgs {
  const void* keys;
  int key64;
  unsigned long long flip;
  int64_t n;
  int bits, nseg;                  // nseg = 0: one segment [0, n)
  int T;                           // rows per tile (tile_prefix's)
  const unsigned long long* offs;  // segment bounds
  const unsigned* tile_prefix;
  const unsigned long long* split;
  unsigned long long* hist;        // [segment][2^bits]
};

// A CTA takes consecutive tiles, so it reloads splitters and adds its counts
// to the segment's once per segment it meets.
__global__ void __launch_bounds__(512) k_sort_hist(SortHistArgs a) {
  __shared__ unsigned long long split[1 << kLevelBits];
  __shared__ unsigned cnt[1 << kLevelBits];
  const int nb = 1 << a.bits, tid = threadIdx.x;
  const int64_t ntiles = a.nseg > 0 ? int64_t(a.tile_prefix[a.nseg]) : (a.n + a.T - 1) / a.T;
  const int64_t per = (ntiles + gridDim.x - 1) / gridDim.x;
  const int64_t t0 = int64_t(blockIdx.x) * per, t1 = t0 + per < ntiles ? t0 + per : ntiles;
  int cur = -1;
  auto flush = [&]() {
    if (cur >= 0 && tid < nb && cnt[tid]) atomicAdd(&a.hist[(size_t(cur) << a.bits) + tid], (unsigned long long)cnt[tid]);
  };
  for (int64_t tile = t0; tile < t1; ++tile) {
    int seg = 0;
    int64_t r0 = tile * a.T, e = a.n;
    if (a.nseg > 0) {
      int lo = 0, hi = a.nseg - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (int64_t(a.tile_prefix[mid]) <= tile) lo = mid;
        else hi = mid - 1;
      }
      seg = lo;
      r0 = int64_t(a.offs[seg]) + (tile - int64_t(a.tile_prefix[seg])) * a.T;
      e = int64_t(a.offs[seg + 1]);
    }
    if (e > r0 + a.T) e = r0 + a.T;
    if (seg != cur) {
      __syncthreads();
      flush();
      __syncthreads();
      cur = seg;
      if (tid < nb) {
        cnt[tid] = 0;
        split[tid] = a.split[(size_t(seg) << a.bits) + tid];
      }
      __syncthreads();
    }
    for (int64_t r = r0 + tid; r < e; r += 4 * 512) {
      unsigned long long k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) k[u] = r + u * 512 < e ? sort_key(a.keys, a.key64, r + u * 512, a.flip) : 0ull;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const unsigned d = gba_range_digit(split, a.bits, k[u]);
        if (r + u * 512 < e) atomicAdd(&cnt[d], 1u);
      }
    }
  }
  __syncthreads();
  flush();
}

struct SortPlanArgs {
  int np;
  const unsigned long long* hist;
  unsigned long long* offs;     // np + 1
  unsigned long long* cursors;
  unsigned* tile_prefix;        // np + 1, or null
  int tile;                     // rows per tile of the next level
  unsigned long long cap;       // keys a bucket may hold (0: any number)
  unsigned* fail;
};

__global__ void __launch_bounds__(1024) k_sort_plan(SortPlanArgs a) {
  __shared__ unsigned long long s_n[32];
  __shared__ unsigned s_t[32];
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  unsigned long long rows = 0;
  unsigned tiles = 0;
  bool over = false;
  for (int base = 0; base < a.np; base += 1024) {
    const int p = base + int(threadIdx.x);
    const unsigned long long c = p < a.np ? a.hist[p] : 0ull;
    const unsigned t = a.tile_prefix ? unsigned((c + a.tile - 1) / a.tile) : 0u;
    over = over || (a.cap && c > a.cap);
    unsigned long long x = c;
    unsigned y = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long xx = __shfl_up_sync(~0u, x, o);
      const unsigned yy = __shfl_up_sync(~0u, y, o);
      if (lane >= unsigned(o)) {
        x += xx;
        y += yy;
      }
    }
    if (lane == 31) {
      s_n[warp] = x;
      s_t[warp] = y;
    }
    __syncthreads();
    unsigned long long before = rows + x - c;
    unsigned tbefore = tiles + y - t;
#pragma unroll
    for (int w = 0; w < 32; ++w) {
      before += w < int(warp) ? s_n[w] : 0ull;
      tbefore += w < int(warp) ? s_t[w] : 0u;
      rows += s_n[w];
      tiles += s_t[w];
    }
    if (p < a.np) {
      a.offs[p] = before;
      a.cursors[p] = before;
      if (a.tile_prefix) a.tile_prefix[p] = tbefore;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    a.offs[a.np] = rows;
    if (a.tile_prefix) a.tile_prefix[a.np] = tiles;
  }
  if (over) atomicOr(a.fail, 1u);
}

// where a bucket's rows come from and go to
struct SortRows {
  const void* keys;
  void* okeys;
  const void* cols[GBA_MAX_AGGS];
  void* ocols[GBA_MAX_AGGS];
  int ncols;
  int col8;  // 1: 8-byte columns, 0: 4-byte ones (group indices)
  int key64;
  int n;     // k_sort_small: groups
  unsigned long long flip;
};

// rows [b0, b0 + n), n <= kBucketCap, put in key order at the same place of
// the output (which may be the input: every column is staged before it is written)
__device__ __forceinline__ void sort_bucket(const SortRows& s, unsigned char* sm, int64_t b0, int n) {
  const CtaOrder<kBucketCap, kBucketThreads, kBucketBins> c(sm);
  const int tid = threadIdx.x;
  for (int i = tid; i < n; i += kBucketThreads)
    c.sk[i] = (s.key64 ? static_cast<const unsigned long long*>(s.keys)[b0 + i]
                       : (unsigned long long)static_cast<const unsigned*>(s.keys)[b0 + i]) ^
              s.flip;
  __syncthreads();
  c.run(n);
  for (int r = tid; r < n; r += kBucketThreads) {
    const unsigned long long k = c.sk[c.order[r]] ^ s.flip;
    if (s.key64) static_cast<unsigned long long*>(s.okeys)[b0 + r] = k;
    else static_cast<unsigned*>(s.okeys)[b0 + r] = unsigned(k);
  }
  for (int a = 0; a < s.ncols; ++a) {
    __syncthreads();
    for (int i = tid; i < n; i += kBucketThreads)
      c.sk[i] = s.col8 ? static_cast<const unsigned long long*>(s.cols[a])[b0 + i]
                       : (unsigned long long)static_cast<const unsigned*>(s.cols[a])[b0 + i];
    __syncthreads();
    for (int r = tid; r < n; r += kBucketThreads) {
      const unsigned long long v = c.sk[c.order[r]];
      if (s.col8) static_cast<unsigned long long*>(s.ocols[a])[b0 + r] = v;
      else static_cast<unsigned*>(s.ocols[a])[b0 + r] = unsigned(v);
    }
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kBucketThreads, 3) k_sort_buckets(SortRows s, const unsigned long long* offs, int nb,
                                                                 const unsigned* fail) {
  extern __shared__ __align__(16) unsigned char sm[];
  if (*fail) return;
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    const unsigned long long lo = offs[b], hi = offs[b + 1];
    if (hi > lo) sort_bucket(s, sm, int64_t(lo), int(hi - lo));
  }
}

// jobs of at most one bucket, one CTA each
__global__ void __launch_bounds__(kBucketThreads, 3) k_sort_small(const SortRows* jobs) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ SortRows s;
  const unsigned* src = reinterpret_cast<const unsigned*>(jobs + blockIdx.x);
  for (int w = threadIdx.x; w < int(sizeof(SortRows) / 4); w += kBucketThreads) reinterpret_cast<unsigned*>(&s)[w] = src[w];
  __syncthreads();
  sort_bucket(s, sm, 0, s.n);
}

__global__ void k_sort_iota(unsigned* idx, int64_t g) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < g; i += int64_t(gridDim.x) * blockDim.x)
    idx[i] = unsigned(i);
}

struct GatherCols {
  const unsigned long long* src[GBA_MAX_AGGS];
  unsigned long long* dst[GBA_MAX_AGGS];
  int n;
};

__global__ void __launch_bounds__(kSortThreads) k_sort_gather(GatherCols c, const unsigned* idx, int64_t g,
                                                              const unsigned* fail) {
  if (fail && *fail) return;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < g; i += int64_t(gridDim.x) * blockDim.x) {
    const unsigned j = __ldg(idx + i);
#pragma unroll
    for (int a = 0; a < GBA_MAX_AGGS; ++a)
      if (a < c.n) c.dst[a][i] = __ldg(c.src[a] + j);
  }
}

size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

size_t stage_bytes(bool key64) { return size_t(kSortTile) * ((key64 ? 8 : 4) + 4); }

struct SortLayout {
  size_t keys_alt, idx0, idx1, look, ctr, aggs, bytes;
};

SortLayout layout_for(const SortJob& j, size_t base) {
  const int64_t ntiles = (j.g + kSortTile - 1) / kSortTile;
  SortLayout L;
  size_t o = base;
  L.keys_alt = o;  o += a256(size_t(j.g) * (j.key64 ? 8 : 4));
  L.idx0 = o;      o += a256(size_t(j.g) * 4);
  L.idx1 = o;      o += a256(size_t(j.g) * 4);
  L.look = o;      o += a256(size_t(ntiles) * 256 * 8);
  L.ctr = o;       o += 256;  // one tile counter per pass
  L.aggs = o;      o += a256(size_t(j.g) * 8) * size_t(j.nagg);
  L.bytes = o - base;
  return L;
}

}  // namespace

// The least-significant-digit sort of the jobs in `todo`; one host round trip
// for their key ranges and one at the end.
static gba_status sort_lsd(gba_context* ctx, const SortJob* jobs, const std::vector<int>& todo, cudaStream_t s) {
  if (todo.empty()) return GBA_OK;
  size_t per_job = 0;
  for (int j : todo) per_job = std::max(per_job, layout_for(jobs[j], 0).bytes);
  const int nt = int(todo.size());
  // front of the workspace: every job's digit counts, group count and pass mask
  const size_t o_hist = 0, o_g = a256(size_t(nt) * 8 * 256 * 4), o_mask = o_g + a256(size_t(nt) * 8);
  const size_t front = o_mask + a256(size_t(nt) * 4);
  gba_status st = gba_ws_reserve(ctx, front + per_job, s);
  if (st != GBA_OK) return st;
  st = gba_small_reserve(ctx, std::max<size_t>(ctx->d_small_bytes, 64 + size_t(nt) * 4));
  if (st != GBA_OK) return st;
  static const cudaError_t smem_ok = [] {
    cudaError_t e = gba_allow_max_smem(k_sort_pass<true>);
    return e != cudaSuccess ? e : gba_allow_max_smem(k_sort_pass<false>);
  }();
  GBA_CUDA_TRY(ctx, smem_ok);
  unsigned char* W = static_cast<unsigned char*>(ctx->ws);
  unsigned* d_hist = reinterpret_cast<unsigned*>(W + o_hist);
  int64_t* d_g = reinterpret_cast<int64_t*>(W + o_g);
  unsigned* d_mask = reinterpret_cast<unsigned*>(W + o_mask);
  unsigned* d_flags = reinterpret_cast<unsigned*>(ctx->d_small);
  std::vector<int64_t> gs(nt);
  for (int t = 0; t < nt; ++t) gs[t] = jobs[todo[t]].g;
  GBA_CUDA_TRY(ctx, cudaMemsetAsync(d_hist, 0, size_t(nt) * 8 * 256 * 4, s));
  GBA_CUDA_TRY(ctx, cudaMemcpyAsync(d_g, gs.data(), size_t(nt) * 8, cudaMemcpyHostToDevice, s));
  GBA_CUDA_TRY(ctx, cudaMemsetAsync(d_flags, 0, 4, s));
  int launches = 0;
  bool any64 = false;
  for (int t = 0; t < nt; ++t) {
    const SortJob& j = jobs[todo[t]];
    const unsigned long long flip = j.key_signed ? (j.key64 ? 1ull << 63 : 1ull << 31) : 0ull;
    const int grid = int(std::min<int64_t>(int64_t(ctx->sms) * 4, (j.g + kSortThreads - 1) / kSortThreads));
    if (j.key64) k_sort_prep<true><<<grid, kSortThreads, 0, s>>>(j.keys, j.g, flip, d_hist + size_t(t) * 2048);
    else k_sort_prep<false><<<grid, kSortThreads, 0, s>>>(j.keys, j.g, flip, d_hist + size_t(t) * 2048);
    GBA_CUDA_TRY(ctx, cudaGetLastError());
    any64 = any64 || j.key64;
    ++launches;
  }
  // 32-bit jobs count 4 positions, 64-bit ones 8: the mask kernel is told the
  // larger and a 32-bit job's positions 4..7 hold zero counts (never "all")
  k_sort_mask<<<nt, kSortThreads, 0, s>>>(d_hist, d_g, any64 ? 8 : 4, d_mask);
  GBA_CUDA_TRY(ctx, cudaGetLastError());
  ++launches;
  GBA_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_small + 64, d_mask, size_t(nt) * 4, cudaMemcpyDeviceToHost, s));
  GBA_CUDA_TRY(ctx, cudaStreamSynchronize(s));
  std::vector<unsigned> mask(nt);
  std::memcpy(mask.data(), ctx->h_small + 64, size_t(nt) * 4);

  const size_t jb = front;
  for (int t = 0; t < nt; ++t) {
    const SortJob& j = jobs[todo[t]];
    const unsigned m = mask[t] & (j.key64 ? 0xffu : 0xfu);
    if (m == 0) continue;
    const unsigned long long flip = j.key_signed ? (j.key64 ? 1ull << 63 : 1ull << 31) : 0ull;
    const SortLayout L = layout_for(j, jb);
    const int64_t ntiles = (j.g + kSortTile - 1) / kSortTile;
    void* alt = W + L.keys_alt;
    unsigned* idxb[2] = {reinterpret_cast<unsigned*>(W + L.idx0), reinterpret_cast<unsigned*>(W + L.idx1)};
    unsigned* ctr = reinterpret_cast<unsigned*>(W + L.ctr);
    GBA_CUDA_TRY(ctx, cudaMemsetAsync(ctr, 0, 8 * 4, s));
    void* cur = j.keys;
    const unsigned* idx_cur = nullptr;
    int np = 0;
    for (int p = 0; p < 8; ++p) {
      if (!(m >> p & 1u)) continue;
      PassArgs a;
      a.keys_in = cur;
      a.idx_in = idx_cur;
      a.keys_out = cur == j.keys ? alt : j.keys;
      a.idx_out = idxb[np & 1];
      a.g = j.g;
      a.flip = flip;
      a.shift = 8 * p;
      a.hist = d_hist + size_t(t) * 2048 + size_t(p) * 256;
      a.look = reinterpret_cast<unsigned long long*>(W + L.look);
      a.tile_ctr = ctr + p;
      a.flags = d_flags;
      GBA_CUDA_TRY(ctx, cudaMemsetAsync(a.look, 0, size_t(ntiles) * 256 * 8, s));
      if (j.key64) k_sort_pass<true><<<unsigned(ntiles), kSortThreads, stage_bytes(true), s>>>(a);
      else k_sort_pass<false><<<unsigned(ntiles), kSortThreads, stage_bytes(false), s>>>(a);
      GBA_CUDA_TRY(ctx, cudaGetLastError());
      ++launches;
      ++np;
      cur = a.keys_out;
      idx_cur = a.idx_out;
    }
    if (cur != j.keys)
      GBA_CUDA_TRY(ctx, cudaMemcpyAsync(j.keys, cur, size_t(j.g) * (j.key64 ? 8 : 4), cudaMemcpyDeviceToDevice, s));
    if (j.nagg > 0) {
      GatherCols c{};
      c.n = j.nagg;
      for (int a = 0; a < j.nagg; ++a) {
        unsigned long long* tmp = reinterpret_cast<unsigned long long*>(W + L.aggs + size_t(a) * a256(size_t(j.g) * 8));
        GBA_CUDA_TRY(ctx, cudaMemcpyAsync(tmp, j.aggs[a], size_t(j.g) * 8, cudaMemcpyDeviceToDevice, s));
        c.src[a] = tmp;
        c.dst[a] = j.aggs[a];
      }
      const int grid = int(std::min<int64_t>(int64_t(ctx->sms) * 8, (j.g + kSortThreads - 1) / kSortThreads));
      k_sort_gather<<<grid, kSortThreads, 0, s>>>(c, idx_cur, j.g, nullptr);
      GBA_CUDA_TRY(ctx, cudaGetLastError());
      ++launches;
    }
  }
  GBA_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_small, d_flags, 4, cudaMemcpyDeviceToHost, s));
  GBA_CUDA_TRY(ctx, cudaStreamSynchronize(s));
  ctx->stats.kernel_launches += launches;
  if (*reinterpret_cast<unsigned*>(ctx->h_small) & GBA_FLAG_WAIT_TIMEOUT) {
    ctx->err = "sort_output: a bounded look-back wait timed out";
    return GBA_ERR_TIMEOUT;
  }
  return GBA_OK;
}

// Splitter bits of a job's two levels (b2 = 0: one level); false: too many
// groups for them.  64 sampled keys per bucket keep a bucket under twice its
// mean (chance of one that is not: 3e-9); at 8 bits a level, 32 samples, the
// mean is at most a third of what a bucket may hold.
static bool sample_levels(int64_t g, int* b1, int* b2) {
  auto bits_for = [&](int64_t per) {
    int b = 1;
    while ((g + per - 1) / per > (int64_t(1) << b)) ++b;
    return b;
  };
  int b = bits_for(kBucketTarget);
  if (b > 2 * (kLevelBits - 1)) b = bits_for(kBucketCap / 3);
  if (b > 2 * kLevelBits) return false;
  *b1 = b <= kLevelBits - 1 ? b : b / 2;
  *b2 = b - *b1;
  return true;
}

// Enqueues the sample sort of one job in the workspace at `base` (null: only
// sizes it); *bytes: the workspace it takes.
static gba_status sort_sample(gba_context* ctx, const SortJob& j, unsigned char* base, size_t* bytes, unsigned* d_fail,
                              int* launches, cudaStream_t s) {
  int b1 = 0, b2 = 0;
  sample_levels(j.g, &b1, &b2);
  const size_t np1 = size_t(1) << b1, np = size_t(1) << (b1 + b2), g = size_t(j.g);
  // up to 4 aggregates travel with their key; more are gathered through the
  // group's index afterwards
  const bool direct = j.nagg <= GBA_MAX_COLS;
  size_t o = 0;
  auto take = [&](size_t b) {
    const size_t at = o;
    o += a256(b);
    return at;
  };
  const size_t kb = j.key64 ? 8 : 4, cb = direct ? 8 : 4;
  const int nc = direct ? j.nagg : 1;
  size_t rows[2][1 + GBA_MAX_COLS];
  for (int x = 0; x < (b2 ? 2 : 1); ++x) {
    rows[x][0] = take(g * kb);
    for (int c = 0; c < nc; ++c) rows[x][1 + c] = take(g * cb);
  }
  const size_t o_idx = direct ? 0 : take(g * 4), o_idx_out = direct ? 0 : take(g * 4);
  const size_t o_agg = direct ? 0 : take(size_t(j.nagg) * a256(g * 8));
  const size_t o_hist1 = take(8 * np1), o_hist2 = take(8 * np);  // cleared together
  const size_t hist_bytes = o - o_hist1;
  const size_t o_split1 = take(8 * np1), o_split2 = take(8 * np);
  const size_t o_offs1 = take(8 * (np1 + 1)), o_offs2 = take(8 * (np + 1));
  const size_t o_cur1 = take(8 * np1), o_cur2 = take(8 * np);
  const size_t o_tiles = take(4 * (np1 + 1));
  *bytes = o;
  if (!base) return GBA_OK;
  auto at = [&](size_t x) { return reinterpret_cast<unsigned long long*>(base + x); };
  const unsigned long long flip = j.key_signed ? (j.key64 ? 1ull << 63 : 1ull << 31) : 0ull;
  GBA_CUDA_TRY(ctx, cudaMemsetAsync(base + o_hist1, 0, hist_bytes, s));

  QDesc in{};
  in.keys = j.keys;
  in.n = j.g;
  in.key64 = j.key64;
  in.ncols = nc;
  for (int c = 0; c < nc; ++c) {
    in.col_type[c] = direct ? GBA_I64 : GBA_U32;
    in.cols[c] = direct ? static_cast<const void*>(j.aggs[c]) : base + o_idx;
  }
  const int wide_grid = int(std::min<int64_t>(int64_t(ctx->sms) * 8, (j.g + 255) / 256));
  if (!direct) {
    k_sort_iota<<<wide_grid, 256, 0, s>>>(reinterpret_cast<unsigned*>(base + o_idx), j.g);
    ++*launches;
  }
  int th[2] = {512, 512};
  const int T1 = gba_part_tile_rows(in, b1, 0, true, ctx->max_smem_optin, &th[0]);
  const int T2 = b2 ? gba_part_tile_rows(in, b2, int(np1), true, ctx->max_smem_optin, &th[1]) : 0;
  for (int x = 0; x < (b2 ? 2 : 1); ++x) {
    const int bits = x ? b2 : b1, nseg = x ? int(np1) : 0, T = x ? T2 : T1;
    unsigned long long* split = at(x ? o_split2 : o_split1);
    k_sort_split<<<x ? unsigned(np1) : 1u, kSampleThreads, order_smem(kSampleCap, kSampleBins), s>>>(
        in.keys, j.key64, flip, j.g, x ? at(o_offs1) : nullptr, bits, split);
    GBA_CUDA_TRY(ctx, cudaGetLastError());
    SortHistArgs h{};
    h.keys = in.keys;
    h.key64 = j.key64;
    h.flip = flip;
    h.n = j.g;
    h.bits = bits;
    h.nseg = nseg;
    h.T = T;
    h.offs = at(o_offs1);
    h.tile_prefix = reinterpret_cast<unsigned*>(base + o_tiles);
    h.split = split;
    h.hist = at(x ? o_hist2 : o_hist1);
    const int64_t tiles = j.g / T + 1 + nseg;
    k_sort_hist<<<unsigned(std::min<int64_t>(tiles, int64_t(ctx->sms) * 4)), 512, 0, s>>>(h);
    GBA_CUDA_TRY(ctx, cudaGetLastError());
    SortPlanArgs pl{};
    pl.np = int(x ? np : np1);
    pl.hist = h.hist;
    pl.offs = at(x ? o_offs2 : o_offs1);
    pl.cursors = at(x ? o_cur2 : o_cur1);
    pl.tile_prefix = !x && b2 ? reinterpret_cast<unsigned*>(base + o_tiles) : nullptr;
    pl.tile = !x && b2 ? T2 : 1;
    pl.cap = x || !b2 ? kBucketCap : 0;
    pl.fail = d_fail;
    k_sort_plan<<<1, 1024, 0, s>>>(pl);
    GBA_CUDA_TRY(ctx, cudaGetLastError());
    PartPass pp{};
    pp.in = in;
    pp.out = in;
    pp.out.keys = base + rows[x][0];
    for (int c = 0; c < nc; ++c) pp.out.cols[c] = base + rows[x][1 + c];
    pp.n = j.g;
    pp.bits = bits;
    pp.nseg = nseg;
    pp.T = T;
    pp.threads = th[x];
    pp.offs = at(o_offs2);
    pp.tile_prefix = h.tile_prefix;
    pp.cursors = pl.cursors;
    pp.flags = reinterpret_cast<unsigned*>(ctx->d_small);
    pp.splitters = split;
    pp.flip = flip;
    pp.fail = d_fail;
    GBA_CUDA_TRY(ctx, gba_launch_part_scatter(pp, int(std::min<int64_t>(tiles, ctx->sms * (1024 / th[x]))), s));
    *launches += 4;
    in = pp.out;
  }
  SortRows r{};
  r.keys = in.keys;
  r.okeys = j.keys;
  r.ncols = nc;
  r.col8 = direct;
  r.key64 = j.key64;
  r.flip = flip;
  for (int c = 0; c < nc; ++c) {
    r.cols[c] = in.cols[c];
    r.ocols[c] = direct ? static_cast<void*>(j.aggs[c]) : base + o_idx_out;
  }
  k_sort_buckets<<<unsigned(std::min<int64_t>(int64_t(np), int64_t(ctx->sms) * 3)), kBucketThreads,
                   order_smem(kBucketCap, kBucketBins), s>>>(r, at(b2 ? o_offs2 : o_offs1), int(np), d_fail);
  GBA_CUDA_TRY(ctx, cudaGetLastError());
  ++*launches;
  if (!direct) {
    GatherCols c{};
    c.n = j.nagg;
    for (int a = 0; a < j.nagg; ++a) {
      unsigned char* tmp = base + o_agg + size_t(a) * a256(g * 8);
      GBA_CUDA_TRY(ctx, cudaMemcpyAsync(tmp, j.aggs[a], g * 8, cudaMemcpyDeviceToDevice, s));
      c.src[a] = reinterpret_cast<unsigned long long*>(tmp);
      c.dst[a] = j.aggs[a];
    }
    k_sort_gather<<<wide_grid, kSortThreads, 0, s>>>(c, reinterpret_cast<unsigned*>(base + o_idx_out), j.g, d_fail);
    GBA_CUDA_TRY(ctx, cudaGetLastError());
    ++*launches;
  }
  return GBA_OK;
}

gba_status gba_sort_groups(gba_context* ctx, const SortJob* jobs, int njobs, cudaStream_t s) {
  std::vector<int> small, sample, lsd;
  size_t most = 0;
  for (int j = 0; j < njobs; ++j) {
    int b1, b2;
    if (jobs[j].g <= 1) continue;
    if (jobs[j].g >= (int64_t(1) << 32)) {
      ctx->err = "sort_output: more than 2^32 - 1 groups";
      return GBA_ERR_INVALID_ARG;
    }
    if (jobs[j].g <= kBucketCap) small.push_back(j);
    else if (sample_levels(jobs[j].g, &b1, &b2)) {
      size_t bytes;
      int unused = 0;
      sort_sample(ctx, jobs[j], nullptr, &bytes, nullptr, &unused, s);
      most = std::max(most, bytes);
      sample.push_back(j);
    } else lsd.push_back(j);
  }
  if (!small.empty() || !sample.empty()) {
    // front of the workspace: the small jobs' descriptors, then one failure
    // word per sampled job (they share the rest, one after another)
    const size_t o_fail = a256(small.size() * sizeof(SortRows)), front = o_fail + a256(4 * sample.size() + 4);
    gba_status st = gba_ws_reserve(ctx, front + most, s);
    if (st != GBA_OK) return st;
    st = gba_small_reserve(ctx, std::max<size_t>(ctx->d_small_bytes, 64 + 4 * sample.size()));
    if (st != GBA_OK) return st;
    static const cudaError_t smem_ok = [] {
      cudaError_t e = gba_allow_max_smem(k_sort_split);
      if (e == cudaSuccess) e = gba_allow_max_smem(k_sort_buckets);
      return e != cudaSuccess ? e : gba_allow_max_smem(k_sort_small);
    }();
    GBA_CUDA_TRY(ctx, smem_ok);
    unsigned char* W = static_cast<unsigned char*>(ctx->ws);
    unsigned* d_fail = reinterpret_cast<unsigned*>(W + o_fail);
    int launches = 0;
    GBA_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_small, 0, 4, s));
    std::vector<SortRows> rows(small.size());
    if (!small.empty()) {
      for (size_t t = 0; t < small.size(); ++t) {
        const SortJob& j = jobs[small[t]];
        SortRows& r = rows[t];
        r = SortRows{};
        r.keys = r.okeys = j.keys;
        r.ncols = j.nagg;
        r.col8 = 1;
        r.key64 = j.key64;
        r.n = int(j.g);
        r.flip = j.key_signed ? (j.key64 ? 1ull << 63 : 1ull << 31) : 0ull;
        for (int a = 0; a < j.nagg; ++a) r.cols[a] = r.ocols[a] = j.aggs[a];
      }
      GBA_CUDA_TRY(ctx, cudaMemcpyAsync(W, rows.data(), rows.size() * sizeof(SortRows), cudaMemcpyHostToDevice, s));
      k_sort_small<<<unsigned(rows.size()), kBucketThreads, order_smem(kBucketCap, kBucketBins), s>>>(
          reinterpret_cast<const SortRows*>(W));
      GBA_CUDA_TRY(ctx, cudaGetLastError());
      ++launches;
    }
    if (!sample.empty()) {
      GBA_CUDA_TRY(ctx, cudaMemsetAsync(d_fail, 0, 4 * sample.size(), s));
      for (size_t t = 0; t < sample.size(); ++t) {
        size_t bytes;
        st = sort_sample(ctx, jobs[sample[t]], W + front, &bytes, d_fail + t, &launches, s);
        if (st != GBA_OK) return st;
      }
      GBA_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_small + 64, d_fail, 4 * sample.size(), cudaMemcpyDeviceToHost, s));
    }
    GBA_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_small, ctx->d_small, 4, cudaMemcpyDeviceToHost, s));
    GBA_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    ctx->stats.kernel_launches += launches;
    if (*reinterpret_cast<unsigned*>(ctx->h_small) & GBA_FLAG_WAIT_TIMEOUT) {
      ctx->err = "sort_output: a bounded wait for a staged tile timed out";
      return GBA_ERR_TIMEOUT;
    }
    // a job whose sample missed its keys' distribution was left as it was
    for (size_t t = 0; t < sample.size(); ++t)
      if (reinterpret_cast<const unsigned*>(ctx->h_small + 64)[t]) lsd.push_back(sample[t]);
  }
  return sort_lsd(ctx, jobs, lsd, s);
}
