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
//                   and aggregates to their final place (k_sort_big_buckets:
//                   the few buckets of two-level jobs of twice the size)
// One level for up to 2^18 groups, two levels above.  Jobs of up to one bucket
// are all sorted in place by one launch (k_sort_small).
//
// Bytes per group of b bytes: 2 (b + key) per level and 2 b for the buckets,
// against 2 (key + 4) for each of up to 8 passes plus the random gather of a
// least-significant-digit sort over (key, index) pairs.  Measured (us, that
// sort / this one): 16.8M int64 groups with 2 aggregates 2714 / 1190, 9.9M with
// 1 aggregate 1390 / 695; 48 queries of up to 2^17 groups, sorted in one launch
// per step, 4200 / 90.  The bucket kernel (2.1 TB/s on the 16.8M groups) is
// bound by its barriers and shared-memory round trips at 3 CTAs of 512 threads
// per SM (2 CTAs: 500 against 380 us), the count by the binary search's
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

// All kernels of the sample sort take an array of jobs, one per blockIdx.y.
struct SortSplitArgs {
  const void* keys;
  int key64;
  unsigned long long flip;
  int64_t n;
  int bits, nseg;                  // nseg = 0: one segment [0, n)
  int sample;                      // keys to sample (at most kSampleCap)
  const unsigned long long* offs;  // segment bounds
  unsigned long long* split;       // [segment][2^bits]
};

// splitters of segment blockIdx.x from an evenly spaced sample of its keys
__global__ void __launch_bounds__(kSampleThreads) k_sort_split(const SortSplitArgs* jobs) {
  extern __shared__ __align__(16) unsigned char sm[];
  const SortSplitArgs a = jobs[blockIdx.y];
  if (int(blockIdx.x) >= (a.nseg > 0 ? a.nseg : 1)) return;
  const void* keys = a.keys;
  const int key64 = a.key64, bits = a.bits;
  const unsigned long long flip = a.flip;
  const int64_t n = a.n;
  const unsigned long long* offs = a.nseg > 0 ? a.offs : nullptr;
  unsigned long long* split = a.split;
  const CtaOrder<kSampleCap, kSampleThreads, kSampleBins> s(sm);
  const int64_t b = offs ? int64_t(offs[blockIdx.x]) : 0, e = offs ? int64_t(offs[blockIdx.x + 1]) : n;
  const int64_t rows = e - b;
  const int m = int(rows < a.sample ? rows : a.sample);
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
__global__ void __launch_bounds__(512) k_sort_hist(const SortHistArgs* jobs) {
  const SortHistArgs a = jobs[blockIdx.y];
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
    const unsigned long long flip = a.flip;
    const int bits = a.bits, rows = int(e - r0);
    auto count = [&](auto keys) {
      for (int r = tid; r < rows; r += 8 * 512) {
        unsigned long long k[8];
        unsigned d[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) k[u] = r + u * 512 < rows ? __ldg(keys + r + u * 512) ^ flip : 0ull;
        gba_range_digits<8>(split, bits, k, d);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (r + u * 512 < rows) atomicAdd(&cnt[d[u]], 1u);
      }
    };
    if (a.key64) count(static_cast<const unsigned long long*>(a.keys) + r0);
    else count(static_cast<const unsigned*>(a.keys) + r0);
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

__global__ void __launch_bounds__(1024) k_sort_plan(const SortPlanArgs* jobs) {
  const SortPlanArgs a = jobs[blockIdx.y];
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

// rows [b0, b0 + n), n <= CAP, put in key order at the same place of
// the output (which may be the input: every column is staged before it is written)
template <bool K64, bool COL8, int CAP = kBucketCap, int THREADS = kBucketThreads, int BINS = kBucketBins>
__device__ __forceinline__ void sort_bucket(const SortRows& s, unsigned char* sm, int64_t b0, int n) {
  const CtaOrder<CAP, THREADS, BINS> c(sm);
  const int tid = threadIdx.x;
  for (int i = tid; i < n; i += THREADS)
    c.sk[i] = (K64 ? static_cast<const unsigned long long*>(s.keys)[b0 + i]
                   : (unsigned long long)static_cast<const unsigned*>(s.keys)[b0 + i]) ^
              s.flip;
  __syncthreads();
  c.run(n);
  for (int r = tid; r < n; r += THREADS) {
    const unsigned long long k = c.sk[c.order[r]] ^ s.flip;
    if (K64) static_cast<unsigned long long*>(s.okeys)[b0 + r] = k;
    else static_cast<unsigned*>(s.okeys)[b0 + r] = unsigned(k);
  }
  for (int a = 0; a < s.ncols; ++a) {
    const void* col = s.cols[a];
    void* ocol = s.ocols[a];
    __syncthreads();
    for (int i = tid; i < n; i += THREADS)
      c.sk[i] = COL8 ? static_cast<const unsigned long long*>(col)[b0 + i]
                     : (unsigned long long)static_cast<const unsigned*>(col)[b0 + i];
    __syncthreads();
    for (int r = tid; r < n; r += THREADS) {
      const unsigned long long v = c.sk[c.order[r]];
      if (COL8) static_cast<unsigned long long*>(ocol)[b0 + r] = v;
      else static_cast<unsigned*>(ocol)[b0 + r] = unsigned(v);
    }
  }
  __syncthreads();
}

// widths (compile time): dispatched once per CTA
template <typename F>
__device__ __forceinline__ void with_widths(const SortRows& s, F&& f) {
  if (s.key64) {
    if (s.col8) f(std::true_type{}, std::true_type{});
    else f(std::true_type{}, std::false_type{});
  } else {
    if (s.col8) f(std::false_type{}, std::true_type{});
    else f(std::false_type{}, std::false_type{});
  }
}

struct SortBucketArgs {
  SortRows rows;
  const unsigned long long* offs;
  int nb;
  const unsigned* fail;
};

__global__ void __launch_bounds__(kBucketThreads, 3) k_sort_buckets(const SortBucketArgs* jobs) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ __align__(8) SortBucketArgs s;
  const unsigned* src = reinterpret_cast<const unsigned*>(jobs + blockIdx.y);
  for (int w = threadIdx.x; w < int(sizeof(SortBucketArgs) / 4); w += kBucketThreads)
    reinterpret_cast<unsigned*>(&s)[w] = src[w];
  __syncthreads();
  if (*s.fail) return;
  with_widths(s.rows, [&](auto K, auto C) {
    for (int b = blockIdx.x; b < s.nb; b += gridDim.x) {
      const unsigned long long lo = s.offs[b], hi = s.offs[b + 1];
      if (hi > lo && hi - lo <= kBucketCap)
        sort_bucket<decltype(K)::value, decltype(C)::value>(s.rows, sm, int64_t(lo), int(hi - lo));
    }
  });
}

// the rare buckets of two-level jobs that are larger than kBucketCap
__global__ void __launch_bounds__(kSampleThreads) k_sort_big_buckets(const SortBucketArgs* jobs) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_big[kSampleThreads];
  __shared__ int s_n;
  const SortBucketArgs& s = jobs[blockIdx.y];
  if (*s.fail) return;
  // a thread looks at one bucket: the few large ones are listed, then sorted
  for (int base = int(blockIdx.x) * kSampleThreads; base < s.nb; base += int(gridDim.x) * kSampleThreads) {
    const int b = base + int(threadIdx.x);
    const bool big = b < s.nb && s.offs[b + 1] - s.offs[b] > kBucketCap;
    if (threadIdx.x == 0) s_n = 0;
    if (!__syncthreads_or(big)) continue;
    if (big) s_big[atomicAdd(&s_n, 1)] = b;
    __syncthreads();
    for (int i = 0; i < s_n; ++i) {
      const unsigned long long lo = s.offs[s_big[i]], hi = s.offs[s_big[i] + 1];
      with_widths(s.rows, [&](auto K, auto C) {
        sort_bucket<decltype(K)::value, decltype(C)::value, kSampleCap, kSampleThreads, kSampleBins>(
            s.rows, sm, int64_t(lo), int(hi - lo));
      });
    }
    __syncthreads();
  }
}

// jobs of at most one bucket, one CTA each
__global__ void __launch_bounds__(kBucketThreads, 3) k_sort_small(const SortRows* jobs) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ SortRows s;
  const unsigned* src = reinterpret_cast<const unsigned*>(jobs + blockIdx.x);
  for (int w = threadIdx.x; w < int(sizeof(SortRows) / 4); w += kBucketThreads) reinterpret_cast<unsigned*>(&s)[w] = src[w];
  __syncthreads();
  if (s.key64) sort_bucket<true, true>(s, sm, 0, s.n);
  else sort_bucket<false, true>(s, sm, 0, s.n);
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
// groups for them.  A bucket of s sampled keys outgrows x times its mean with a
// chance of about exp(-s (x - 1 - ln x)).  One level: s = 64, x = 2, 3e-9.  Two:
// a first-level segment of 128 sampled keys may be 1.27 times its mean, so a few
// buckets in 10^4 pass kBucketCap (k_sort_big_buckets takes them), and none
// twice that: x = 3, 1e-25.  At 8 bits a level (s = 32, segments up to 1.53
// times their mean, a mean of a third of kBucketCap) x = 4, 1e-22.
static bool sample_levels(int64_t g, int* b1, int* b2) {
  auto bits_for = [&](int64_t per) {
    int b = 1;
    while ((g + per - 1) / per > (int64_t(1) << b)) ++b;
    return b;
  };
  int b = bits_for(kBucketTarget);
  if (b <= kLevelBits - 1) {
    *b1 = b;
    *b2 = 0;
    return true;
  }
  if (b > 2 * (kLevelBits - 1)) b = bits_for(kBucketCap / 3);
  if (b > 2 * kLevelBits) return false;
  *b1 = b / 2;
  *b2 = b - *b1;
  return true;
}

namespace {

// One job of the sample sort: its shape and where its arrays are.
struct SampleJob {
  SortJob j;
  int b1, b2;
  bool direct;  // up to 4 aggregates travel with their key; more are gathered through the group's index
  int nc;       // columns that travel
  QDesc in;     // the level's input rows
  int T[2], th[2];
  size_t rows[2][1 + GBA_MAX_COLS];
  size_t idx, idx_out, agg, hist[2], split[2], offs[2], cur[2], tiles;

  size_t np(int x) const { return size_t(1) << (x ? b1 + b2 : b1); }
};

}  // namespace

// Enqueues the sample sort of the jobs todo[first, last) in the workspace from
// offset `front` on (dry: only sizes it); *bytes: the workspace they take.
// Every step is one launch for all of them.
static gba_status sort_sample(gba_context* ctx, const SortJob* jobs, const std::vector<int>& todo, size_t first,
                              size_t last, size_t front, bool dry, size_t* bytes, unsigned* d_fail, int* launches,
                              cudaStream_t s) {
  std::vector<SampleJob> v(last - first);
  const size_t nj = v.size();
  size_t o = front;
  auto take = [&](size_t b) {
    const size_t at = o;
    o += a256(b);
    return at;
  };
  // the counts come first: they are cleared together
  for (size_t t = 0; t < nj; ++t) {
    SampleJob& q = v[t];
    q.j = jobs[todo[first + t]];
    sample_levels(q.j.g, &q.b1, &q.b2);
    q.direct = q.j.nagg <= GBA_MAX_COLS;
    q.nc = q.direct ? q.j.nagg : 1;
    q.hist[0] = take(8 * q.np(0));
    q.hist[1] = q.b2 ? take(8 * q.np(1)) : 0;
  }
  const size_t hist_bytes = o - front;
  for (SampleJob& q : v) {
    const size_t g = size_t(q.j.g), kb = q.j.key64 ? 8 : 4, cb = q.direct ? 8 : 4;
    for (int x = 0; x < (q.b2 ? 2 : 1); ++x) {
      q.rows[x][0] = take(g * kb);
      for (int c = 0; c < q.nc; ++c) q.rows[x][1 + c] = take(g * cb);
      q.split[x] = take(8 * q.np(x));
      q.offs[x] = take(8 * (q.np(x) + 1));
      q.cur[x] = take(8 * q.np(x));
    }
    q.idx = q.direct ? 0 : take(g * 4);
    q.idx_out = q.direct ? 0 : take(g * 4);
    q.agg = q.direct ? 0 : take(size_t(q.j.nagg) * a256(g * 8));
    q.tiles = take(4 * (q.np(0) + 1));
  }
  // argument arrays
  const size_t o_args = o;
  const size_t a_split = take(2 * nj * sizeof(SortSplitArgs)), a_hist = take(2 * nj * sizeof(SortHistArgs));
  const size_t a_plan = take(2 * nj * sizeof(SortPlanArgs)), a_pass = take(2 * nj * sizeof(PartPass));
  const size_t a_bucket = take(nj * sizeof(SortBucketArgs));
  *bytes = o - front;
  if (dry) return GBA_OK;

  unsigned char* W = static_cast<unsigned char*>(ctx->ws);
  auto at = [&](size_t x) { return reinterpret_cast<unsigned long long*>(W + x); };
  std::vector<unsigned char> args(o - o_args);
  auto arg = [&](size_t x) { return args.data() + (x - o_args); };
  GBA_CUDA_TRY(ctx, cudaMemsetAsync(W + front, 0, hist_bytes, s));
  auto wide_grid = [&](int64_t g) { return int(std::min<int64_t>(int64_t(ctx->sms) * 8, (g + 255) / 256)); };
  for (SampleJob& q : v) {
    q.in = QDesc{};
    q.in.keys = q.j.keys;
    q.in.n = q.j.g;
    q.in.key64 = q.j.key64;
    q.in.ncols = q.nc;
    for (int c = 0; c < q.nc; ++c) {
      q.in.col_type[c] = q.direct ? GBA_I64 : GBA_U32;
      q.in.cols[c] = q.direct ? static_cast<const void*>(q.j.aggs[c]) : W + q.idx;
    }
    if (!q.direct) {
      k_sort_iota<<<wide_grid(q.j.g), 256, 0, s>>>(reinterpret_cast<unsigned*>(W + q.idx), q.j.g);
      GBA_CUDA_TRY(ctx, cudaGetLastError());
      ++*launches;
    }
  }
  // Per level: the jobs that have it, ordered so that one launch's scatter
  // passes (key width, columns, CTA shape) are consecutive.
  struct Pass {
    size_t begin, end;
    int64_t tiles;
  };
  std::vector<size_t> order[2];
  std::vector<Pass> passes[2];
  int64_t segs[2] = {1, 1}, tiles_most[2] = {0, 0};
  for (int x = 0; x < 2; ++x) {
    for (size_t t = 0; t < nj; ++t)
      if (x == 0 || v[t].b2) order[x].push_back(t);
    for (size_t t : order[x])
      v[t].T[x] = gba_part_tile_rows(v[t].in, x ? v[t].b2 : v[t].b1, x ? int(v[t].np(0)) : 0, true, ctx->max_smem_optin,
                                     &v[t].th[x]);
    auto cls = [&](size_t t) { return (v[t].j.key64 * 8 + v[t].nc) * 2 + (v[t].th[x] == 1024) + (v[t].direct ? 0 : 64); };
    std::stable_sort(order[x].begin(), order[x].end(), [&](size_t p, size_t q) { return cls(p) < cls(q); });
    for (size_t i = 0; i < order[x].size(); ++i) {
      const size_t t = order[x][i];
      const int64_t tiles = v[t].j.g / v[t].T[x] + 1 + (x ? int64_t(v[t].np(0)) : 0);
      if (i == 0 || cls(order[x][i - 1]) != cls(t)) passes[x].push_back(Pass{i, i, 0});
      passes[x].back().end = i + 1;
      passes[x].back().tiles = std::max(passes[x].back().tiles, tiles);
      tiles_most[x] = std::max(tiles_most[x], tiles);
      if (x) segs[1] = std::max<int64_t>(segs[1], int64_t(v[t].np(0)));
    }
  }
  for (int x = 0; x < 2; ++x)
    for (size_t i = 0; i < order[x].size(); ++i) {
      const size_t t = order[x][i], slot = size_t(x) * nj + i;
      SampleJob& q = v[t];
      const unsigned long long flip = q.j.key_signed ? (q.j.key64 ? 1ull << 63 : 1ull << 31) : 0ull;
      const int bits = x ? q.b2 : q.b1, nseg = x ? int(q.np(0)) : 0;
      SortSplitArgs sp{};
      sp.keys = q.in.keys;
      sp.key64 = q.j.key64;
      sp.flip = flip;
      sp.n = q.j.g;
      sp.bits = bits;
      sp.nseg = nseg;
      sp.sample = x == 0 && q.b2 ? kSampleCap : std::min(kSamplePer << bits, kSampleCap);
      sp.offs = x ? at(q.offs[0]) : nullptr;
      sp.split = at(q.split[x]);
      SortHistArgs h{};
      h.keys = q.in.keys;
      h.key64 = q.j.key64;
      h.flip = flip;
      h.n = q.j.g;
      h.bits = bits;
      h.nseg = nseg;
      h.T = q.T[x];
      h.offs = sp.offs;
      h.tile_prefix = reinterpret_cast<unsigned*>(W + q.tiles);
      h.split = sp.split;
      h.hist = at(q.hist[x]);
      const bool ends = x || !q.b2;  // the level whose buckets are sorted in shared memory
      SortPlanArgs pl{};
      pl.np = int(q.np(x));
      pl.hist = h.hist;
      pl.offs = at(q.offs[x]);
      pl.cursors = at(q.cur[x]);
      pl.tile_prefix = ends ? nullptr : reinterpret_cast<unsigned*>(W + q.tiles);
      pl.tile = ends ? 1 : q.T[1];
      pl.cap = !ends ? 0 : x ? kSampleCap : kBucketCap;
      pl.fail = d_fail + first + t;
      PartPass pp{};
      pp.in = q.in;
      pp.out = q.in;
      pp.out.keys = W + q.rows[x][0];
      for (int c = 0; c < q.nc; ++c) pp.out.cols[c] = W + q.rows[x][1 + c];
      pp.n = q.j.g;
      pp.bits = bits;
      pp.nseg = nseg;
      pp.T = q.T[x];
      pp.threads = q.th[x];
      pp.offs = x ? at(q.offs[1]) : nullptr;
      pp.tile_prefix = h.tile_prefix;
      pp.cursors = pl.cursors;
      pp.flags = reinterpret_cast<unsigned*>(ctx->d_small);
      pp.splitters = sp.split;
      pp.flip = flip;
      pp.fail = pl.fail;
      std::memcpy(arg(a_split) + slot * sizeof(sp), &sp, sizeof(sp));
      std::memcpy(arg(a_hist) + slot * sizeof(h), &h, sizeof(h));
      std::memcpy(arg(a_plan) + slot * sizeof(pl), &pl, sizeof(pl));
      std::memcpy(arg(a_pass) + slot * sizeof(pp), &pp, sizeof(pp));
      q.in = pp.out;
      if (!ends) continue;
      SortBucketArgs bk{};
      bk.rows.keys = q.in.keys;
      bk.rows.okeys = q.j.keys;
      bk.rows.ncols = q.nc;
      bk.rows.col8 = q.direct;
      bk.rows.key64 = q.j.key64;
      bk.rows.flip = flip;
      for (int c = 0; c < q.nc; ++c) {
        bk.rows.cols[c] = q.in.cols[c];
        bk.rows.ocols[c] = q.direct ? static_cast<void*>(q.j.aggs[c]) : W + q.idx_out;
      }
      bk.offs = at(q.offs[x]);
      bk.nb = int(q.np(x));
      bk.fail = pl.fail;
      std::memcpy(arg(a_bucket) + t * sizeof(bk), &bk, sizeof(bk));
    }
  GBA_CUDA_TRY(ctx, cudaMemcpyAsync(W + o_args, args.data(), args.size(), cudaMemcpyHostToDevice, s));
  // CTAs per job: `most` over all jobs, each at least one
  auto per_job = [&](int64_t want, int64_t most, size_t njobs) {
    return unsigned(std::max<int64_t>(1, std::min<int64_t>(want, (most + int64_t(njobs) - 1) / int64_t(njobs))));
  };
  for (int x = 0; x < 2; ++x) {
    const size_t n = order[x].size(), slot = size_t(x) * nj;
    if (n == 0) continue;
    k_sort_split<<<dim3(unsigned(segs[x]), unsigned(n)), kSampleThreads, order_smem(kSampleCap, kSampleBins), s>>>(
        reinterpret_cast<const SortSplitArgs*>(W + a_split) + slot);
    GBA_CUDA_TRY(ctx, cudaGetLastError());
    k_sort_hist<<<dim3(per_job(tiles_most[x], int64_t(ctx->sms) * 4, n), unsigned(n)), 512, 0, s>>>(
        reinterpret_cast<const SortHistArgs*>(W + a_hist) + slot);
    GBA_CUDA_TRY(ctx, cudaGetLastError());
    k_sort_plan<<<dim3(1, unsigned(n)), 1024, 0, s>>>(reinterpret_cast<const SortPlanArgs*>(W + a_plan) + slot);
    GBA_CUDA_TRY(ctx, cudaGetLastError());
    *launches += 3;
    for (const Pass& p : passes[x]) {
      const size_t np = p.end - p.begin;
      const PartPass* host = reinterpret_cast<const PartPass*>(arg(a_pass)) + slot + p.begin;
      GBA_CUDA_TRY(ctx, gba_launch_part_scatter_many(
                            host, reinterpret_cast<const PartPass*>(W + a_pass) + slot + p.begin, int(np),
                            int(per_job(p.tiles, int64_t(ctx->sms) * (1024 / host->threads), np)), s));
      ++*launches;
    }
  }
  int64_t nb_most = 1;
  for (const SampleJob& q : v) nb_most = std::max<int64_t>(nb_most, int64_t(q.np(q.b2 ? 1 : 0)));
  k_sort_buckets<<<dim3(per_job(nb_most, int64_t(ctx->sms) * 3, nj), unsigned(nj)), kBucketThreads,
                   order_smem(kBucketCap, kBucketBins), s>>>(reinterpret_cast<const SortBucketArgs*>(W + a_bucket));
  GBA_CUDA_TRY(ctx, cudaGetLastError());
  ++*launches;
  if (!order[1].empty()) {
    k_sort_big_buckets<<<dim3(per_job(nb_most, ctx->sms, nj), unsigned(nj)), kSampleThreads,
                         order_smem(kSampleCap, kSampleBins), s>>>(reinterpret_cast<const SortBucketArgs*>(W + a_bucket));
    GBA_CUDA_TRY(ctx, cudaGetLastError());
    ++*launches;
  }
  for (size_t t = 0; t < nj; ++t) {
    const SampleJob& q = v[t];
    if (q.direct) continue;
    const size_t g = size_t(q.j.g);
    GatherCols c{};
    c.n = q.j.nagg;
    for (int a = 0; a < q.j.nagg; ++a) {
      unsigned char* tmp = W + q.agg + size_t(a) * a256(g * 8);
      GBA_CUDA_TRY(ctx, cudaMemcpyAsync(tmp, q.j.aggs[a], g * 8, cudaMemcpyDeviceToDevice, s));
      c.src[a] = reinterpret_cast<unsigned long long*>(tmp);
      c.dst[a] = q.j.aggs[a];
    }
    k_sort_gather<<<wide_grid(q.j.g), kSortThreads, 0, s>>>(c, reinterpret_cast<unsigned*>(W + q.idx_out), q.j.g,
                                                            d_fail + first + t);
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
    else if (sample_levels(jobs[j].g, &b1, &b2)) sample.push_back(j);
    else lsd.push_back(j);
  }
  // sampled jobs go together as long as 4 GiB of workspace hold them
  std::vector<size_t> parts;  // first job of every part
  size_t unused_bytes = 0;
  int unused = 0;
  for (size_t t = 0, sum = 0; t < sample.size(); ++t) {
    sort_sample(ctx, jobs, sample, t, t + 1, 0, true, &unused_bytes, nullptr, &unused, s);
    sum += unused_bytes;
    if (t == 0 || sum > (size_t(4) << 30)) {
      parts.push_back(t);
      sum = unused_bytes;
    }
  }
  for (size_t p = 0; p < parts.size(); ++p) {
    sort_sample(ctx, jobs, sample, parts[p], p + 1 < parts.size() ? parts[p + 1] : sample.size(), 0, true, &unused_bytes,
                nullptr, &unused, s);
    most = std::max(most, unused_bytes);
  }
  if (!small.empty() || !sample.empty()) {
    // front of the workspace: the small jobs' descriptors, then one failure
    // word per sampled job (their parts share the rest, one after another)
    const size_t o_fail = a256(small.size() * sizeof(SortRows)), front = o_fail + a256(4 * sample.size() + 4);
    gba_status st = gba_ws_reserve(ctx, front + most, s);
    if (st != GBA_OK) return st;
    st = gba_small_reserve(ctx, std::max<size_t>(ctx->d_small_bytes, 64 + 4 * sample.size()));
    if (st != GBA_OK) return st;
    static const cudaError_t smem_ok = [] {
      cudaError_t e = gba_allow_max_smem(k_sort_split);
      if (e == cudaSuccess) e = gba_allow_max_smem(k_sort_buckets);
      if (e == cudaSuccess) e = gba_allow_max_smem(k_sort_big_buckets);
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
      for (size_t p = 0; p < parts.size(); ++p) {
        st = sort_sample(ctx, jobs, sample, parts[p], p + 1 < parts.size() ? parts[p + 1] : sample.size(), front, false,
                         &unused_bytes, d_fail, &launches, s);
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
