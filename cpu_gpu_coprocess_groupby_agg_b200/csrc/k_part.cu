// Radix hash partitioning + intra-partition aggregation (sm_100a).
//
// Replaces the reference's partitioner and phase 2:
//   * cal_kv_intra_group_ind / kv_inter_group_insert (kernel.cu:189-291) -
//     per-block shared histogram of murmur(k) % P, global atomicAdd block
//     offsets, CUB exclusive scan, unstaged 8-byte scatter;
//   * groupby_agg_and_statistic_kernel / device_reduce_kernel /
//     collect_kv_in_ht (kernel.cu:294-406) - per merged partition, a global
//     linear-probe table, a block counter tree-reduce and a CUB scan +
//     compaction, driven from host threads with a sync per chunk
//     (groupby_agg_intra_partition.cu:159-279).
// Here, without a host round trip between the kernels:
//   k_part_hist     one read of the keys counts every final partition
//   k_part_plan     one CTA: partition bounds, write cursors of both passes,
//                   tiles of the second pass, pieces of hot partitions
//   k_part_scatter  per tile: rows staged by asynchronous copies, ranked by
//                   digit in shared memory, room in each digit's output
//                   reserved with one atomic per digit and tile, runs of equal
//                   digits written contiguously
//   k_part_agg      one CTA per final partition at a time (dynamic queue):
//                   shared-memory table with 32-bit atomics where exact,
//                   rows whose key cannot enter the table go to an HBM
//                   fallback table; groups are written straight to the output
#include "batch_kernels.h"
#include "gba_internal.cuh"
#include "part_kernels.h"
#include "smem_table.cuh"

namespace {
#include "stream_rows.cuh"

// partition digit: `bits` bits of the hash below its top `shift_hi` bits
__device__ __forceinline__ unsigned digit_of(uint64_t key, int shift_hi, int bits) {
  return (part_hash(key) << shift_hi) >> (32 - bits);
}

// ---- counts of the final partitions ---------------------------------------------
// The counters of 2^kHistBits partitions fill 128 KB of shared memory; a finer
// fan-out takes one sweep of the keys per 2^kHistBits partitions (blockIdx.y).
constexpr int kHistBits = 15;
constexpr int kHistThreads = 1024;
constexpr int kHistIlp = 8;

template <bool K64>
__global__ void __launch_bounds__(kHistThreads) k_part_hist(const void* keys, int64_t n, int bits,
                                                            unsigned long long* hist, const unsigned* skip) {
  extern __shared__ unsigned cnt[];
  const int sub = bits < kHistBits ? bits : kHistBits;
  const int nb = 1 << sub;
  const unsigned y = blockIdx.y;
  for (int i = threadIdx.x; i < nb; i += kHistThreads) cnt[i] = 0;
  __syncthreads();
  const int64_t step = int64_t(gridDim.x) * (kHistThreads * kHistIlp);
  for (int64_t r0 = int64_t(blockIdx.x) * (kHistThreads * kHistIlp); r0 < n; r0 += step) {
    // set by the row sample that runs beside this kernel: the counts are not needed
    if (skip && *reinterpret_cast<const volatile unsigned*>(skip)) break;
    uint64_t k[kHistIlp];
#pragma unroll
    for (int u = 0; u < kHistIlp; ++u) {
      const int64_t r = r0 + u * kHistThreads + threadIdx.x;
      k[u] = 0;
      if (r < n)
        k[u] = K64 ? __ldcs(static_cast<const unsigned long long*>(keys) + r)
                   : __ldcs(static_cast<const unsigned*>(keys) + r);
    }
#pragma unroll
    for (int u = 0; u < kHistIlp; ++u) {
      const int64_t r = r0 + u * kHistThreads + threadIdx.x;
      const unsigned d = digit_of(k[u], 0, bits);
      if (r < n && (d >> sub) == y) atomicAdd(&cnt[d & (nb - 1)], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb; i += kHistThreads)
    if (cnt[i]) atomicAdd(&hist[(size_t(y) << sub) + i], (unsigned long long)cnt[i]);
}

// exclusive prefix over the block (v per thread); every thread gets the total
__device__ __forceinline__ unsigned long long block_excl_scan(unsigned long long v, unsigned long long* total) {
  __shared__ unsigned long long warp_sums[32];
  const unsigned lane = lane_id(), w = threadIdx.x >> 5;
  unsigned long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    unsigned long long y = __shfl_up_sync(GBA_FULL_MASK, x, o);
    if (lane >= unsigned(o)) x += y;
  }
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    unsigned long long s = lane < unsigned(nw) ? warp_sums[lane] : 0ull;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      unsigned long long y = __shfl_up_sync(GBA_FULL_MASK, s, o);
      if (lane >= unsigned(o)) s += y;
    }
    if (lane < unsigned(nw)) warp_sums[lane] = s;
  }
  __syncthreads();
  const unsigned long long before = (w ? warp_sums[w - 1] : 0ull) + x - v;
  *total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return before;
}

constexpr int kPlanPer = 4;  // partitions per thread and round of the plan

// ---- plan: one CTA turns the counts into every later kernel's bounds --------------
__global__ void __launch_bounds__(1024) k_part_plan(PartPlanArgs a) {
  __shared__ int s_pieces, s_hot;
  if (threadIdx.x == 0) s_pieces = s_hot = 0;
  __syncthreads();
  const int bits = a.bits1 + a.bits2;
  const int np = 1 << bits;
  const int mask2 = (1 << a.bits2) - 1;
  unsigned long long total = 0;
  for (int base = 0; base < np; base += 1024 * kPlanPer) {
    const int p0 = base + int(threadIdx.x) * kPlanPer;
    unsigned long long c[kPlanPer], sum = 0;
#pragma unroll
    for (int i = 0; i < kPlanPer; ++i) {
      c[i] = 0;
      if (p0 + i < np)
        for (int x = 0; x < 1 << a.hist_shift; ++x) c[i] += a.hist[(size_t(p0 + i) << a.hist_shift) + x];
      sum += c[i];
    }
    unsigned long long chunk;
    unsigned long long run = total + block_excl_scan(sum, &chunk);
    total += chunk;
#pragma unroll
    for (int i = 0; i < kPlanPer; ++i) {
      const int p = p0 + i;
      if (p >= np) break;
      a.offs[p] = run;
      if (a.bits2 > 0) a.cursors2[p] = run;
      if ((p & mask2) == 0) a.cursors1[p >> a.bits2] = run;
      if (c[i] > (unsigned long long)a.hot_rows) {
        const int k = int((c[i] + a.piece_rows - 1) / a.piece_rows);
        const int at = atomicAdd(&s_pieces, k);
        atomicAdd(&s_hot, 1);
        const unsigned long long end = run + c[i];
        for (int j = 0; j < k && at + j < a.max_pieces; ++j) {
          const unsigned long long b = run + (unsigned long long)j * a.piece_rows;
          a.pieces[at + j] = PartPiece{(long long)b, (long long)(b + a.piece_rows < end ? b + a.piece_rows : end)};
        }
      }
      run += c[i];
    }
  }
  if (threadIdx.x == 0) a.offs[np] = total;
  __syncthreads();
  if (a.bits2 > 0) {
    const int nseg = 1 << a.bits1;  // at most 1024
    unsigned long long tiles = 0;
    if (int(threadIdx.x) < nseg) {
      const unsigned long long rows =
          a.offs[size_t(threadIdx.x + 1) << a.bits2] - a.offs[size_t(threadIdx.x) << a.bits2];
      tiles = (rows + a.tile2 - 1) / a.tile2;
    }
    const unsigned long long before = block_excl_scan(tiles, &total);
    if (int(threadIdx.x) < nseg) a.tile_prefix[threadIdx.x] = unsigned(before);
    if (threadIdx.x == 0) a.tile_prefix[nseg] = unsigned(total);
  }
  if (threadIdx.x == 0) {
    a.plan->npieces = s_pieces < a.max_pieces ? s_pieces : a.max_pieces;
    a.plan->fb_cap = a.fb_cap + (unsigned long long)s_hot * a.fb_per_hot;
  }
}

// ---- staged scatter ---------------------------------------------------------------
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

constexpr int kScatterRows = 4096;  // rows per tile at most

// A column of a tile: `bytes` at src (aligned to the element width w) go to
// dst + (src & 15), so source and destination share their 16-byte phase and
// everything but the partial first and last 16 bytes moves as one bulk copy
// whatever row the tile starts at.  dst is 16-byte aligned and holds bytes + 16.
struct StageSpan {
  unsigned mis, end;    // the bytes are [mis, end) after dst
  unsigned head, tail;  // [head, tail) are whole granules
};
__device__ __forceinline__ StageSpan stage_span(const unsigned char* src, unsigned bytes) {
  StageSpan x;
  x.mis = unsigned(reinterpret_cast<uintptr_t>(src)) & 15u;
  x.end = x.mis + bytes;
  const unsigned lo = (x.mis + 15u) & ~15u, hi = x.end & ~15u;
  x.head = lo < x.end ? lo : x.end;
  x.tail = hi > x.head ? hi : x.head;
  return x;
}
// the partial granules: at most 3 elements each, one per thread of j = 0..7
__device__ __forceinline__ void stage_ends(unsigned char* dst, const unsigned char* src, const StageSpan& x, unsigned w,
                                           int j) {
  const unsigned o = j < 4 ? x.mis + unsigned(j) * w : x.tail + unsigned(j - 4) * w;
  if (o < (j < 4 ? x.head : x.end)) {
    if (w == 8) cp_async8(dst + o, src + (o - x.mis));
    else cp_async4(dst + o, src + (o - x.mis));
  }
}

// A CTA takes tiles round-robin.  While tile i is ranked and written, tile
// i + 1's bulk copies are in flight into the other buffer.  The rows are not
// moved in shared memory: only their order is (4 bytes per row: its digit and
// place in the tile), and the writing threads fetch their row through it.
// NC: value columns (compile time).  IdxT: row numbers of the output (32 bits
// unless there are 2^32 rows).  THREADS: 512 (two CTAs per SM, one's copies
// and barriers behind the other's work) or 1024 (one CTA with tiles of twice
// the rows, for passes whose runs would be short).
// RANGE: the digit is the key's place among the segment's splitters (the
// key-ordered output, k_sort.cu) instead of bits of its hash.
template <bool K64, int NC, typename IdxT, int THREADS, bool RANGE>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_part_scatter(PartPass one, const PartPass* many) {
  // RANGE: pass blockIdx.y of an array
  __shared__ __align__(8) unsigned char s_pass[RANGE ? sizeof(PartPass) : 8];
  if (RANGE) {
    for (int w = threadIdx.x; w < int(sizeof(PartPass) / 4); w += THREADS)
      reinterpret_cast<unsigned*>(s_pass)[w] = reinterpret_cast<const unsigned*>(many + blockIdx.y)[w];
    __syncthreads();
  }
  const PartPass& p = RANGE ? *reinterpret_cast<const PartPass*>(s_pass) : one;
  if (RANGE && *p.fail) return;  // the whole pass: set by an earlier kernel
  constexpr int kScatterThreads = THREADS;
  constexpr int kScatterRpt = kScatterRows / THREADS;
  extern __shared__ __align__(16) unsigned char sm[];
  typedef typename std::conditional<K64, unsigned long long, unsigned>::type KeyT;
  constexpr unsigned kb = K64 ? 8 : 4;
  constexpr int kCols = NC > 0 ? NC : 1;
  const int nb = 1 << p.bits, T = p.T, tid = threadIdx.x;
  const unsigned lane = lane_id(), warp = tid >> 5;
  IdxT* gbase = reinterpret_cast<IdxT*>(sm);
  unsigned* lofs = reinterpret_cast<unsigned*>(sm + size_t(nb) * 8);
  unsigned* hist = lofs + nb;
  unsigned* segs = hist + nb;  // second pass: tile prefix of the segments
  unsigned* order = segs + (p.nseg > 0 ? p.nseg + 2 : 0);
  unsigned long long* split = nullptr;  // RANGE: the current segment's splitters
  if (RANGE) {
    split = reinterpret_cast<unsigned long long*>((reinterpret_cast<uintptr_t>(order) + 7) & ~uintptr_t(7));
    order = reinterpret_cast<unsigned*>(split + nb);
  }
  int split_seg = -1;
  unsigned char* buf0 = reinterpret_cast<unsigned char*>(order + T);
  buf0 = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(buf0) + 15) & ~uintptr_t(15));
  __shared__ unsigned wsum[kScatterThreads / 32];
  __shared__ uint64_t bars[2];
  __shared__ int s_abort;
  unsigned cw[kCols], coff[kCols];  // column widths and offsets inside a buffer
  unsigned buf_bytes = ((unsigned(T) * kb + 15) & ~15u) + 16;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    cw[c] = gba_type_bytes(p.in.col_type[c]);
    coff[c] = buf_bytes;
    buf_bytes += ((unsigned(T) * cw[c] + 15) & ~15u) + 16;
  }
  for (int d = tid; d < nb; d += kScatterThreads) hist[d] = 0;
  if (p.nseg > 0)
    for (int i = tid; i <= p.nseg; i += kScatterThreads) segs[i] = p.tile_prefix[i];
  if (tid == 0) {
    s_abort = 0;
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_fence_init();
  }
  __syncthreads();
  const int64_t ntiles = p.nseg > 0 ? int64_t(segs[p.nseg]) : (p.n + T - 1) / T;

  // rows [r0, r0 + rows) of a tile and its segment
  auto locate = [&](int64_t tile, int64_t& r0, int& rows, int& seg) {
    if (p.nseg == 0) {
      seg = 0;
      r0 = tile * T;
      rows = int(p.n - r0 < T ? p.n - r0 : T);
    } else {
      int lo = 0, hi = p.nseg - 1;
      while (lo < hi) {  // last segment whose first tile is at or before `tile`
        const int mid = (lo + hi + 1) >> 1;
        if (int64_t(segs[mid]) <= tile) lo = mid;
        else hi = mid - 1;
      }
      seg = lo;
      const int64_t b = int64_t(p.offs[size_t(lo) << p.bits]), e = int64_t(p.offs[size_t(lo + 1) << p.bits]);
      r0 = b + (tile - segs[lo]) * T;
      rows = int(e - r0 < T ? e - r0 : T);
    }
  };
  // thread 0 issues the bulk copies, 8 threads of warp 1 + c the ends of
  // column c (the key is column 0)
  auto stage = [&](int64_t r0, int rows, int b) {
    if (warp > NC + 1) return;
    unsigned char* dst[1 + NC];
    const unsigned char* src[1 + NC];
    StageSpan x[1 + NC];
    dst[0] = buf0 + size_t(b) * buf_bytes;
    src[0] = static_cast<const unsigned char*>(p.in.keys) + r0 * kb;
    x[0] = stage_span(src[0], unsigned(rows) * kb);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      dst[1 + c] = dst[0] + coff[c];
      src[1 + c] = static_cast<const unsigned char*>(p.in.cols[c]) + r0 * cw[c];
      x[1 + c] = stage_span(src[1 + c], unsigned(rows) * cw[c]);
    }
    if (tid == 0) {
      unsigned tx = 0;
#pragma unroll
      for (int c = 0; c <= NC; ++c) tx += x[c].tail - x[c].head;
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&bars[b], tx);
#pragma unroll
      for (int c = 0; c <= NC; ++c)
        if (x[c].tail > x[c].head)
          bulk_g2s(dst[c] + x[c].head, src[c] + (x[c].head - x[c].mis), x[c].tail - x[c].head, &bars[b]);
    } else if (warp > 0 && lane < 8) {
#pragma unroll
      for (int c = 0; c <= NC; ++c)
        if (int(warp) == 1 + c) stage_ends(dst[c], src[c], x[c], c == 0 ? kb : cw[c > 0 ? c - 1 : 0], int(lane));
      cp_async_commit();
    }
  };

  int64_t tile = blockIdx.x, r0 = 0;
  int rows = 0, seg = 0, b = 0;
  unsigned phase = 0;  // bit x: parity to wait for on buffer x
  if (tile < ntiles) {
    locate(tile, r0, rows, seg);
    stage(r0, rows, 0);
  }
  for (; tile < ntiles; tile += gridDim.x, b ^= 1) {
    cp_async_wait_all();
    if (!mbar_wait_bounded(&bars[b], (phase >> b) & 1u, p.flags)) s_abort = 1;
    phase ^= 1u << b;
    __syncthreads();  // the tile has landed; the other buffer has been written out
    if (s_abort) {
      // the copies of this tile are the only ones in flight: wait for them
      // (bounded) before the shared memory is released
      for (unsigned k = 0; tid == 0 && k < (1u << 22); ++k)
        if (mbar_try_wait(&bars[b], ((phase >> b) & 1u) ^ 1u)) break;
      break;
    }
    const unsigned char* src = buf0 + size_t(b) * buf_bytes;
    const KeyT* skey = reinterpret_cast<const KeyT*>(
        src + ((reinterpret_cast<uintptr_t>(p.in.keys) + size_t(r0) * kb) & 15));
    const unsigned char* scol[kCols];
#pragma unroll
    for (int c = 0; c < NC; ++c)
      scol[c] = src + coff[c] + ((reinterpret_cast<uintptr_t>(p.in.cols[c]) + size_t(r0) * cw[c]) & 15);
    const int nrows = rows;
    if (RANGE && split_seg != seg) {  // (uniform over the CTA)
      split_seg = seg;
      for (int i = tid; i < nb; i += kScatterThreads) split[i] = p.splitters[(size_t(seg) << p.bits) + i];
      __syncthreads();
    }
    unsigned long long* cursors = p.cursors + (size_t(seg) << (p.nseg > 0 ? p.bits : 0));
    if (tile + gridDim.x < ntiles) {
      locate(tile + gridDim.x, r0, rows, seg);
      stage(r0, rows, b ^ 1);
    }
    // every row's digit and its rank among the tile's rows of that digit
    unsigned dr[kScatterRpt];
    if constexpr (RANGE) {
      unsigned long long k[kScatterRpt];
#pragma unroll
      for (int i = 0; i < kScatterRpt; ++i) {
        const int j = i * kScatterThreads + tid;
        k[i] = j < nrows ? skey[j] ^ KeyT(p.flip) : 0ull;
      }
      gba_range_digits<kScatterRpt>(split, p.bits, k, dr);
    }
#pragma unroll
    for (int i = 0; i < kScatterRpt; ++i) {
      const int j = i * kScatterThreads + tid;
      if (j < nrows) {
        const unsigned d = RANGE ? dr[i] : digit_of(skey[j], p.shift_hi, p.bits);
        dr[i] = d << 16 | atomicAdd(&hist[d], 1u);
      }
    }
    __syncthreads();
    // offsets of the digits inside the tile, and room in their output
    const int per = nb > kScatterThreads ? nb / kScatterThreads : 1;  // 1 or 2
    unsigned cnt[2] = {0, 0};
    IdxT res[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int d = tid * per + i;
      if (i < per && d < nb) {
        cnt[i] = hist[d];
        hist[d] = 0;
        if (cnt[i]) res[i] = IdxT(atomicAdd(&cursors[d], (unsigned long long)cnt[i]));
      }
    }
    unsigned x = cnt[0] + cnt[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(GBA_FULL_MASK, x, o);
      if (lane >= unsigned(o)) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (tid * per < nb) {
      unsigned before = 0;
#pragma unroll
      for (int w = 0; w < kScatterThreads / 32; ++w) before += w < int(warp) ? wsum[w] : 0u;
      unsigned run = before + x - cnt[0] - cnt[1];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int d = tid * per + i;
        if (i < per && d < nb) {
          lofs[d] = run;
          gbase[d] = res[i] - run;
          run += cnt[i];
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kScatterRpt; ++i) {
      const int j = i * kScatterThreads + tid;
      if (j < nrows) order[lofs[dr[i] >> 16] + (dr[i] & 0xffffu)] = (dr[i] & 0xffff0000u) | unsigned(j);
    }
    __syncthreads();
    // consecutive threads write consecutive rows of the tile's digit order:
    // each digit's run lands in one contiguous range
#pragma unroll 4
    for (int j = tid; j < nrows; j += kScatterThreads) {
      const unsigned o = order[j];
      const unsigned row = o & 0xffffu;
      const IdxT dst = gbase[o >> 16] + IdxT(j);
      if ((unsigned long long)dst >= (unsigned long long)p.n) continue;  // only if keys changed after they were counted
      // QDesc carries const pointers; the pass's output buffers are writable
      static_cast<KeyT*>(const_cast<void*>(p.out.keys))[dst] = skey[row];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        void* oc = const_cast<void*>(p.out.cols[c]);
        if (cw[c] == 8)
          static_cast<unsigned long long*>(oc)[dst] = reinterpret_cast<const unsigned long long*>(scol[c])[row];
        else
          static_cast<unsigned*>(oc)[dst] = reinterpret_cast<const unsigned*>(scol[c])[row];
      }
    }
  }
}

// ---- per-partition aggregation ------------------------------------------------------
// 512 threads; MINB = 2 or 3 CTAs per SM (gba_run_partition chooses).  Three
// keep more warps in flight for the shared-memory round trips, two hold tables
// of 1.5 times the groups.  Measured (us, 2 against 3): 2^27 rows of SUM +
// COUNT over 2^24 ids 1006 / 891, 10M distinct keys 161 / 142, the 2^26-row
// skewed query (5 aggregates) 1087 / 1034.
constexpr int kAggThreads = 512;
constexpr int kAggWarps = kAggThreads / 32;

// rows per lane in flight
template <typename Sig, int MINB>
__host__ __device__ constexpr int part_agg_rows() {
  return (Sig::NA <= 2 ? 4 : Sig::NA <= 4 ? 2 : 1) / (MINB == 3 && Sig::NA <= 4 ? 2 : 1);
}
// rows a warp may have set aside: up to 31 left over plus a whole chunk
template <typename Sig, int MINB>
__host__ __device__ constexpr int part_agg_queue() {
  return 32 * part_agg_rows<Sig, MINB>() + 32;
}

// shared-memory adds under a predicate, without a branch
__device__ __forceinline__ unsigned atom_shared_add_if(bool p, uint32_t addr, unsigned v) {
  unsigned old = 0;
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %3, 0;\n @q atom.shared.add.u32 %0, [%1], %2;\n}\n"
               : "+r"(old)
               : "r"(addr), "r"(v), "r"(unsigned(p))
               : "memory");
  return old;
}
__device__ __forceinline__ void red_shared_add_if(bool p, uint32_t addr, unsigned v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q red.shared.add.u32 [%0], %1;\n}\n" ::"r"(addr), "r"(v),
               "r"(unsigned(p))
               : "memory");
}

// Accumulator updates of R rows (row i only where ok[i]): the adds are
// predicated, not branched around, so the warp stays together.
template <bool K64, typename Sig, int R>
__device__ __forceinline__ void part_apply(const SmemTable<K64>& t, const QDesc& q, const int (&slot)[R],
                                           const unsigned long long (&v)[R][Sig::NA], const bool (&ok)[R]) {
#pragma unroll
  for (int a = 0; a < Sig::NA; ++a) {
    const int op = Sig::op(q, a);
    const int w = Sig::woff(q, a);
    const uint32_t lo = smem_u32(t.acc) + uint32_t(w) * uint32_t(t.SS) * 4u;
    if (op == ACC_CNT) {
#pragma unroll
      for (int i = 0; i < R; ++i) red_shared_add_if(ok[i], lo + uint32_t(slot[i]) * 4u, 1u);
    } else if (op == ACC_ADD_I) {
      unsigned old[R];
#pragma unroll
      for (int i = 0; i < R; ++i) old[i] = atom_shared_add_if(ok[i], lo + uint32_t(slot[i]) * 4u, unsigned(v[i][a]));
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const unsigned x = unsigned(v[i][a]);
        const unsigned hi = unsigned(v[i][a] >> 32) + ((old[i] + x) < old[i] ? 1u : 0u);
        red_shared_add_if(ok[i] && hi != 0u, lo + uint32_t(t.SS + slot[i]) * 4u, hi);
      }
    } else {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (!ok[i]) continue;
        if (op == ACC_ADD_F)
          smem_fsum(smem_ref<K64>(t, w, slot[i]), smem_ref<K64>(t, w + 2, slot[i]), smem_ref<K64>(t, w + 4, slot[i]),
                    __longlong_as_double(v[i][a]));
        else smem_acc(op, smem_ref<K64>(t, w, slot[i]), v[i][a]);
      }
      __syncwarp();
    }
  }
}

__device__ __forceinline__ unsigned cas_shared_if(bool p, uint32_t addr, unsigned cmp, unsigned val) {
  unsigned old = 0;
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %4, 0;\n @q atom.shared.cas.b32 %0, [%1], %2, %3;\n}\n"
               : "+r"(old)
               : "r"(addr), "r"(cmp), "r"(val), "r"(unsigned(p))
               : "memory");
  return old;
}
__device__ __forceinline__ unsigned long long cas_shared_if(bool p, uint32_t addr, unsigned long long cmp,
                                                            unsigned long long val) {
  unsigned long long old = 0;
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %4, 0;\n @q atom.shared.cas.b64 %0, [%1], %2, %3;\n}\n"
               : "+l"(old)
               : "r"(addr), "l"(cmp), "l"(val), "r"(unsigned(p))
               : "memory");
  return old;
}

// row r of the rows that start at keys / cols
template <bool K64, typename Sig>
__device__ __forceinline__ uint64_t part_load(const QDesc& q, const void* keys, const void* const (&cols)[GBA_MAX_COLS],
                                              unsigned r, unsigned long long (&raw)[GBA_MAX_COLS]) {
#pragma unroll
  for (int c = 0; c < GBA_MAX_COLS; ++c) {
    raw[c] = 0ull;
    if (c < Sig::ncols(q))
      raw[c] = gba_type_bytes(Sig::coltype(q, c)) == 8 ? __ldg(static_cast<const unsigned long long*>(cols[c]) + r)
                                                       : __ldg(static_cast<const unsigned*>(cols[c]) + r);
  }
  return K64 ? __ldg(static_cast<const unsigned long long*>(keys) + r) : __ldg(static_cast<const unsigned*>(keys) + r);
}

// A table of the CTA: hash slots plus the list of the claimed ones (a
// partition's groups in claiming order), so that emitting the groups and
// clearing the table touch only those.
template <bool K64>
struct PartTable {
  SmemTable<K64> st;
  unsigned short* list;
  unsigned* ngroups;
};

// One set-aside row per lane (lanes that are not live idle): rows whose key is
// not in its home bucket and found no room there, and the all-ones key.  A bucket counts as walked only when
// it was read full without the key, so a key either has a slot or never gets
// one; a key without a slot within nbk buckets goes to the fallback table.
template <bool K64, typename Sig>
__device__ __forceinline__ void part_slow_rows(const PartTable<K64>& t, const QDesc& q, const GTable& fb, int nbk,
                                               const void* keys, const void* const (&cols)[GBA_MAX_COLS], unsigned r,
                                               bool live, unsigned* flags) {
  typedef typename SmemTable<K64>::KeyW KeyW;
  constexpr int SPB = BucketT<K64>::SPB;
  const KeyW empty = smem_empty_key<K64>();
  const unsigned lane = lane_id();
  const int nb = t.st.S / SPB;
  unsigned long long raw[GBA_MAX_COLS] = {0ull, 0ull, 0ull, 0ull};
  uint64_t key = empty;
  if (live) key = part_load<K64, Sig>(q, keys, cols, r, raw);
  unsigned long long v[1][Sig::NA];
  row_contrib<Sig>(q, raw, v[0]);
  const uint32_t h = table_hash(key);
  int b = bucket_home<K64>(t.st, h), walked = 0;
  int slot[1] = {0};
  bool ok[1] = {false};
  bool claimed = false;
  bool pend = live && KeyW(key) != empty;
  if (live && !pend) smem_apply_side<K64, Sig>(t.st, q, v[0]);
  bool miss = false;
#pragma unroll 1
  while (__any_sync(GBA_FULL_MASK, pend)) {
    KeyW kb[SPB];
    ld_bucket<K64>(t.st.keys, b, kb);
    int at = -1, room = -1;
#pragma unroll
    for (int e = SPB - 1; e >= 0; --e) {
      if (kb[e] == KeyW(key)) at = e;
      if (kb[e] == empty) room = e;
    }
    if (pend && at < 0 && room >= 0) {
      // a lost claim leaves the row pending at the same bucket, unless the
      // winner holds the same key
      const KeyW prev = atomicCAS(&t.st.keys[b * SPB + room], empty, KeyW(key));
      claimed = prev == empty;
      if (claimed || prev == KeyW(key)) at = room;
    }
    __syncwarp();
    if (pend) {
      if (at >= 0) {
        slot[0] = b * SPB + at;
        ok[0] = true;
        pend = false;
      } else if (room < 0) {
        b = b + 1 == nb ? 0 : b + 1;
        if (++walked >= nbk || walked >= nb) {
          miss = true;
          pend = false;
        }
      }
    }
  }
  const unsigned m = __ballot_sync(GBA_FULL_MASK, claimed);
  if (m) {
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(t.ngroups, unsigned(__popc(m)));
    base = __shfl_sync(GBA_FULL_MASK, base, 0);
    if (claimed) t.list[base + __popc(m & ((1u << lane) - 1u))] = (unsigned short)slot[0];
  }
  part_apply<K64, Sig, 1>(t.st, q, slot, v, ok);
  if (miss) {
    gtable_insert<K64, Sig>(fb, q, key, h, v[0], flags);
    atomicOr(flags, GBA_FLAG_PART_OVERFLOW);
  }
  __syncwarp();
}

// The kernel is bound by instruction issue (ncu on 2^25 rows of SUM + COUNT by
// int64 keys: 65% of the issue slots, DRAM at 23%), so the common row is kept
// short and free of branches: load, hash, one 16-byte bucket, a predicated
// claim if the key is new there, predicated shared adds.  The other rows (keys
// displaced from a full home bucket, lost claims) are set aside in a queue of
// their warp and handled 32 at a time, with all lanes busy; handled where they
// occurred, they split nearly every warp.
template <bool K64, typename Sig, int MINB>
__global__ void __launch_bounds__(kAggThreads, MINB) k_part_agg(PartAgg a) {
  extern __shared__ __align__(16) unsigned char sm[];
  typedef typename SmemTable<K64>::KeyW KeyW;
  constexpr int R = part_agg_rows<Sig, MINB>();
  constexpr int SPB = BucketT<K64>::SPB;
  constexpr int kQueue = part_agg_queue<Sig, MINB>();
  const QDesc& q = a.rows;
  __shared__ unsigned s_item, s_ngroups;
  __shared__ unsigned long long s_base;
  __shared__ unsigned s_queue[kAggWarps][kQueue];
  const uint64_t emptyk = K64 ? EMPTY64 : uint64_t(EMPTY32);
  const int tid = threadIdx.x;
  const unsigned lane = lane_id(), warp = tid >> 5;
  PartTable<K64> t;
  t.st = smem_table_carve<K64>(sm, a.S, Sig::nwords(q));
  t.list = reinterpret_cast<unsigned short*>(sm + smem_table_bytes(a.S, K64, Sig::nwords(q)));
  t.ngroups = &s_ngroups;
  unsigned* queue = s_queue[warp];
  smem_table_init<K64, Sig>(t.st, q);
  GTable fb = a.fallback;
  fb.cap = a.plan->fb_cap;
  const unsigned npieces = unsigned(a.plan->npieces);
  const unsigned nitems = npieces + unsigned(a.nparts);
  if (tid == 0) {
    s_item = atomicAdd(a.ctr, 1u);
    s_ngroups = 0;
  }
  for (;;) {
    __syncthreads();  // the table is clear and s_item is set
    const unsigned item = s_item;
    if (item >= nitems) break;
    const bool piece = item < npieces;
    int64_t b, e;
    if (piece) {
      b = a.pieces[item].row_begin;
      e = a.pieces[item].row_end;
    } else {
      b = int64_t(a.offs[item - npieces]);
      e = int64_t(a.offs[item - npieces + 1]);
      if (e - b > a.hot_rows) e = b;  // its pieces are items of their own
    }
    unsigned next = 0;
    if (tid == 0) next = atomicAdd(a.ctr, 1u);
    const unsigned n = unsigned(e - b);
    const void* keys = static_cast<const KeyW*>(q.keys) + b;
    const void* cols[GBA_MAX_COLS];
#pragma unroll
    for (int c = 0; c < GBA_MAX_COLS; ++c)
      cols[c] = c < Sig::ncols(q)
                    ? static_cast<const unsigned char*>(q.cols[c]) + b * gba_type_bytes(Sig::coltype(q, c))
                    : nullptr;
    unsigned nq = 0;  // rows set aside by this warp
    for (unsigned c0 = warp * (32 * R); c0 < n; c0 += kAggThreads * R) {
      KeyW key[R];
      unsigned long long v[R][Sig::NA];
      int slot[R];
      bool ok[R];
      {
        unsigned long long raw[R][GBA_MAX_COLS];
#pragma unroll
        for (int u = 0; u < R; ++u) {
          const unsigned r = c0 + u * 32 + lane;
          key[u] = KeyW(emptyk);
#pragma unroll
          for (int c = 0; c < GBA_MAX_COLS; ++c) raw[u][c] = 0ull;
          if (r < n) key[u] = KeyW(part_load<K64, Sig>(q, keys, cols, r, raw[u]));
        }
#pragma unroll
        for (int u = 0; u < R; ++u) row_contrib<Sig>(q, raw[u], v[u]);
      }
      KeyW kb[R][SPB];
#pragma unroll
      for (int u = 0; u < R; ++u) {
        slot[u] = bucket_home<K64>(t.st, table_hash(key[u]));
        ld_bucket<K64>(t.st.keys, slot[u], kb[u]);
      }
#pragma unroll
      for (int u = 0; u < R; ++u) {
        int at = 0;
        bool hit = false;
#pragma unroll
        for (int x = 0; x < SPB; ++x) {
          const bool m = kb[u][x] == key[u];
          at = m ? x : at;
          hit = hit || m;
        }
        slot[u] = slot[u] * SPB + at;
        ok[u] = hit && key[u] != KeyW(emptyk);  // an empty slot is no match for the all-ones key
      }
      // new keys claim the first empty slot of their home bucket, all rows'
      // claims in flight together
      bool want[R], any = false;
#pragma unroll
      for (int u = 0; u < R; ++u) {
        want[u] = !ok[u] && key[u] != KeyW(emptyk) && kb[u][SPB - 1] == KeyW(emptyk);
        any = any || want[u];
      }
      if (__any_sync(GBA_FULL_MASK, any)) {
        KeyW prev[R];
#pragma unroll
        for (int u = 0; u < R; ++u) {
          int room = SPB - 1;
#pragma unroll
          for (int x = SPB - 2; x >= 0; --x) room = kb[u][x] == KeyW(emptyk) ? x : room;
          if (want[u]) slot[u] = slot[u] / SPB * SPB + room;
          prev[u] = cas_shared_if(want[u], smem_u32(t.st.keys + slot[u]), KeyW(emptyk), key[u]);
        }
        unsigned m[R], total = 0;
#pragma unroll
        for (int u = 0; u < R; ++u) {
          m[u] = __ballot_sync(GBA_FULL_MASK, want[u] && prev[u] == KeyW(emptyk));
          total += __popc(m[u]);
          ok[u] = ok[u] || (want[u] && (prev[u] == KeyW(emptyk) || prev[u] == key[u]));
        }
        unsigned base = 0;
        if (lane == 0 && total) base = atomicAdd(t.ngroups, total);
        base = __shfl_sync(GBA_FULL_MASK, base, 0);
#pragma unroll
        for (int u = 0; u < R; ++u) {
          if (m[u] >> lane & 1u) t.list[base + __popc(m[u] & ((1u << lane) - 1u))] = (unsigned short)slot[u];
          base += __popc(m[u]);
        }
        __syncwarp();
      }
      part_apply<K64, Sig, R>(t.st, q, slot, v, ok);
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const unsigned r = c0 + u * 32 + lane;
        const bool aside = !ok[u] && r < n;
        const unsigned m = __ballot_sync(GBA_FULL_MASK, aside);
        if (aside) queue[nq + __popc(m & ((1u << lane) - 1u))] = r;
        nq += __popc(m);
      }
      __syncwarp();
      const bool last = c0 + kAggThreads * R >= n;
      while (nq >= 32 || (last && nq > 0)) {
        const unsigned take = nq < 32 ? nq : 32;
        nq -= take;
        const unsigned r = lane < take ? queue[nq + lane] : 0u;
        part_slow_rows<K64, Sig>(t, q, fb, a.nbk, keys, cols, r, lane < take, a.flags);
      }
    }
    __syncthreads();
    const unsigned total = s_ngroups;
    const bool side = *t.st.side_present() != 0u;
    __syncthreads();
    if (tid == 0) {
      s_item = next;
      s_ngroups = 0;
      if (!piece && total + (side ? 1u : 0u))
        s_base = atomicAdd(a.out.count, (unsigned long long)total + (side ? 1u : 0u));
    }
    __syncthreads();
    const unsigned long long pos = s_base;
    for (unsigned g = tid; g < total; g += kAggThreads) {
      const int i = t.list[g];
      const uint64_t k = t.st.keys[i];
      unsigned long long x[Sig::NA];
#pragma unroll
      for (int c = 0; c < Sig::NA; ++c) x[c] = smem_acc_read<K64, Sig>(t.st, q, c, i);
      smem_slot_reset<K64, Sig>(t.st, q, i);
      if (piece) {
        // a piece of a hot partition: its keys recur in the other pieces, so
        // its groups are merged in the HBM table and emitted from there
        gtable_insert<K64, Sig>(fb, q, k, table_hash(k), x, a.flags);
      } else if (pos + g < (unsigned long long)a.out.capacity) {
        if (K64) static_cast<unsigned long long*>(a.out.keys)[pos + g] = k;
        else static_cast<unsigned*>(a.out.keys)[pos + g] = unsigned(k);
#pragma unroll
        for (int c = 0; c < Sig::NA; ++c) a.out.accs[c][pos + g] = x[c];
      }
    }
    if (side && tid == 0) {
      unsigned long long x[Sig::NA];
#pragma unroll
      for (int c = 0; c < Sig::NA; ++c) x[c] = smem_acc_read<K64, Sig>(t.st, q, c, -1);
      if (piece) {
        gtable_insert<K64, Sig>(fb, q, emptyk, 0u, x, a.flags);
      } else {
        const unsigned long long sp = pos + total;
        if (sp < (unsigned long long)a.out.capacity) {
          if (K64) static_cast<unsigned long long*>(a.out.keys)[sp] = EMPTY64;
          else static_cast<unsigned*>(a.out.keys)[sp] = EMPTY32;
#pragma unroll
          for (int c = 0; c < Sig::NA; ++c) a.out.accs[c][sp] = x[c];
        }
      }
      smem_side_reset<K64, Sig>(t.st, q);
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------
size_t gba_part_scatter_smem(const QDesc& q, int bits, int nseg, int T, bool range) {
  const size_t nb = size_t(1) << bits;
  size_t b = (range ? nb * 8 + 8 : 0) + nb * (8 + 4 + 4) + (nseg > 0 ? size_t(nseg + 2) * 4 : 0) + size_t(T) * 4 + 16;
  auto col = [&](size_t w) { return ((size_t(T) * w + 15) & ~size_t(15)) + 16; };
  size_t rows = col(q.key64 ? 8 : 4);
  for (int c = 0; c < q.ncols; ++c) rows += col(gba_type_bytes(q.col_type[c]));
  return b + 2 * rows;
}

// dynamic shared memory of k_part_agg with S slots: the table and the list of
// its claimed slots
size_t gba_part_agg_smem(const QDesc& q, int S) { return smem_table_bytes(S, q.key64, q.nwords) + size_t(S) * 2 + 16; }

// slots of k_part_agg's table with `ctas` CTAs per SM: what a CTA's share of
// the SM's shared memory (each CTA loses 1 KB to the system) holds beside the
// kernel's static part
int gba_part_agg_slots(const QDesc& q, int ctas, int max_smem_optin) {
  size_t fixed = 0;
  gba_dispatch_sig(q, [&](auto, auto sig) -> cudaError_t {
    using Sig = decltype(sig);
    fixed = size_t(kAggWarps) * (ctas == 3 ? part_agg_queue<Sig, 3>() : part_agg_queue<Sig, 2>()) * 4 + 64;
    return cudaSuccess;
  });
  const size_t room = (size_t(max_smem_optin) + 1024) / size_t(ctas) - 1024 - fixed - gba_part_agg_smem(q, 0) - 64;
  const size_t slot = (q.key64 ? 8 : 4) + 4 * size_t(q.nwords) + 2;
  return int(room / slot < 16384 ? room / slot : 16384) / 4 * 4;
}

int gba_part_scatter_max_tile() { return kScatterRows; }

cudaError_t gba_launch_part_hist(const QDesc& q, int bits, unsigned long long* hist, int sms, const unsigned* skip,
                                 cudaStream_t s) {
  const int sub = bits < kHistBits ? bits : kHistBits;
  const size_t smem = (size_t(1) << sub) * 4;
  auto go = [&](auto kernel) -> cudaError_t {
    cudaError_t e = gba_allow_max_smem(kernel);
    if (e != cudaSuccess) return e;
    const int64_t want = (q.n + kHistThreads * kHistIlp - 1) / (kHistThreads * kHistIlp);
    const int64_t most = int64_t(sms) * (smem <= 64 * 1024 ? 2 : 1);
    const dim3 grid(unsigned(want < 1 ? 1 : want < most ? want : most), 1u << (bits - sub));
    kernel<<<grid, kHistThreads, smem, s>>>(q.keys, q.n, bits, hist, skip);
    return cudaGetLastError();
  };
  return q.key64 ? go(k_part_hist<true>) : go(k_part_hist<false>);
}

cudaError_t gba_launch_part_plan(const PartPlanArgs& a, cudaStream_t s) {
  k_part_plan<<<1, 1024, 0, s>>>(a);
  return cudaGetLastError();
}

namespace {
// one pass (many null) or a device array of `n` RANGE passes whose host copies
// start at &p: all of one key width, column count and CTA shape
cudaError_t launch_scatter(const PartPass& p, const PartPass* many, int n, int grid, cudaStream_t s) {
  size_t smem = 0;
  for (int i = 0; i < n; ++i) {
    const PartPass& x = (&p)[i];
    // the kernel's digit scan takes at most two digits per thread
    if (x.bits < 1 || (1 << x.bits) > 1024 || x.T > kScatterRows || (x.threads != 512 && x.threads != 1024))
      return cudaErrorInvalidValue;
    const size_t b = gba_part_scatter_smem(x.in, x.bits, x.nseg, x.T, many != nullptr);
    smem = b > smem ? b : smem;
  }
  auto go = [&](auto kernel) -> cudaError_t {
    cudaError_t e = gba_allow_max_smem(kernel);
    if (e != cudaSuccess) return e;
    kernel<<<dim3(unsigned(grid), unsigned(n)), p.threads, smem, s>>>(p, many);
    return cudaGetLastError();
  };
  auto shape = [&](auto K, auto I, auto N, auto R) -> cudaError_t {
    constexpr bool k64 = decltype(K)::value, range = decltype(R)::value;
    constexpr int nc = decltype(N)::value;
    using IdxT = decltype(I);
    return p.threads == 1024 ? go(k_part_scatter<k64, nc, IdxT, 1024, range>)
                             : go(k_part_scatter<k64, nc, IdxT, 512, range>);
  };
  auto cols = [&](auto K, auto I, auto R) -> cudaError_t {
    switch (p.in.ncols) {
      case 0: return shape(K, I, std::integral_constant<int, 0>{}, R);
      case 1: return shape(K, I, std::integral_constant<int, 1>{}, R);
      case 2: return shape(K, I, std::integral_constant<int, 2>{}, R);
      case 3: return shape(K, I, std::integral_constant<int, 3>{}, R);
      case 4: return shape(K, I, std::integral_constant<int, 4>{}, R);
    }
    return cudaErrorInvalidValue;
  };
  const bool wide = p.n >= (int64_t(1) << 32);
  const std::true_type yes{};
  const std::false_type no{};
  if (many) {
    if (wide) return cudaErrorInvalidValue;
    return p.in.key64 ? cols(yes, 0u, yes) : cols(no, 0u, yes);
  }
  if (p.in.key64) return wide ? cols(yes, 0ull, no) : cols(yes, 0u, no);
  return wide ? cols(no, 0ull, no) : cols(no, 0u, no);
}
}  // namespace

cudaError_t gba_launch_part_scatter(const PartPass& p, int grid, cudaStream_t s) {
  return launch_scatter(p, nullptr, 1, grid, s);
}
cudaError_t gba_launch_part_scatter_many(const PartPass* host, const PartPass* device, int n, int grid, cudaStream_t s) {
  return launch_scatter(*host, device, n, grid, s);
}

cudaError_t gba_launch_part_agg(const PartAgg& a, int ctas, int grid, cudaStream_t s) {
  const size_t smem = gba_part_agg_smem(a.rows, a.S);
  auto go = [&](auto kernel) -> cudaError_t {
    cudaError_t e = gba_allow_max_smem(kernel);
    if (e != cudaSuccess) return e;
    kernel<<<grid, kAggThreads, smem, s>>>(a);
    return cudaGetLastError();
  };
  return gba_dispatch_sig(a.rows, [&](auto K, auto sig) -> cudaError_t {
    constexpr bool k64 = decltype(K)::value;
    using Sig = decltype(sig);
    return ctas == 3 ? go(k_part_agg<k64, Sig, 3>) : go(k_part_agg<k64, Sig, 2>);
  });
}
