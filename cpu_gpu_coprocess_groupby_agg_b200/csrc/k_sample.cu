// Row sample of a key column, for queries sized without the estimator.
//
// Plain sizing knows only the row count, which over-partitions a query of few
// groups (2^25 rows of 64 groups: 2^15 partitions) and keeps it from the table
// strategy.  k_sample_gather fetches the keys of 8192 rows spread over the
// column; k_sample_count counts them, each CTA a sixteenth of the hash range:
// how many are distinct, seen once, seen twice, and the most frequent one's
// rows.  One CTA doing both took 15-28 us (8192 address translations and
// 8192 shared-memory compare-and-swaps in series on one SM), the two take
// about 8, beside the partition count they run next to.
// No counterpart in the reference.
#include "gba_internal.cuh"
#include "sample_kernels.h"

namespace {

constexpr int kThreads = 512;
constexpr int kCtas = GBA_SAMPLE_ROWS / kThreads;  // 16
constexpr int kSlots = 2048;                       // about 512 keys per CTA
constexpr int kProbes = 64;

template <bool K64>
__global__ void __launch_bounds__(kThreads) k_sample_gather(const void* keys, int64_t n, unsigned* hashes) {
  // one row of each of 8192 equal stretches, at a place of its own inside it,
  // so that a period of the rows is not met in step
  const int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x;
  const int64_t lo = n * i / GBA_SAMPLE_ROWS, hi = n * (i + 1) / GBA_SAMPLE_ROWS;
  const int64_t r =
      lo + int64_t(__umul64hi((unsigned long long)(i + 1) * 0x9e3779b97f4a7c15ull, (unsigned long long)(hi - lo)));
  const uint64_t k =
      K64 ? __ldg(static_cast<const unsigned long long*>(keys) + r) : __ldg(static_cast<const unsigned*>(keys) + r);
  const unsigned x = fast_hash(k, 0xc4ceb9fe1a85ec53ull);
  hashes[i] = x ? x : 1u;
}

__global__ void __launch_bounds__(kThreads) k_sample_count(const unsigned* hashes, double n, double few, unsigned* words,
                                                           SampleResult* out) {
  __shared__ unsigned hash[kSlots], cnt[kSlots];  // hash 0: empty
  __shared__ unsigned s_sum[4], s_last;
  const int tid = threadIdx.x;
  for (int i = tid; i < kSlots; i += kThreads) hash[i] = cnt[i] = 0;
  if (tid < 4) s_sum[tid] = 0;
  __syncthreads();
  unsigned d = 0, f1 = 0, f2 = 0, most = 0;
#pragma unroll
  for (int u = 0; u < kCtas; ++u) {
    const unsigned h = hashes[u * kThreads + tid];
    if (h >> 28 != blockIdx.x) continue;
    unsigned s = h & (kSlots - 1);
    int p = 0;
    for (; p < kProbes; ++p) {
      const unsigned prev = atomicCAS(&hash[s], 0u, h);
      if (prev == 0u || prev == h) break;
      s = (s + 1) & (kSlots - 1);
    }
    if (p < kProbes) {
      atomicAdd(&cnt[s], 1u);
    } else {  // a crowded table: the key counts as one of its own
      ++d;
      ++f1;
    }
  }
  __syncthreads();
  for (int i = tid; i < kSlots; i += kThreads) {
    const unsigned c = cnt[i];
    d += c != 0;
    f1 += c == 1;
    f2 += c == 2;
    most = c > most ? c : most;
  }
  d = __reduce_add_sync(GBA_FULL_MASK, d);
  f1 = __reduce_add_sync(GBA_FULL_MASK, f1);
  f2 = __reduce_add_sync(GBA_FULL_MASK, f2);
  most = __reduce_max_sync(GBA_FULL_MASK, most);
  if (lane_id() == 0) {
    atomicAdd(&s_sum[0], d);
    atomicAdd(&s_sum[1], f1);
    atomicAdd(&s_sum[2], f2);
    atomicMax(&s_sum[3], most);
  }
  __syncthreads();
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) atomicAdd(&words[i], s_sum[i]);
    atomicMax(&words[3], s_sum[3]);
    __threadfence();
    s_last = atomicAdd(&words[4], 1u) == kCtas - 1;
    if (s_last) {
      __threadfence();
      SampleResult r;
      r.distinct = __ldcg(&words[0]);
      r.once = __ldcg(&words[1]);
      r.twice = __ldcg(&words[2]);
      r.most = __ldcg(&words[3]);
      r.groups = gba_groups_of_sample(r.distinct, r.once, r.twice, r.most, n);
      r.few = r.groups <= few;
      *out = r;
      if (r.few) atomicExch(&words[5], 1u);
    }
  }
}

}  // namespace

cudaError_t gba_launch_sample(const void* keys, bool key64, int64_t n, double few, unsigned* hashes, unsigned* words,
                              SampleResult* out, cudaStream_t s) {
  if (n < GBA_SAMPLE_ROWS) return cudaErrorInvalidValue;
  if (key64) k_sample_gather<true><<<kCtas, kThreads, 0, s>>>(keys, n, hashes);
  else k_sample_gather<false><<<kCtas, kThreads, 0, s>>>(keys, n, hashes);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_sample_count<<<kCtas, kThreads, 0, s>>>(hashes, double(n), few, words, out);
  return cudaGetLastError();
}
