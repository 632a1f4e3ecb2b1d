// Host-visible interface of the row sample (k_sample.cu).
#pragma once
#include <math.h>

#include "gba_kernels.h"

constexpr int GBA_SAMPLE_ROWS = 8192;

struct SampleResult {
  double groups;                       // estimate for all rows
  unsigned few;                        // 1: at most the `few` groups the caller asked about
  unsigned distinct, once, twice, most;  // keys of the sample: all, seen once, seen twice; rows of the most frequent
};

// Group estimate of n rows from their sample.  Every key seen again: the
// sample holds them all but for rare ones.  Else, for evenly used keys (the
// most frequent one within what chance gives), Chao's estimate from the keys
// seen once and twice (Chao, 1984), with a margin; for skewed ones, whose rare
// keys it misses, four times the guaranteed-error estimate
// sqrt(n / rows) * once + rest (Charikar et al., 2000).  A sample of almost
// only distinct keys says no more than the row count.
__host__ __device__ inline double gba_groups_of_sample(unsigned distinct, unsigned once, unsigned twice, unsigned most,
                                                       double n) {
  const double s = GBA_SAMPLE_ROWS, d = distinct, f1 = once, f2 = twice > 1 ? twice : 1.0;
  double est = n;
  if (once == 0) {
    est = d + 1.0;
  } else if (twice >= 20 || f1 <= 0.9 * s) {
    const double chao = d + f1 * f1 / (2.0 * f2);
    const double each = s / chao;  // rows per key in the sample
    if (double(most) <= each + 6.0 * sqrt(each) + 6.0) {
      est = 1.3 * chao;
    } else {
      const double gee = sqrt(n / s) * f1 + (d - f1);
      est = 4.0 * (gee > chao ? gee : chao);
    }
  }
  return est < n ? est : n;
}

constexpr size_t GBA_SAMPLE_SCRATCH = GBA_SAMPLE_ROWS * 4;
// words: 5 cleared device words (4 sums and a ticket) followed by the skip
// flag, set when there are at most `few` groups; hashes: GBA_SAMPLE_SCRATCH
// device bytes; out: pinned host memory
cudaError_t gba_launch_sample(const void* keys, bool key64, int64_t n, double few, unsigned* hashes, unsigned* words,
                              SampleResult* out, cudaStream_t s);
