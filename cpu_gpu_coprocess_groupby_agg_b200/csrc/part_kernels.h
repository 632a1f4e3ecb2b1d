// Host-visible interface of the radix-partition strategy kernels (k_part.cu).
#pragma once
#include "gba_kernels.h"

// A run of rows of one hot partition (too many rows for one CTA): its groups
// are merged in the HBM fallback table.
struct PartPiece {
  long long row_begin, row_end;
};

// What the plan kernel tells the kernels after it (device memory).
struct PartPlan {
  unsigned long long fb_cap;  // slots of the fallback table
  int npieces;
  int pad;
};

// k_part_plan: from the 2^(bits1 + bits2) partition counts to bounds.
struct PartPlanArgs {
  int bits1, bits2;  // digit bits of the two passes (bits2 = 0: one pass)
  const unsigned long long* hist;
  int hist_shift;                // counts per partition: 2^hist_shift consecutive ones
  unsigned long long* offs;      // first row of every partition, then n
  unsigned long long* cursors1;  // write cursors of the first pass
  unsigned long long* cursors2;  // of the second pass
  unsigned* tile_prefix;         // second pass: first tile of every first-pass segment, then all tiles
  int tile2;                     // rows per tile of the second pass
  int64_t hot_rows, piece_rows;  // partitions of more than hot_rows rows are cut into pieces
  PartPiece* pieces;
  int max_pieces;
  unsigned long long fb_cap, fb_per_hot;  // fallback slots, plus those per hot partition
  PartPlan* plan;
};

// One partition pass over `bits` hash bits below the `shift_hi` bits already
// used.  nseg = 0: the rows [0, n) are one segment; else the segments are the
// first pass's partitions, segment s starting at offs[s << bits].
struct PartPass {
  QDesc in;   // rows read (keys + value columns)
  QDesc out;  // rows written (keys + value columns, same types)
  int64_t n;
  int shift_hi, bits;
  int nseg;
  int T;                        // rows per tile (<= gba_part_scatter_max_tile())
  int threads;                  // 512 (two CTAs per SM) or 1024 (one)
  const unsigned long long* offs;
  const unsigned* tile_prefix;  // nseg + 1 entries
  unsigned long long* cursors;  // [segment][digit]
  unsigned* flags;
  // digits by key range (key-ordered output) instead of by hash: 2^bits - 1
  // splitters per segment ([segment][2^bits] words) of keys ^ flip; the pass is
  // skipped when *fail is set
  const unsigned long long* splitters;
  unsigned long long flip;
  const unsigned* fail;
};

// Final aggregation: one shared-memory table per partition (or piece).
struct PartAgg {
  QDesc rows;                      // partitioned rows + aggregate spec
  const unsigned long long* offs;  // nparts + 1 entries
  int nparts;
  const PartPiece* pieces;
  const PartPlan* plan;
  int64_t hot_rows;
  unsigned* ctr;                   // dynamic work queue (zeroed before launch)
  int S;                           // shared table slots (whole 16-byte buckets)
  int nbk;                         // buckets probed before a row goes to the fallback table
  GTable fallback;                 // keys whose probe window is full + pieces (its cap: plan->fb_cap)
  unsigned* flags;
  OutDesc out;
};

size_t gba_part_scatter_smem(const QDesc& q, int bits, int nseg, int T, bool range = false);
// rows per tile of a pass, and its CTA shape (threads)
int gba_part_tile_rows(const QDesc& q, int bits, int nseg, bool range, int max_smem_optin, int* threads);
int gba_part_scatter_max_tile();
// shared table slots of k_part_agg with 2 or 3 CTAs per SM
int gba_part_agg_slots(const QDesc& q, int ctas, int max_smem_optin);
size_t gba_part_agg_smem(const QDesc& q, int S);
// skip: a device word; once it is set the kernel stops early (null: never)
cudaError_t gba_launch_part_hist(const QDesc& q, int bits, unsigned long long* hist, int sms, const unsigned* skip,
                                 cudaStream_t s);
cudaError_t gba_launch_part_plan(const PartPlanArgs& a, cudaStream_t s);
cudaError_t gba_launch_part_scatter(const PartPass& p, int grid, cudaStream_t s);
// n passes by key range (splitters set), of one key width, column count and
// CTA shape, in one launch of `grid` CTAs each; host and device: the same array
cudaError_t gba_launch_part_scatter_many(const PartPass* host, const PartPass* device, int n, int grid, cudaStream_t s);
cudaError_t gba_launch_part_agg(const PartAgg& a, int ctas, int grid, cudaStream_t s);
