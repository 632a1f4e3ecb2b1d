// Host driver of the radix-partition strategy and the strategy choice.
//
// Fan-out: the reference uses a fixed P=300 (test/test.cu:96) and then merges
// small partitions greedily so each merged partition fills a global table of
// `Capacity` slots (groupby_agg_intra_partition.cu:13-48).  Here the fan-out is
// chosen so that every final partition's groups fill at most kGroupsPerTable
// of one CTA's shared-memory table, split over one or two MSD passes so each
// scatter pass keeps its write runs long.  The host only launches: bounds,
// cursors and the pieces of hot partitions are computed on the device.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "gba_context.h"
#include "gba_plan.h"
#include "part_kernels.h"
#include "sample_kernels.h"

namespace {

constexpr size_t kAlign = 256;
int tbytes(int t) { return gba_type_bytes(t); }

struct Carver {
  size_t off = 0;
  size_t take(size_t bytes) {
    const size_t o = off;
    off = gba_round_up(off + bytes, kAlign);
    return o;
  }
};

// Groups aimed at per partition, as a share of the shared table's slots.  An
// estimate is taken with a margin of 1.25, so it may fill more; the row count
// (plain sizing) is reached when nearly every key is distinct.  The power of
// two leaves between half of this and this.
constexpr double kLearnedFill = 0.76, kPlainFill = 0.6;
// digit bits up to which one scatter pass is used
constexpr int kOnePassBits = 9;
// fewest partition bits of a large query
constexpr int kFewPartBits = 9;
// partition bits up to which one sweep of the keys counts every partition
constexpr int kOneSweepBits = 15;

size_t row_bytes(const QDesc& q) {
  size_t b = q.key64 ? 8 : 4;
  for (int c = 0; c < q.ncols; ++c) b += tbytes(q.col_type[c]);
  return b;
}

}  // namespace

// Rows per tile: two CTAs of 512 threads per SM, each with two tiles of rows in
// flight; where a digit's run in such a tile would be under 24 rows, one CTA of
// 1024 threads with larger tiles (measured, two CTAs against one: 2^28 rows of
// 24 bytes in 7 + 8 bits 5.73 against 5.03 ms; 2^27 rows of 16 bytes in 6 + 7
// bits 1.64 against 2.09 ms).
int gba_part_tile_rows(const QDesc& q, int bits, int nseg, bool range, int max_smem_optin, int* threads) {
  auto fit = [&](size_t budget) {
    int T = gba_part_scatter_max_tile();
    while (T > 512 && gba_part_scatter_smem(q, bits, nseg, T, range) > budget) T -= 256;
    return T;
  };
  const int T = fit(size_t(max_smem_optin) / 2 - 1536);
  *threads = T >> bits < 24 && T < gba_part_scatter_max_tile() ? 1024 : 512;
  return *threads == 512 ? T : fit(size_t(max_smem_optin) - 1536);
}

double gba_table_groups(const gba_context* ctx, const QDesc& q) {
  return 0.9 * gba_part_agg_slots(q, 2, ctx->max_smem_optin);  // 0.45 of the table one CTA per SM holds
}

int gba_choose_strategy(const gba_context* ctx, const QDesc& q, const gba_knobs& k, double predicted_groups,
                        const GbaPlan& p) {
  (void)k;
  (void)p;
  // The table strategy where a CTA's shared table holds every group, or where
  // the query is too small for the partition kernels' launches; the partition
  // strategy beyond.  Measured (us, table / partition, SUM + COUNT by int64
  // keys, without the estimator): 2^25 rows of 1000 groups 160 / 415, of 16000
  // groups 965 / 400; 2^26 rows of 2^18 groups 1550 / 890, of 2^20 1840 / 1250;
  // 2^20 rows of 1024 groups 80 / 93.
  const double groups = predicted_groups > 0 ? predicted_groups : double(q.n);
  if (groups <= gba_table_groups(ctx, q)) return GBA_STRATEGY_TABLE;
  const double table_bytes = groups / 0.7 * 8.0 * gba_gt_stride(q.naccs);
  return q.n <= (int64_t(1) << 20) && table_bytes <= 80.0 * (1 << 20) ? GBA_STRATEGY_TABLE : GBA_STRATEGY_PARTITION;
}

// A plain-sized query of more than 2^20 rows is sampled first (below, the
// table strategy takes it in any case).
bool gba_sample_wanted(const QDesc& q, const gba_knobs& k) {
  return k.sizing == GBA_SIZING_PLAIN && k.strategy == GBA_STRATEGY_AUTO && k.partition_bits <= 0 &&
         q.n > (int64_t(1) << 20);
}

// The sample runs on the copy stream beside the partition count by the row
// count's fan-out, whose counts (at the front of the workspace, *counted_bits)
// a partition run coarsens to its own; the count stops early where the sample
// finds few groups.  Returns once the sample is there.
gba_status gba_sample_groups(gba_context* ctx, const QDesc& q, const gba_knobs& k, double few, cudaStream_t s,
                             double* groups, bool* is_few, int* counted_bits) {
  PartShape by_rows;
  gba_part_shape(ctx, q, k, -1.0, &by_rows);
  const size_t front = gba_round_up(size_t(8) << by_rows.bits, kAlign);
  // room for the run that follows, so that the counts stay where they are: one
  // with two passes takes the most, and its smaller parts shrink with its bits
  size_t bytes = 0;
  int unused = 0;
  gba_part_enqueue(ctx, q, nullptr, by_rows, 0, nullptr, &bytes, nullptr, nullptr, &unused, s);
  const size_t hashes = front + bytes;
  gba_status st = gba_ws_reserve(ctx, hashes + GBA_SAMPLE_SCRATCH, s);
  if (st != GBA_OK) return st;
  unsigned char* W = static_cast<unsigned char*>(ctx->ws);
  unsigned* words = reinterpret_cast<unsigned*>(ctx->d_small + 32);
  SampleResult* r = reinterpret_cast<SampleResult*>(ctx->h_small + 64);  // pinned: written from the device
  GBA_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_small, 0, 64, s));
  GBA_CUDA_TRY(ctx, cudaMemsetAsync(W, 0, front, s));
  GBA_CUDA_TRY(ctx, cudaEventRecord(ctx->ev[7], s));
  GBA_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->copy_stream, ctx->ev[7], 0));
  GBA_CUDA_TRY(ctx, gba_launch_sample(q.keys, q.key64 != 0, q.n, few, reinterpret_cast<unsigned*>(W + hashes), words, r,
                                      ctx->copy_stream));
  GBA_CUDA_TRY(ctx, cudaEventRecord(ctx->ev[6], ctx->copy_stream));
  GBA_CUDA_TRY(ctx, gba_launch_part_hist(q, by_rows.bits, reinterpret_cast<unsigned long long*>(W), ctx->sms, words + 5, s));
  // (later work of the stream also follows the sample)
  GBA_CUDA_TRY(ctx, cudaStreamWaitEvent(s, ctx->ev[6], 0));
  GBA_CUDA_TRY(ctx, cudaEventSynchronize(ctx->ev[6]));
  ctx->stats.kernel_launches += 3;
  *groups = r->groups;
  *is_few = r->few != 0;
  *counted_bits = by_rows.bits;
  return GBA_OK;
}

// Fan-out and table shape of a query's partition run.
void gba_part_shape(const gba_context* ctx, const QDesc& q, const gba_knobs& k, double predicted_groups, PartShape* sh) {
  sh->groups = double(std::max<int64_t>(q.n, 1));
  const bool learned = k.sizing == GBA_SIZING_LEARNED && predicted_groups > 0;
  if (learned) sh->groups = std::min(sh->groups, predicted_groups * 1.25 + 64);
  else if (predicted_groups > 0) sh->groups = std::min(sh->groups, predicted_groups);  // sampled
  auto slots = [&](int ctas) {
    const int s = gba_part_agg_slots(q, ctas, ctx->max_smem_optin);
    return k.smem_slots > 0 ? std::max(32, std::min(s, k.smem_slots) / 4 * 4) : s;
  };
  auto fan_out = [&](int ctas) {
    const double per_table = (learned ? kLearnedFill : kPlainFill) * slots(ctas);
    const int bits = int(std::ceil(std::log2(std::max(1.0, sh->groups / per_table))));
    return std::max(1, std::min(k.partition_bits > 0 ? k.partition_bits : bits, 20));
  };
  // three aggregation CTAs per SM unless their smaller tables cost another
  // pass over the rows or another sweep of the keys
  int b3 = fan_out(3), b2 = fan_out(2);
  // A large query gets at least 2^9 partitions, and at 2^9 two CTAs per SM: 512
  // partitions fill 86% of two rounds of 296 CTAs, but 58% of 444.  Measured on
  // 16M rows of 200k groups, 4 aggregates (us, aggregation + scatter): 8 bits
  // 322 + 138, 9 bits 198 + 150, 11 bits in two passes 189 + 201.
  if (k.partition_bits <= 0 && q.n > (int64_t(1) << 20)) {
    b3 = std::max(b3, kFewPartBits);
    b2 = std::max(b2, kFewPartBits);
  }
  sh->ctas = b3 > b2 && (b3 > kOneSweepBits || (b2 <= kOnePassBits && b3 > kOnePassBits)) ? 2 : 3;
  if (b2 == kFewPartBits && k.partition_bits <= 0) sh->ctas = 2;
  sh->S = slots(sh->ctas);
  sh->bits = sh->ctas == 3 ? b3 : b2;
}

// Enqueues a partition run in the workspace at `base` (null: only sizes it;
// *bytes: the workspace it takes).  status: GBA_PART_STATUS cleared device
// bytes that receive the flags (offset 0) and the group count (offset 8).
// counted: the counts of 2^counted_bits (at least as many) partitions, when
// they were made before.
gba_status gba_part_enqueue(gba_context* ctx, const QDesc& q, const gba_output* out, const PartShape& sh,
                            int smem_probe_cap, unsigned char* base, size_t* bytes, unsigned char* status,
                            GbaTimer* tm, int* launches, cudaStream_t s, const unsigned long long* counted,
                            int counted_bits) {
  const int64_t n = q.n;
  const int S = sh.S, B = sh.bits;
  // a partition of more than 2 Lp rows (a hot key) is cut into pieces of Lp
  const int64_t Lp = std::max<int64_t>(32768, n / (int64_t(ctx->sms) * 8));
  const int64_t max_split = n / (2 * Lp) + 1, max_pieces = 2 * (n / Lp) + 2;
  // one pass up to kOnePassBits digit bits, else two, the first one with the
  // fewer digits: its runs are spread over the whole row buffer (measured on
  // 2^28 rows of 24 bytes, 15 bits: 5.73 ms as 7 + 8, 6.73 as 8 + 7)
  const int b1 = B <= kOnePassBits ? B : B / 2, b2 = B - b1;
  const int64_t nparts = int64_t(1) << B;
  int th1 = 512, th2 = 512;
  const int T1 = gba_part_tile_rows(q, b1, 0, false, ctx->max_smem_optin, &th1);
  const int T2 = b2 > 0 ? gba_part_tile_rows(q, b2, 1 << b1, false, ctx->max_smem_optin, &th2) : 0;
  const uint64_t fb_cap = std::max<uint64_t>(1 << 16, uint64_t(std::min<double>(sh.groups * 0.02, 1 << 24)));

  Carver cv;
  size_t buf[2][1 + GBA_MAX_COLS];
  for (int x = 0; x < (b2 > 0 ? 2 : 1); ++x) {
    buf[x][0] = cv.take(size_t(n) * (q.key64 ? 8 : 4));
    for (int c = 0; c < q.ncols; ++c) buf[x][1 + c] = cv.take(size_t(n) * tbytes(q.col_type[c]));
  }
  const size_t o_zero = cv.take(8 * size_t(nparts));  // counts (cleared)
  const size_t o_offs = cv.take(8 * size_t(nparts + 1));
  const size_t o_cur1 = cv.take(8 << b1);
  const size_t o_cur2 = cv.take(b2 > 0 ? 8 * size_t(nparts) : 8);
  const size_t o_tiles = cv.take((4 << b1) + 4);
  const size_t o_pieces = cv.take(sizeof(PartPiece) * size_t(max_pieces));
  const size_t o_plan = cv.take(sizeof(PartPlan));
  // the fallback table goes last: its size is decided on the device
  const size_t o_fb = cv.take((fb_cap + 1 + uint64_t(max_split) * uint64_t(S) * 2) * size_t(gba_gt_stride(q.naccs)) * 8);
  *bytes = cv.off;
  if (!base) return GBA_OK;
  unsigned char* W = base;
  unsigned* d_flags = reinterpret_cast<unsigned*>(status);
  unsigned long long* d_count = reinterpret_cast<unsigned long long*>(status + 8);
  auto words = [&](size_t o) { return reinterpret_cast<unsigned long long*>(W + o); };
  if (!counted) GBA_CUDA_TRY(ctx, cudaMemsetAsync(W + o_zero, 0, 8 * size_t(nparts), s));
  PartPlanArgs pl{};
  pl.bits1 = b1;
  pl.bits2 = b2;
  pl.hist = counted ? counted : words(o_zero);
  pl.hist_shift = counted ? counted_bits - B : 0;
  pl.offs = words(o_offs);
  pl.cursors1 = words(o_cur1);
  pl.cursors2 = words(o_cur2);
  pl.tile_prefix = reinterpret_cast<unsigned*>(W + o_tiles);
  pl.tile2 = T2;
  pl.hot_rows = 2 * Lp;
  pl.piece_rows = Lp;
  pl.pieces = reinterpret_cast<PartPiece*>(W + o_pieces);
  pl.max_pieces = int(max_pieces);
  pl.fb_cap = fb_cap;
  pl.fb_per_hot = uint64_t(S) * 2;
  pl.plan = reinterpret_cast<PartPlan*>(W + o_plan);
  if (tm) tm->begin(3);
  if (!counted) GBA_CUDA_TRY(ctx, gba_launch_part_hist(q, B, words(o_zero), ctx->sms, nullptr, s));
  GBA_CUDA_TRY(ctx, gba_launch_part_plan(pl, s));
  if (tm) tm->end();

  QDesc in = q;
  for (int x = 0; x < (b2 > 0 ? 2 : 1); ++x) {
    PartPass pp{};
    pp.in = in;
    pp.out = q;
    pp.out.keys = W + buf[x][0];
    for (int c = 0; c < q.ncols; ++c) pp.out.cols[c] = W + buf[x][1 + c];
    pp.n = n;
    pp.shift_hi = x == 0 ? 0 : b1;
    pp.bits = x == 0 ? b1 : b2;
    pp.nseg = x == 0 ? 0 : 1 << b1;
    pp.T = x == 0 ? T1 : T2;
    pp.threads = x == 0 ? th1 : th2;
    pp.offs = words(o_offs);
    pp.tile_prefix = pl.tile_prefix;
    pp.cursors = words(x == 0 ? o_cur1 : o_cur2);
    pp.flags = d_flags;
    const int64_t tiles = n / pp.T + 1 + pp.nseg;
    if (tm) tm->begin(3);
    GBA_CUDA_TRY(ctx, gba_launch_part_scatter(pp, int(std::min<int64_t>(tiles, ctx->sms * (1024 / pp.threads))), s));
    if (tm) tm->end();
    in = pp.out;
  }

  // final aggregation over the 2^B partitions, then the fallback table
  GTable fb;
  fb.base = words(o_fb);
  fb.cap = fb_cap;
  fb.probe_cap = 256;
  GBA_CUDA_TRY(ctx, gba_launch_table_init(fb, q, ctx->sms * 4, s, &pl.plan->fb_cap));
  PartAgg pa{};
  pa.rows = in;
  pa.offs = words(o_offs);
  pa.nparts = int(nparts);
  pa.pieces = pl.pieces;
  pa.plan = pl.plan;
  pa.hot_rows = 2 * Lp;
  pa.ctr = reinterpret_cast<unsigned*>(status + 20);
  pa.S = S;
  pa.nbk = std::max(smem_probe_cap, 64) / (q.key64 ? 2 : 4);
  pa.fallback = fb;
  pa.flags = d_flags;
  pa.out.keys = out->keys;
  for (int a = 0; a < GBA_MAX_AGGS; ++a) pa.out.accs[a] = static_cast<unsigned long long*>(out->aggs[a]);
  pa.out.capacity = out->capacity;
  pa.out.count = d_count;
  if (tm) tm->begin(1);
  GBA_CUDA_TRY(ctx, gba_launch_part_agg(pa, sh.ctas, int(std::min<int64_t>(nparts + max_pieces, ctx->sms * sh.ctas)), s));
  if (tm) tm->end();
  if (tm) tm->begin(2);
  GBA_CUDA_TRY(ctx, gba_launch_compact(
                        fb, q, pa.out, int(std::max<uint64_t>(1, std::min<uint64_t>(ctx->sms * 8, fb.cap / 256))), s,
                        &pl.plan->fb_cap));
  if (tm) tm->end();
  *launches += b2 > 0 ? 7 : 6;
  return GBA_OK;
}

gba_status gba_run_partition(gba_context* ctx, const QDesc& q, const gba_output* out, const gba_knobs& k,
                             const GbaPlan& p, double predicted_groups, cudaStream_t s, int64_t* n_groups,
                             int counted_bits) {
  ctx->stats.strategy = GBA_STRATEGY_PARTITION;
  PartShape sh;
  gba_part_shape(ctx, q, k, predicted_groups, &sh);
  if (counted_bits > 0 && sh.bits > counted_bits) gba_part_shape(ctx, q, k, -1.0, &sh);
  for (int attempt = 0;; ++attempt) {
    ctx->stats.partition_bits = sh.bits;
    size_t bytes = 0;
    int launches = 0;
    gba_part_enqueue(ctx, q, out, sh, p.smem_probe_cap, nullptr, &bytes, nullptr, nullptr, &launches, s);
    // (a workspace that had to grow would lose the counts at its front)
    const size_t counts = gba_round_up(size_t(8) << counted_bits, kAlign);
    const bool counted = attempt == 0 && counted_bits >= sh.bits && counts + bytes <= ctx->ws_bytes;
    const size_t front = counted ? counts : 0;
    gba_status st = gba_ws_reserve(ctx, front + bytes, s);
    if (st != GBA_OK) return st;
    if (!counted) GBA_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_small, 0, GBA_PART_STATUS, s));
    GbaTimer tm{ctx, s, k.timing != 0};
    unsigned char* W = static_cast<unsigned char*>(ctx->ws);
    st = gba_part_enqueue(ctx, q, out, sh, p.smem_probe_cap, W + front, &bytes, ctx->d_small, &tm, &launches, s,
                          counted ? reinterpret_cast<unsigned long long*>(W) : nullptr, counted_bits);
    if (st != GBA_OK) return st;
    GBA_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_small, ctx->d_small, 16, cudaMemcpyDeviceToHost, s));
    GBA_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    tm.collect();
    ctx->stats.main_rows += q.n;
    ctx->stats.main_bytes += q.n * int64_t(row_bytes(q));
    ctx->stats.kernel_launches += launches;
    const unsigned flags = *reinterpret_cast<unsigned*>(ctx->h_small);
    const unsigned long long count = *reinterpret_cast<unsigned long long*>(ctx->h_small + 8);
    if (flags & GBA_FLAG_WAIT_TIMEOUT) {
      ctx->err = "a bounded wait for a staged tile timed out";
      return GBA_ERR_TIMEOUT;
    }
    if (flags & GBA_FLAG_TABLE_OVERFLOW) {
      if (attempt >= k.max_regrow || sh.bits >= 20) {
        ctx->err = "partition fallback table overflow after " + std::to_string(attempt) + " retries";
        return GBA_ERR_TABLE_OVERFLOW;
      }
      ctx->stats.regrows++;
      sh.bits = std::min(20, sh.bits + 2);
      sh.groups *= 4;
      continue;
    }
    ctx->stats.preagg = 0;
    ctx->stats.table_slots = int64_t(sh.S);
    *n_groups = int64_t(count);
    ctx->stats.n_groups = int64_t(count);
    if (int64_t(count) > out->capacity) {
      ctx->err = "output capacity " + std::to_string(out->capacity) + " < " + std::to_string(count) + " groups";
      return GBA_ERR_OUTPUT_CAPACITY;
    }
    return GBA_OK;
  }
}
