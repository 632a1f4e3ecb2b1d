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

int gba_choose_strategy(const gba_context* ctx, const QDesc& q, const gba_knobs& k, double predicted_groups,
                        const GbaPlan& p) {
  (void)k;
  // The HBM-table strategy is fast while its table stays resident in L2
  // (126 MB; measured: random 64-bit atomics run at ~190 G/s below ~96 MB of
  // table and fall to 20-60 G/s above it).  Beyond that the partition
  // strategy's shared-memory tables win.
  const double slot = 8.0 * gba_gt_stride(q.naccs);
  const double groups = predicted_groups > 0 ? predicted_groups : double(q.n);
  (void)p;
  if (groups <= 1.1 * gba_part_agg_slots(q, 2, ctx->max_smem_optin)) return GBA_STRATEGY_TABLE;  // shared table holds all groups
  const double table_bytes = groups / 0.7 * slot;
  return table_bytes <= 80.0 * (1 << 20) ? GBA_STRATEGY_TABLE : GBA_STRATEGY_PARTITION;
}

gba_status gba_run_partition(gba_context* ctx, const QDesc& q, const gba_output* out, const gba_knobs& k,
                             const GbaPlan& p, double predicted_groups, cudaStream_t s, int64_t* n_groups) {
  ctx->stats.strategy = GBA_STRATEGY_PARTITION;
  const int64_t n = q.n;
  double groups = double(std::max<int64_t>(n, 1));
  const bool learned = k.sizing == GBA_SIZING_LEARNED && predicted_groups > 0;
  if (learned) groups = std::min(groups, predicted_groups * 1.25 + 64);
  auto slots = [&](int ctas) {
    const int s = gba_part_agg_slots(q, ctas, ctx->max_smem_optin);
    return k.smem_slots > 0 ? std::max(32, std::min(s, k.smem_slots) / 4 * 4) : s;
  };
  auto fan_out = [&](int ctas) {
    const double per_table = (learned ? kLearnedFill : kPlainFill) * slots(ctas);
    const int bits = int(std::ceil(std::log2(std::max(1.0, groups / per_table))));
    return std::max(1, std::min(k.partition_bits > 0 ? k.partition_bits : bits, 20));
  };
  // three aggregation CTAs per SM unless their smaller tables cost another
  // pass over the rows or another sweep of the keys
  const int b3 = fan_out(3), b2cta = fan_out(2);
  const int ctas = b3 > b2cta && (b3 > kOneSweepBits || (b2cta <= kOnePassBits && b3 > kOnePassBits)) ? 2 : 3;
  const int S = slots(ctas);
  int B = ctas == 3 ? b3 : b2cta;
  const size_t rb = row_bytes(q);
  // a partition of more than 2 Lp rows (a hot key) is cut into pieces of Lp
  const int64_t Lp = std::max<int64_t>(32768, n / (int64_t(ctx->sms) * 8));
  const int64_t max_split = n / (2 * Lp) + 1, max_pieces = 2 * (n / Lp) + 2;

  for (int attempt = 0;; ++attempt) {
    // one pass up to kOnePassBits digit bits, else two, the first one with the
    // fewer digits: its runs are spread over the whole row buffer (measured on
    // 2^28 rows of 24 bytes, 15 bits: 5.73 ms as 7 + 8, 6.73 as 8 + 7)
    const int b1 = B <= kOnePassBits ? B : B / 2, b2 = B - b1;
    ctx->stats.partition_bits = B;
    const int64_t nparts = int64_t(1) << B;
    int th1 = 512, th2 = 512;
    const int T1 = gba_part_tile_rows(q, b1, 0, false, ctx->max_smem_optin, &th1);
    const int T2 = b2 > 0 ? gba_part_tile_rows(q, b2, 1 << b1, false, ctx->max_smem_optin, &th2) : 0;
    const uint64_t fb_cap = std::max<uint64_t>(1 << 16, uint64_t(std::min<double>(groups * 0.02, 1 << 24)));

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
    gba_status st = gba_ws_reserve(ctx, cv.off, s);
    if (st != GBA_OK) return st;
    unsigned char* W = static_cast<unsigned char*>(ctx->ws);
    unsigned* d_flags = reinterpret_cast<unsigned*>(ctx->d_small);
    unsigned long long* d_count = reinterpret_cast<unsigned long long*>(ctx->d_small + 8);
    auto words = [&](size_t o) { return reinterpret_cast<unsigned long long*>(W + o); };
    GBA_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_small, 0, 64, s));
    GBA_CUDA_TRY(ctx, cudaMemsetAsync(W + o_zero, 0, 8 * size_t(nparts), s));
    GbaTimer tm{ctx, s, k.timing != 0};

    PartPlanArgs pl{};
    pl.bits1 = b1;
    pl.bits2 = b2;
    pl.hist = words(o_zero);
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
    tm.begin(3);
    GBA_CUDA_TRY(ctx, gba_launch_part_hist(q, B, words(o_zero), ctx->sms, s));
    GBA_CUDA_TRY(ctx, gba_launch_part_plan(pl, s));
    tm.end();

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
      tm.begin(3);
      GBA_CUDA_TRY(ctx, gba_launch_part_scatter(pp, int(std::min<int64_t>(tiles, ctx->sms * (1024 / pp.threads))), s));
      tm.end();
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
    pa.ctr = reinterpret_cast<unsigned*>(ctx->d_small + 20);
    pa.S = S;
    pa.nbk = std::max(p.smem_probe_cap, 64) / (q.key64 ? 2 : 4);
    pa.fallback = fb;
    pa.flags = d_flags;
    pa.out.keys = out->keys;
    for (int a = 0; a < GBA_MAX_AGGS; ++a) pa.out.accs[a] = static_cast<unsigned long long*>(out->aggs[a]);
    pa.out.capacity = out->capacity;
    pa.out.count = d_count;
    tm.begin(1);
    GBA_CUDA_TRY(ctx, gba_launch_part_agg(pa, ctas, int(std::min<int64_t>(nparts + max_pieces, ctx->sms * ctas)), s));
    tm.end();
    ctx->stats.main_rows += n;
    ctx->stats.main_bytes += n * int64_t(rb);
    tm.begin(2);
    GBA_CUDA_TRY(ctx, gba_launch_compact(
                          fb, q, pa.out, int(std::max<uint64_t>(1, std::min<uint64_t>(ctx->sms * 8, fb.cap / 256))), s,
                          &pl.plan->fb_cap));
    tm.end();
    GBA_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_small, ctx->d_small, 16, cudaMemcpyDeviceToHost, s));
    GBA_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    tm.collect();
    ctx->stats.kernel_launches += b2 > 0 ? 7 : 6;
    const unsigned flags = *reinterpret_cast<unsigned*>(ctx->h_small);
    const unsigned long long count = *reinterpret_cast<unsigned long long*>(ctx->h_small + 8);
    if (flags & GBA_FLAG_WAIT_TIMEOUT) {
      ctx->err = "a bounded wait for a staged tile timed out";
      return GBA_ERR_TIMEOUT;
    }
    if (flags & GBA_FLAG_TABLE_OVERFLOW) {
      if (attempt >= k.max_regrow || B >= 20) {
        ctx->err = "partition fallback table overflow after " + std::to_string(attempt) + " retries";
        return GBA_ERR_TABLE_OVERFLOW;
      }
      ctx->stats.regrows++;
      B = std::min(20, B + 2);
      groups *= 4;
      continue;
    }
    ctx->stats.preagg = 0;
    ctx->stats.table_slots = int64_t(S);
    *n_groups = int64_t(count);
    ctx->stats.n_groups = int64_t(count);
    if (int64_t(count) > out->capacity) {
      ctx->err = "output capacity " + std::to_string(out->capacity) + " < " + std::to_string(count) + " groups";
      return GBA_ERR_OUTPUT_CAPACITY;
    }
    return GBA_OK;
  }
}
