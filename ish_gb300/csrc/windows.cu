// windows.cu -- long records scored as overlapping windows.
//
// With a free target start, the best alignment of a query against a long
// record never spans more than a bounded number of record rows: a path over S
// rows makes at most one diagonal step per query column, so at least S - Q rows
// are a gap in the query, and its score is at most TOP - open - (S - Q - 1) * ext
// with TOP the sum of the columns' largest scores; the best score is at least
// LOW, the full-query diagonal's sum of the columns' smallest scores
// (semi-global), or positive (local).  So S <= O = Q + 1 + (TOP - open - LOW) /
// ext.  (The matrix's largest score in place of each column's made O 1,440 rows
// for 120 residues and blosum62, where it is about 750.)
//
// A window of a record that starts at row s runs the same recurrence from a
// top boundary that only holds paths the whole record also has: for s = 0 the
// query's own, for s > 0 the fixed-query-start one, H(s-1, j) = -(open +
// ext*j) -- a start on the free left boundary at row s-1 followed by a query
// gap.  (A free query start may begin a path at any query column on row 0
// only; letting a later window begin one there would invent alignments.)  It
// then scores every cell at most as high as the whole record does (its paths
// are a subset), and exactly as high at every cell whose best path starts
// inside the window.  Windows that
// overlap by O rows therefore hold, for the record's best cell (the first
// row, then the smallest column, of its maximum), that cell's exact value in
// some window, and no cell before it reaches that value in any window.  The
// record's result is the window result with the largest score, then the
// smallest record row, then the smallest query column -- exactly the
// whole-record result, end coordinates and tie rules included:
//   semi-global with free target start and end and a fixed query end (the
//     target-end maximum of semi_global_aln/striped.mojo:436-450);
//   local alignment (local_aln/striped.mojo:395-428).
//
// The point is load balance: a pass over records of very unequal lengths is
// bound by its longest record pairs, one group each, however many groups
// finish early.  Windows of equal length spread those records over all
// groups.  This file decides when to window, builds the window view of the
// set (windows of the long records plus the other records whole, longest
// first), scores it with the wavefront kernel into per-window results, and
// folds them per record on the device.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

#include "host.h"

namespace ish {

// Folds the window results of sorted entries (entry e: slots [cs[e], cs[e+1]),
// window w starting at record row start[w]) into their outputs: a warp for each
// of the first `multi` entries, a thread for each of the others, which are one
// window.  (With a thread for every entry, 60 records of 10 kb - 400 kb in 25,600
// windows of a 20-nt query took about 500 us to fold, 52 so; scoring them 76.)
__global__ void k_merge_windows(const uint32_t *orig_s, uint32_t n, uint32_t multi, const uint32_t *cs,
                                const uint32_t *start, const int32_t *ws, const int32_t *wq, const int32_t *wt,
                                int mode, OutDev out, Decision dec) {
  const uint32_t lane = threadIdx.x & 31, items = multi + (n - multi + 31) / 32;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < items; i += (gridDim.x * blockDim.x) >> 5) {
    const bool whole = i < multi;
    const uint32_t e = whole ? i : multi + (i - multi) * 32 + lane;
    if (e >= n) continue;
    const uint32_t a = cs[e], b = cs[e + 1];
    bool any = false;
    int bs = 0, bq = 0;
    long long bt = -1;
    // equal scores carry rows of the same kind (all -1 when nothing beat the
    // initial best), so the row and column order the ties
    auto take = [&](int sc, int tq, long long tt) {
      if (any && !(sc > bs || (sc == bs && tt >= 0 && (tt < bt || (tt == bt && tq < bq))))) return;
      any = true;
      bs = sc;
      bq = tq;
      bt = tt;
    };
    for (uint32_t w = whole ? a + lane : a; w < b; w += whole ? 32 : 1)
      take(ws[w], wq[w], wt[w] >= 0 ? (long long)wt[w] + start[w] : -1);
    if (whole) {
      for (int o = 16; o > 0; o >>= 1) {
        const bool has = __shfl_down_sync(0xffffffffu, any, o);
        const int sc = __shfl_down_sync(0xffffffffu, bs, o), tq = __shfl_down_sync(0xffffffffu, bq, o);
        const long long tt = __shfl_down_sync(0xffffffffu, bt, o);
        if (has) take(sc, tq, tt);
      }
      if (lane) continue;
    }
    const uint32_t o = orig_s[e];
    if (out.score) out.score[o] = bs;
    if (out.qend) out.qend[o] = bq;
    if (out.tend) out.tend[o] = (int32_t)bt;
    if (out.hit) out.hit[o] = decide(mode, bs, bq, (int)bt, dec);
  }
}

namespace host {

// The query as windows past row 0 run it: its start fixed.
static Query &fixed_start_of(Query &q) {
  if (!(q.algo == ISH_ALGO_SEMI_GLOBAL && (q.ends & ISH_FREE_QUERY_START))) return q;
  if (!q.fixed_start) {
    q.fixed_start.reset(new Query());
    clone_params(q, *q.fixed_start);
    q.fixed_start->ends = q.ends & ~ISH_FREE_QUERY_START;
  }
  return *q.fixed_start;
}

bool windowable_whole(const Query &q) { return !(q.algo == ISH_ALGO_SEMI_GLOBAL && (q.ends & ISH_FREE_QUERY_START)); }

// Rows two windows of a record must share (see above), or 0 when no bound
// holds for this query.
uint64_t window_overlap(const Query &q) {
  const int mode = q.algo == ISH_ALGO_LOCAL ? SW : SG;
  if (q.ext < 1 || q.Q == 0) return 0;
  if (mode == SG && !((q.ends & ISH_FREE_TARGET_START) && (q.ends & ISH_FREE_TARGET_END) &&
                      !(q.ends & ISH_FREE_QUERY_END)))
    return 0;
  const long long low = mode == SG ? q.col_min_sum : 0;
  const long long top = q.col_max_sum - q.open - low;
  const long long o = (long long)q.Q + 2 + std::max(0LL, (top + q.ext - 1) / q.ext);
  return (uint64_t)((o + 15) & ~15LL);
}

// Windows pay when the longest record exceeds ISH_WINDOW_QUARTERS / 4 of the
// rows a group scores on average: its pair alone would then outlast the pass.
// Measured with 4, 5 and 8 quarters on 1,000 to 200,000 proteins (20 to 1,000
// residues) where they differ: 60,000, local, 340 residues 1,679 / 1,681 / 1,962 us
// and 460 residues 2,106 / 2,107 / 2,182; 200,000, semi-global, 180 residues 1,777 /
// 1,780 / 1,877, but 220 residues 2,206 / 2,176 / 2,176 and local 180 residues 2,686
// / 2,640 / 2,643.
#ifndef ISH_WINDOW_QUARTERS
#define ISH_WINDOW_QUARTERS 5
#endif

// The window stride for scoring `rs` with groups of the given shape, or 0
// when windows would not help: the longest record must exceed 1.25x the rows a
// group scores on average (see above) and one window.  Narrow windows spread
// the records over more groups and wide ones repeat fewer rows, so strides are
// compared by a model.  With pairs of windows for less than half the groups, a
// pass takes one window at the rate of that many warps; with more, all rows at
// the full device's rate and 0.4 windows for the uneven end (0.3 to 0.5 measured
// alike, 0.8 and 1.2 worse; one round that just fits is not trusted to).  With a
// stride of at least 8 x O, 10 records of 10 kb - 1 Mb made 32 windows for 1,000
// nt (11.4 ms; 2.2 ms with this rule), 200 records 1,102 (11.7 ms; 8.4 ms).
uint64_t window_stride(const ish_ctx *ctx, const RecordSet &rs, uint64_t O, int G, int K, int mode) {
  const int lean = wave_lean(ctx, K, mode, PROF_S32);
  // groups in flight and the rows each would score on average (two records
  // per pair share their rows)
  const uint64_t groups = (uint64_t)ctx->num_sms * wave_sm_threads(K, lean) / G;
  const uint64_t avg_rows = rs.total / 2 / std::max<uint64_t>(groups, 1);
  if (rs.max_len * 4 <= avg_rows * ISH_WINDOW_QUARTERS) return 0;
  // rows in records longer than 2^(i/8) (all of them where the set has no
  // histogram)
  constexpr int BINS = 8 * 33;
  std::vector<double> above(BINS + 1, 0.0);
  auto bin_of = [](double len) { return std::min(BINS - 1, std::max(0, (int)(8 * std::log2(std::max(len, 1.0))))); };
  for (uint32_t b = 1; b < rs.hist.size(); ++b)
    if (rs.hist[b]) {
      const double len = b < 32768 ? b : 32768 + 32.0 * (b - 32768) + 16;
      above[bin_of(len)] += len * rs.hist[b];
    }
  if (rs.hist.empty()) above[BINS - 1] = (double)rs.total;
  for (int i = BINS - 1; i >= 0; --i) above[i] += above[i + 1];
  const double warps = (double)groups * G / 32;
  uint64_t best = 0;
  double best_t = 1e300;
  for (double w = 256; w + O < rs.max_len; w *= 1.08) {
    const double cut = above[bin_of(w + O)];  // rows that are cut into windows
    const double work = (rs.total + cut * (double)O / w) / 2;
    const double pairs = std::ceil((cut / w + rs.n) / 2);
    const double full = row_clocks(ctx, mode, K, G, warps);
    const double t = 2 * pairs >= groups ? work / groups * full + 0.4 * (w + O) * full
                                         : 1.15 * (w + O) * row_clocks(ctx, mode, K, G, pairs * G / 32);
    if (t < best_t) {
      best_t = t;
      best = ((uint64_t)w + 15) & ~15ull;
    }
  }
  return best + O < rs.max_len ? best : 0;
}

// Builds the window view of sorted entries [0, nonempty) of rs (stride W,
// overlap O) into V, unless V already holds it.  split: the windows at record
// row 0 first (a second launch scores the others).
int build_window_view(ish_ctx *ctx, const RecordSet &rs, uint32_t nonempty, uint64_t W, uint64_t O, bool split,
                      WindowView &V, cudaStream_t s) {
  if (V.nw && V.W == W && V.O == O && V.split == split && V.entries == nonempty) return ISH_OK;
  V.nw = 0;  // (its buffers may be those of an earlier view)
  std::vector<uint32_t> len(nonempty);
  std::vector<uint64_t> off(nonempty);
  CU(cudaStreamSynchronize(s));
  CU(cudaMemcpy(len.data(), rs.len_s.p, (size_t)nonempty * 4, cudaMemcpyDeviceToHost));
  CU(cudaMemcpy(off.data(), rs.off_s.p, (size_t)nonempty * 8, cudaMemcpyDeviceToHost));
  // slots: the windows of entry e are [cs[e], cs[e+1]); each has a first
  // record row, a length and a code offset
  std::vector<uint32_t> cs(nonempty + 1), wstart, wlen;
  std::vector<uint64_t> woff;
  V.multi = 0;
  for (uint32_t e = 0; e < nonempty; ++e) {
    cs[e] = (uint32_t)wstart.size();
    const uint64_t L = len[e];
    if (L <= W + O) {
      wstart.push_back(0);
      wlen.push_back((uint32_t)L);
      woff.push_back(off[e]);
      continue;
    }
    V.multi = e + 1;
    // window k covers [k * W, (k + 1) * W + O): the cells it adds to the windows
    // before it lie O rows or more below its start
    for (uint64_t st = 0;; st += W) {
      const uint64_t en = std::min<uint64_t>(L, st + W + O);
      wstart.push_back((uint32_t)st);
      wlen.push_back((uint32_t)(en - st));
      woff.push_back(off[e] + st);
      if (en == L) break;
    }
  }
  const uint32_t nw = (uint32_t)wstart.size();
  cs[nonempty] = nw;
  // the view: longest first, with split those that start at record row 0 before
  // the others (pairs of similar length; a long window at the end of a launch runs
  // alone: 60,000 proteins, local, 460 residues 3,129 us with the others always
  // behind, 2,112 us so)
  std::vector<uint32_t> order(nw);
  std::iota(order.begin(), order.end(), 0u);
  std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
    if (split && (wstart[a] == 0) != (wstart[b] == 0)) return wstart[a] == 0;
    return wlen[a] > wlen[b];
  });
  uint32_t n_first = 0;
  while (n_first < nw && (!split || wstart[order[n_first]] == 0)) ++n_first;
  std::vector<uint32_t> vlen(nw), vslot(nw);
  std::vector<uint64_t> voff(nw);
  uint64_t vtotal = 0;
  for (uint32_t i = 0; i < nw; ++i) {
    vlen[i] = wlen[order[i]];
    voff[i] = woff[order[i]];
    vslot[i] = order[i];
    vtotal += vlen[i];
  }
  CU(V.off.ensure((size_t)nw * 8));
  CU(V.len.ensure((size_t)nw * 4));
  CU(V.slot.ensure((size_t)nw * 4));
  CU(V.start.ensure((size_t)nw * 4));
  CU(V.cs.ensure((size_t)(nonempty + 1) * 4));
  CU(cudaMemcpyAsync(V.off.p, voff.data(), (size_t)nw * 8, cudaMemcpyHostToDevice, s));
  CU(cudaMemcpyAsync(V.len.p, vlen.data(), (size_t)nw * 4, cudaMemcpyHostToDevice, s));
  CU(cudaMemcpyAsync(V.slot.p, vslot.data(), (size_t)nw * 4, cudaMemcpyHostToDevice, s));
  CU(cudaMemcpyAsync(V.start.p, wstart.data(), (size_t)nw * 4, cudaMemcpyHostToDevice, s));
  CU(cudaMemcpyAsync(V.cs.p, cs.data(), (size_t)(nonempty + 1) * 4, cudaMemcpyHostToDevice, s));
  CU(cudaStreamSynchronize(s));  // the arrays are temporaries
  V.W = W;
  V.O = O;
  V.split = split;
  V.entries = nonempty;
  V.nw = nw;
  V.n_first = n_first;
  V.total = vtotal;
  V.max_len = *std::max_element(vlen.begin(), vlen.end());
  return ISH_OK;
}

// A record set over rs's codes whose entries are the windows of V (the
// buffers are borrowed: the view is never released).
RecordSet window_set(const RecordSet &rs, const WindowView &V) {
  RecordSet view;
  view.n = V.nw;
  view.total = V.total;
  view.max_len = V.max_len;
  view.codes = rs.codes;
  view.off_s = V.off;
  view.len_s = V.len;
  view.orig_s = V.slot;
  return view;
}

// Folds per-window results into the records' outputs.
int merge_windows(ish_ctx *ctx, const RecordSet &rs, uint32_t nonempty, const WindowView &V, const Query &q,
                  const int32_t *ws, const int32_t *wq, const int32_t *wt, OutDev out, cudaStream_t s,
                  uint32_t *kernels) {
  const int mode = q.algo == ISH_ALGO_LOCAL ? SW : SG;
  const uint64_t warps = V.multi + ceil_div(nonempty - V.multi, 32);
  const uint32_t nb = std::max<uint32_t>(1, std::min<uint32_t>(ceil_div(warps * 32, 256), (uint32_t)ctx->num_sms * 8));
  k_merge_windows<<<nb, 256, 0, s>>>(rs.orig_s.as<const uint32_t>(), nonempty, V.multi, V.cs.as<const uint32_t>(),
                                     V.start.as<const uint32_t>(), ws, wq, wt, mode, out,
                                     Decision{q.max_score, q.thr});
  if (kernels)
    ++*kernels;  // a captured launch: the caller counts it per replay
  else
    ++ctx->launches;
  CU(cudaGetLastError());
  return ISH_OK;
}

// Scores sorted entries [0, nonempty) of rs through the window view when its
// longest records would bound the pass; *done is false when it did nothing.
// The view is built once per (set, stride, overlap) and kept with the set.
int launch_windows(ish_ctx *ctx, Query &q, RecordSet &rs, uint32_t nonempty, OutDev out, cudaStream_t s,
                   bool *done) {
  *done = false;
  if (!ctx->windows_on || ctx->kernel != ISH_KERNEL_AUTO || nonempty == 0 || nonempty > (1u << 22)) return ISH_OK;
  const uint64_t O = window_overlap(q);
  if (!O) return ISH_OK;
  const int mode = q.algo == ISH_ALGO_LOCAL ? SW : SG;
  int G, K, layout;
  pick_shape(ctx, q, &G, &K, &layout);
  if (!G || !wave_fits(q, G, K, layout) || !regime(q, G * K).fast) return ISH_OK;
  const uint64_t W = window_stride(ctx, rs, O, G, K, mode);
  if (!W) return ISH_OK;
  WindowView &V = rs.windows;
  int rc = build_window_view(ctx, rs, nonempty, W, O, !windowable_whole(q), V, s);
  if (rc) return rc;
  const uint32_t nw = V.nw;
  WindowOut &R = ctx->window_out;
  CU(R.score.ensure((size_t)nw * 4));
  CU(R.qend.ensure((size_t)nw * 4));
  CU(R.tend.ensure((size_t)nw * 4));
  CU(R.hit.ensure((size_t)nw));
  // Sets without a histogram (reversed prefixes) may hold empty entries, which no
  // kernel writes: their end row is 0.
  if (rs.hist.empty()) CU(cudaMemsetAsync(R.tend.p, 0, (size_t)nw * 4, s));
  RecordSet view = window_set(rs, V);
  pick_shape(ctx, q, &G, &K, &layout, &view);  // the windows may be few
  OutDev wout{R.score.as<int32_t>(), R.qend.as<int32_t>(), R.tend.as<int32_t>(), R.hit.as<uint8_t>()};
  Query &qc = fixed_start_of(q);
  if (&qc == &q) {
    rc = launch_wave_range(ctx, q, view, 0, nw, wout, G, K, layout, s);
  } else {
    rc = launch_wave_range(ctx, q, view, 0, V.n_first, wout, G, K, layout, s);
    if (!rc && nw > V.n_first) rc = launch_wave_range(ctx, qc, view, V.n_first, nw - V.n_first, wout, G, K, layout, s);
  }
  if (!rc)
    rc = merge_windows(ctx, rs, nonempty, V, q, R.score.as<const int32_t>(), R.qend.as<const int32_t>(),
                       R.tend.as<const int32_t>(), out, s, nullptr);
  if (rc) return rc;
  ctx->last_windows = nw;
  *done = true;
  return ISH_OK;
}

}  // namespace host
}  // namespace ish
