// ish_gpu.cu -- host side of libish_gpu.so: the C ABI declared in
// include/ish_gpu.h.  It owns device memory, pinned staging and the engine
// stream, packs record sets in HBM, builds query profiles and picks and
// launches the scoring kernels.
#include <algorithm>
#include <cerrno>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "host.h"

using namespace ish;

using namespace ish::host;

namespace ish {
namespace host {

thread_local std::string g_open_error;
thread_local std::string *thread_error = nullptr;
std::atomic<int64_t> g_alloc_fault{-1};

int fail(ish_ctx *c, int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (thread_error) *thread_error = buf;
  else if (c) c->err = buf;
  else g_open_error = buf;
  return code;
}

void release_query(Query &q) {
  q.plain_prof.release();
  q.plain_hinit.release();
  for (auto &l : q.layouts) {
    l.second.prof.release();
  }
  q.layouts.clear();
  for (auto &kv : q.exact_prof) kv.second.release();
  q.exact_prof.clear();
  if (q.reverse) release_query(*q.reverse);
  q.reverse.reset();
  if (q.fixed_start) release_query(*q.fixed_start);
  q.fixed_start.reset();
}

void release_set(RecordSet &rs) {
  DevBuf *b[] = {&rs.codes, &rs.off_s, &rs.len_s, &rs.orig_s, &rs.inv};
  for (DevBuf *x : b) x->release();
  rs.windows.release();
}

// Freed sets keep their device buffers for the next load: at most two sets,
// each with packed codes under a sixteenth of device memory (at least 1 GiB),
// so the cache stays small next to HBM; an allocation of codes that fails gives
// the cached buffers back first (ensure_codes).
static constexpr size_t kSpareSets = 2;
static size_t spare_codes_max(const ish_ctx *ctx) { return std::max<size_t>(size_t(1) << 30, ctx->mem_total / 16); }

void recycle_set(ish_ctx *ctx, RecordSet &rs) {
  rs.windows.clear();
  if (!rs.codes.p || rs.codes.cap > spare_codes_max(ctx)) {
    release_set(rs);
    return;
  }
  if (ctx->spare_sets.size() >= kSpareSets) {
    release_set(ctx->spare_sets.front());
    ctx->spare_sets.erase(ctx->spare_sets.begin());
  }
  RecordSet keep;
  keep.codes = rs.codes;
  keep.off_s = rs.off_s;
  keep.len_s = rs.len_s;
  keep.orig_s = rs.orig_s;
  keep.inv = rs.inv;  // (inv_ready is not kept: the next set rebuilds it)
  keep.windows = rs.windows;
  ctx->spare_sets.push_back(keep);
  rs.codes = rs.off_s = rs.len_s = rs.orig_s = rs.inv = DevBuf{};
  rs.inv_ready = false;
  rs.windows = WindowView{};
}

// Hands `rs` the spare buffers with the smallest code area that holds
// codes_bytes (buffers that are still too small grow in DevBuf::ensure).
void take_spare_set(ish_ctx *ctx, RecordSet &rs, size_t codes_bytes) {
  if (rs.codes.p || ctx->spare_sets.empty()) return;
  size_t pick = ctx->spare_sets.size();
  for (size_t i = 0; i < ctx->spare_sets.size(); ++i) {
    const size_t cap = ctx->spare_sets[i].codes.cap;
    if (cap >= codes_bytes && (pick == ctx->spare_sets.size() || cap < ctx->spare_sets[pick].codes.cap)) pick = i;
  }
  if (pick == ctx->spare_sets.size()) return;
  RecordSet &sp = ctx->spare_sets[pick];
  rs.codes = sp.codes;
  rs.off_s = sp.off_s;
  rs.len_s = sp.len_s;
  rs.orig_s = sp.orig_s;
  rs.inv = sp.inv;
  rs.windows = sp.windows;
  ctx->spare_sets.erase(ctx->spare_sets.begin() + pick);
}

// Gives back start finding's buffers, and the window views and inverse orders of
// freed sets; false where there were none.
static bool give_back_starts(ish_ctx *ctx) {
  WindowView &v = ctx->starts_windows;
  size_t held = ctx->starts_ws.cap + ctx->starts_codes.cap + v.off.cap;
  for (const RecordSet &sp : ctx->spare_sets) held += sp.inv.cap;
  if (!held) return false;
  ctx->starts_ws.release();
  ctx->starts_codes.release();
  v.release();
  for (RecordSet &sp : ctx->spare_sets) {
    sp.inv.release();
    sp.windows.release();
  }
  return true;
}

cudaError_t grow(ish_ctx *ctx, DevBuf &b, size_t bytes) {
  cudaError_t e = b.ensure(bytes);
  if (e == cudaErrorMemoryAllocation && give_back_starts(ctx)) {
    (void)cudaGetLastError();
    e = b.ensure(bytes);
  }
  return e;
}

void compute_rows(Query &q) {
  const int A = q.alphabet;
  q.rowmap.assign(256, 0);
  q.rep.clear();
  std::map<std::vector<int8_t>, int> seen;
  std::vector<int8_t> key(q.Q);
  for (int c = 0; c < A; ++c) {
    for (int j = 0; j < q.Q; ++j) key[j] = q.M[(size_t)c * A + q.q[j]];
    auto it = seen.find(key);
    if (it == seen.end()) {
      it = seen.emplace(key, (int)q.rep.size()).first;
      q.rep.push_back((uint8_t)c);
    }
    q.rowmap[c] = (uint8_t)it->second;
  }
  q.rows = (int)q.rep.size();
}

int matrix_alphabet_ok(uint32_t alphabet) { return alphabet >= 1 && alphabet <= 256; }

// Safe-regime checks (see engine.cuh): the fast kernels evaluate plain Gotoh
// in 16-bit lanes; the result equals the reference's striped int16 pass when
// gap_open > gap_extend and no lane value of the reference can saturate or
// wrap.  Bounds are conservative.

// Whether a shape usually runs the lean build (see the kernels' launch bounds in
// kernels.cuh), from 200,000 proteins (G = 8 and 16; 16- and 32-bit profiles) and
// 200,000 reads of 150 (G = 4 and 8; pair profile).  Semi-global rows need so few
// registers that the builds with more warps are ahead or level: 0-6 % at K = 25..32
// (K = 27 -3 %), 4-17 % at K = 34..48.  Local alignment keeps a row maximum and
// more state, and its builds with more warps spill from K = 25 on but for 34 (24 to
// 52 bytes read back at K = 25..27, 36 and 38, 60 to 240 elsewhere).  On proteins the
// lean build is ahead by 0-7 % at K = 27..32 and, where it has 8 warps against 12,
// 10 % behind at K = 34..38, level at 42 and 3-12 % ahead from 44 (32 threads: 1.6
// times at 46).  Pair profiles, with half the loads in flight, keep the 12 warps 3
// to 14 % ahead at all K from 34.  (lean_for weighs the set in.)
int wave_lean(const ish_ctx *ctx, int K, int mode, int layout) {
  if (!wave_has_lean(K)) return 0;
  if (ctx->force_lean >= 0) return ctx->force_lean;
  return mode == SW && ((K >= 27 && K <= 32) || (K >= 42 && layout != PROF_PAIR));
}

// Semi-global rows are held in frames that rise by ext per row and drop back
// to 0 every R rows, R a power of two with R * ext <= 2048 (the headroom the
// regime keeps above the largest score).
int frame_rows(int ext) {
  int R = 1;
  while (R < (1 << 20) && (long)2 * R * std::max(ext, 1) <= 2048) R *= 2;
  return R;
}

Regime regime(const Query &q, int qpad) {
  Regime r;
  if (q.Q == 0) return r;
  if (!(q.open > q.ext) || q.ext < 0) return r;
  const long top = (long)(q.Q + 1) * std::max(q.mmax, 1);
  if (top > 30000) return r;
  if (q.algo == ISH_ALGO_LOCAL) {
    r.fast = true;
    r.max_safe_len = ~0ull;
    return r;
  }
  if (q.open + q.ext > 10000) return r;
  if (frame_rows(q.ext) < WAVE_RPS_SG) return r;  // row frames reset at step boundaries (see frame_rows)
  const long base = 2L * q.open + (long)q.ext * (qpad + 3) + std::abs(q.mmin) + 64;
  if (base > 30000) return r;
  r.fast = true;
  if (q.ends & ISH_FREE_TARGET_START) {
    r.max_safe_len = ~0ull;
  } else {
    const long room = 30000 - base - q.open;
    r.max_safe_len = q.ext > 0 ? (uint64_t)(room / q.ext) : ~0ull;
  }
  return r;
}

int neg_limit_of(int open, int mmin) {
  // v_neg_limit (ishlib/matcher/alignment/semi_global_aln/striped.mojo:329-334)
  const int16_t o = (int16_t)open;
  if ((int16_t)(-o) < (int16_t)mmin) return (int16_t)(-32768 + o + 1);
  return (int16_t)(-32768 - mmin + 1);
}

// Scheduler clocks of one warp-row (one row of 32 / G record pairs) with the
// warps of a full SM taking turns, and of one row of a warp that has its
// scheduler to itself (the chain of its columns, shuffles and loads).  Straight
// lines through measurements at G = 8 and 16, proteins, K = 4..64 (semi-global 87
// at K = 4, 180 at 16, 326 at 32, 384 at 38, 631 at 60; local 184, 258, 468, 561,
// 1,032; alone 451 / 752 at K = 32, 619 / 1,074 at 48), with what the builds with
// fewer warps add, and wide groups (32 threads 9 % at K = 16..32 on proteins: most
// steps of a warp start a pair in one of its threads).
// `lean` is the build; where the other one is the usual choice, it costs what that
// measured (see wave_lean).
static double warp_row_clocks(const ish_ctx *ctx, int mode, int K, int G, int layout, int lean) {
  double c = 1.0 + 0.1 * (G / 32.0) * (G / 32.0);
  if (mode == SG) c *= (50 + 8.6 * K) * (K > 48 ? 1.1 : 1.0);
  else c *= (50 + 13.3 * K) * (K > 48 ? 1.11 + 0.02 * std::max(0, K - 56) : K > 40 ? 1.08 : 1.0);
  if (lean == wave_lean(ctx, K, mode, layout)) return c;
  if (!lean) return c * (K <= 32 ? 1.04 : G < 32 ? 1.08 : 1.3);
  return c * (mode == SG ? (K <= 32 ? 1.05 : 1.1) : K <= 26 ? 1.02 : K < 40 ? 1.1 : layout == PROF_PAIR ? 1.07 : 1.0);
}
static double lone_row_clocks(int mode, int K) { return mode == SG ? 150 + 9.5 * K : 200 + 17.5 * K; }

// Warps per scheduler of a full SM, by the kernels' launch bounds.
static double full_warps(int K, int lean) { return wave_sm_threads(K, lean) / 128; }

// Clocks in which each of `warps` warps on the device advances by one row: from
// one warp per scheduler to a full SM about linear (K = 32: 451 alone, 740 with
// two, 1,300 with four).
static double build_row_clocks(const ish_ctx *ctx, int K, int lean, double warps, double full, double lone) {
  const double w = std::max(1.0, warps / (4.0 * ctx->num_sms)), cap = full_warps(K, lean);
  return lone + (w - 1) / (cap - 1) * std::max(0.0, cap * full - lone);
}
double row_clocks(const ish_ctx *ctx, int mode, int K, int G, double warps) {
  const int lean = wave_lean(ctx, K, mode, PROF_S32);
  return build_row_clocks(ctx, K, lean, warps, warp_row_clocks(ctx, mode, K, G, PROF_S32, lean), lone_row_clocks(mode, K));
}

// Modelled time of one query against `set` (null: many records) with G threads x
// K columns and a build: every group's share of the rows at the rate of the warps
// in flight, then what the longest pair has left, alone (it ran at the same rate
// as the others until then), and the group's last thread, 4 rows behind each
// before it.  `share` queries run at once.  Four costs come on top of a row:
//   - in local alignment, the ends of records shorter than proteins (reads of 150
//     against proteins: 28 to 40 clocks at K = 8, 49 to 65 at 24, 62 at 40, 102 at
//     56);
//   - in groups narrower than a quarter-warp, the pairs that the other groups of
//     the warp begin and end (reads of 150: 32 groups per warp 115 clocks more than
//     four, 16 groups 45, eight 11; local half as much again);
//   - there, with too large a profile to repeat their slices (profile_slots), bank
//     conflicts (proteins, four threads: 849 -> 1,261 clocks at K = 52 -> 54, local
//     1,260 -> 1,564);
//   - with a free query end, the steps taken row by row while a record's end goes
//     through the group (reads of 150, K = 24: 40 clocks for eight threads, 77 for
//     16, 162 for 32; proteins 29 for 16, 57 for 32).
// Of 500 measured times (3,000 to 200,000 proteins, 20 to 2,047 residues, every
// shape and build without windows) the model is off by 6 % (standard deviation; 13
// % with the longest pair taken to run alone from the start), and the shape it
// takes is 0.2 % slower than the best, at most 8 %.
struct ShapeCost {
  double each = 0, clocks = 0;  // rows of a group; modelled clocks
};
static ShapeCost shape_cost(const ish_ctx *ctx, const Query &q, int G, int K, int layout, int lean, const RecordSet *set,
                            double share) {
  const int mode = q.algo == ISH_ALGO_LOCAL ? SW : SG;
  const double n = set ? std::max(1.0, (double)set->n - set->n_empty) : 0, length = set ? std::max(1.0, set->total / n) : 350;
  double more = mode == SW ? 260 * (40 + K) * std::max(0.0, 1 / length - 1 / 350.0) : 0.0, times = 1;
  if (mode == SG && (q.ends & ISH_FREE_QUERY_END)) more = (150 + 28 * K) * std::min(0.25, G / length);
  const double narrow = G < 8 ? (mode == SG ? 500 : 750) * (32 / G - 4) / length : 0.0;
  if (G < 8 && profile_slots(layout, q.rows, G, K) < 8) {
    if (layout == PROF_PAIR) times = mode == SG ? 1.1 : 1.0;
    else times = mode == SG ? 1.55 : 1.2;
  }
  const double row = (warp_row_clocks(ctx, mode, K, G, layout, lean) + more + narrow) * times;
  ShapeCost c;
  if (!set) {
    c.clocks = G * row;
    return c;
  }
  const double lone = (lone_row_clocks(mode, K) + more) * times;
  const double pairs = std::max(1.0, n / 2) * share, rows = set->total / 2.0 * share;
  const double warps = std::max(1.0, std::min(std::ceil(pairs * G / 32), 4.0 * ctx->num_sms * full_warps(K, lean)));
  c.each = rows * G / 32 / warps;
  c.clocks = c.each * build_row_clocks(ctx, K, lean, warps, row, lone) +
             (std::max(0.0, (double)set->max_len - c.each) + 4 * G) * lone;
  return c;
}

// The build for a shape and a set, and the modelled clocks with it.  Where all
// pairs are in flight at once in the build with fewer warps, the other one has no
// more of them, and fewer registers (3,000 proteins: 2 % behind to 23 % ahead at K
// = 25..46).  Else, where the longest pair has much more than its share of the
// rows, the one with the smaller modelled time: with fewer warps that pair runs
// faster (15,000 proteins, 32 threads x 32 columns: 1,376 us with 512 threads per
// SM, 1,222 with 384).
static double shape_clocks(const ish_ctx *ctx, const Query &q, int G, int K, int layout, const RecordSet *set, double share,
                           int *build = nullptr) {
  const int usual = wave_lean(ctx, K, q.algo == ISH_ALGO_LOCAL ? SW : SG, layout);
  ShapeCost c = shape_cost(ctx, q, G, K, layout, usual, set, share);
  int lean = usual;
  if (set && wave_has_lean(K) && ctx->force_lean < 0) {
    const bool all = (set->n - set->n_empty) / 2.0 * share * G / 32 <= 4.0 * ctx->num_sms * full_warps(K, 1);
    if (all ? !usual : set->max_len > 1.5 * c.each) {
      const ShapeCost o = shape_cost(ctx, q, G, K, layout, !usual, set, share);
      if (all || o.clocks < 0.97 * c.clocks) {
        c = o;
        lean = !usual;
      }
    }
  }
  if (build) *build = lean;
  return c.clocks;
}
double shape_rate(const ish_ctx *ctx, const Query &q, int G, int K, int layout) {
  return shape_clocks(ctx, q, G, K, layout, nullptr, 1);
}
int lean_for(const ish_ctx *ctx, const Query &q, int G, int K, int layout, const RecordSet *set, double share) {
  int lean = 0;
  shape_clocks(ctx, q, G, K, layout, set, share, &lean);
  return lean;
}

// Columns per thread (K) and threads per group (G) with the smallest modelled
// time among those with G*K >= Q + 1.  Kernels exist for every K <= 32 and even
// K up to 64.
int wave_k_available(int k) { return (k >= 1 && k <= 32) || (k > 32 && k <= WAVE_KMAX && !(k & 1)); }

static int shape_layout(const ish_ctx *ctx, const Query &q, int G, int K) {
  if (ctx->force_layout >= 0) return ctx->force_layout;
  return G ? choose_layout(ctx, q.rows, G, K, q.algo == ISH_ALGO_LOCAL ? SW : SG, q.ends) : (int)PROF_S16;
}

static void choose_shape(const ish_ctx *ctx, const Query &q, const RecordSet *set, double share, int *G, int *K) {
  // Of shapes that the model does not tell apart a launch for several queries takes
  // the widest group: near-equal queries then have the same columns, and one kernel
  // (six of 26 to 31 nt against 1,000 lines 99 -> 77 us).
  const double same = set && share > 1 ? 1.04 : 1.0;
  double bestc = 1e30;
  int bg = 0, bk = 0;
  for (int g = 1; g <= 32; g <<= 1) {
    if (ctx->force_G && g != ctx->force_G) continue;
    int k = ctx->force_K ? ctx->force_K : (q.Q + 1 + g - 1) / g;
    if (!ctx->force_K && k > 32) k = (k + 1) & ~1;
    if (!wave_k_available(k) || g * k < q.Q + 1) continue;
    const double c = shape_clocks(ctx, q, g, k, shape_layout(ctx, q, g, k), set, share);
    if (c < bestc * same) {
      bestc = std::min(c, bestc);
      bg = g;
      bk = k;
    }
  }
  *G = bg;
  *K = bk;
}

// Autotuner key: mode, profile rows (the profile's size) and query length.
uint64_t tune_key(int mode, int rows, int Q) { return ((uint64_t)mode << 48) | ((uint64_t)rows << 32) | (uint32_t)Q; }

// Row stride (in words) of a profile layout.  Strides are an odd number of
// 16-byte units: the eight threads of a quarter-warp read consecutive rows
// with 16-byte loads, and an odd stride spreads them over all 32 banks.
int layout_stride(int layout, int K) {
  if (layout == PROF_S16) {
    int kp = (K + 7) & ~7;
    return ((kp / 8) & 1) ? kp : kp + 8;
  }
  int kp = (K + 3) & ~3;
  return ((kp / 4) & 1) ? kp : kp + 4;
}

static size_t slots_bytes(int layout, int alphabet, int slots, int K) {
  const size_t per = (size_t)slots * layout_stride(layout, K);
  if (layout == PROF_PAIR) return (size_t)alphabet * alphabet * per * 4;
  if (layout == PROF_S32) return (size_t)alphabet * per * 4;
  return (size_t)alphabet * per * 2;
}

// Thread slices per profile row.  A quarter-warp loads 16 bytes per thread, and
// eight consecutive slices of a row lie in different banks, so groups of eight
// threads or more never conflict; narrower groups of a quarter-warp read rows
// of different codes that start at the same banks.  Their slices are repeated
// up to eight per row, one set for each group of the quarter-warp, as long as
// the profile stays at 44 KB (three blocks of a batched launch still fit an SM with
// local alignment's widest rows beside it).  Measured on 300,000 proteins, semi-global: four
// threads x 16 columns 4,155 -> 6,565 GCUPS, x 38 columns 4,661 -> 7,924.
int profile_slots(int layout, int alphabet, int G, int K) {
  return G < 8 && slots_bytes(layout, alphabet, 8, K) <= 44 * 1024 ? 8 : G;
}

size_t layout_bytes(int layout, int alphabet, int G, int K) {
  return slots_bytes(layout, alphabet, profile_slots(layout, alphabet, G, K), K);
}

// Shared memory of a wavefront block: the profile, a slot word per thread, and
// (local alignment) wave_save_words(K) save words per thread (see wave.cuh).
static size_t wave_smem(size_t prof_area, int threads, int K, int mode) {
  return prof_area + (size_t)threads * 4 * (1 + (mode == SW ? wave_save_words(K) : 0));
}
// What a block may ask for: 227 KB less the kernels' static copy of their
// parameters.
static constexpr size_t WAVE_SMEM_MAX = 226 * 1024;

// Threads of the largest block of this shape that fits beside the profile: all
// the SM's registers allow, or fewer where their saved rows do not fit.
static int wave_fit_threads(size_t prof_area, int K, int mode, int lean) {
  if (prof_area > WAVE_SMEM_MAX) return 0;
  const size_t warp = wave_smem(0, 32, K, mode);
  return (int)std::min<size_t>(wave_sm_threads(K, lean), (WAVE_SMEM_MAX - prof_area) / warp * 32);
}

// The pair layout (no per-column work to assemble a record pair's word, half
// the shared-memory loads of the 32-bit one) while all of an SM's threads fit
// beside it; else 32-bit single-code words: for semi-global while three quarters
// of them do, for local alignment while all do; else 16-bit words, whose PRMT per
// column costs semi-global what up to a quarter of the warps do and local
// alignment next to nothing (32 threads on 120,000 proteins, 32-bit / 16-bit: 52
// columns 16.4 / 16.8 ms with all threads beside both, 56 columns 22.4 / 18.0
// with three quarters beside the first).
// Measured: 1,000 nt x 200,000 reads, semi-global, 7,820 GCUPS with the 115 KB
// pair profile, 6,920 with 32-bit words, 5,930 with 16-bit ones; 1,501 residues x
// 100,000 proteins 7,440 with the 160 KB 32-bit profile, 6,600 with 16-bit words;
// 1,900 residues, local, where 96 of 256 threads fit beside the 32-bit profile,
// 3,165 against 4,670 with 16-bit words.
// With a free query end every thread copies its row to local memory where a
// record ends, and wide groups on short records do little else: the copies have
// to stay in the L1 that the profile leaves of 256 KB.  160,000 reads of 150 nt,
// 32 threads, pair / 32-bit profile: 44 columns (208 KB with the copies) 7.2 /
// 7.9 ms, 48 (240) 10.4 / 8.6, 60 (253) 14.6 / 13.1, 64 (281) 31.4 / 14.0.
// 120,000 proteins, 32-bit / 16-bit: 56 (241) 16.4 / 17.0, 60 (245) 17.6 / 17.6,
// 62 (271) 28.9 / 18.1.
int choose_layout(const ish_ctx *ctx, int rows, int G, int K, int mode, int ends) {
  auto threads = [&](int layout) { return wave_sm_threads(K, wave_lean(ctx, K, mode, layout)); };
  auto fit = [&](int layout, size_t most) {
    const size_t prof = ((layout_bytes(layout, rows, G, K) + 15) & ~(size_t)15) + 256;
    if (mode == SG && (ends & ISH_FREE_QUERY_END) && prof + (size_t)threads(layout) * K * 4 > most * 1024) return 0;
    return wave_fit_threads(prof, K, mode, wave_lean(ctx, K, mode, layout));
  };
  if (fit(PROF_PAIR, 224) == threads(PROF_PAIR)) return PROF_PAIR;
  if (4 * fit(PROF_S32, 246) >= (mode == SG ? 3 : 4) * threads(PROF_S32)) return PROF_S32;
  return PROF_S16;
}

// For a set with few or very unequal records a wider group can finish sooner
// than the shape with the highest rate: 3,000 proteins against 120 residues ran
// 31 columns per thread at the pace of the longest record's one group.  The
// padded query counts towards the fast regime's bounds, so a shape for the set is
// taken only where it keeps the query and the set's longest record inside them.
// The autotuner's choice stands for the shape with the highest rate; it was timed
// on records of like lengths, so a set's few or uneven ones still count.
void pick_shape(ish_ctx *ctx, const Query &q, int *G, int *K, int *layout, const RecordSet *set, double share) {
  const int mode = q.algo == ISH_ALGO_LOCAL ? SW : SG;
  auto it = ctx->tuned.find(tune_key(mode, q.rows, q.Q));
  const bool tuned = !ctx->force_G && !ctx->force_K && ctx->force_layout < 0 && it != ctx->tuned.end();
  if (tuned) {
    *G = it->second.G;
    *K = it->second.K;
    *layout = it->second.layout >= 0 ? it->second.layout : shape_layout(ctx, q, *G, *K);
  } else {
    choose_shape(ctx, q, nullptr, 1, G, K);
    *layout = shape_layout(ctx, q, *G, *K);
  }
  if (!set || !*G) return;
  int g = 0, k = 0;
  choose_shape(ctx, q, set, share, &g, &k);
  const int l = shape_layout(ctx, q, g, k);
  // (closer than that the model does not tell shapes apart, or knows less than the
  // autotuner)
  if (!g || shape_clocks(ctx, q, g, k, l, set, share) >
                (tuned ? 0.9 : 0.97) * shape_clocks(ctx, q, *G, *K, *layout, set, share))
    return;
  const Regime r = regime(q, g * k);
  if (!r.fast || set->max_len > r.max_safe_len || !wave_fits(q, g, k, l)) return;
  *G = g;
  *K = k;
  *layout = l;
}

int build_wave_layout(ish_ctx *ctx, Query &q, int G, int K, int layout, WaveLayout **out) {
  const long key = ((long)G << 20) | ((long)K << 8) | layout;
  auto it = q.layouts.find(key);
  if (it != q.layouts.end()) {
    *out = &it->second;
    return ISH_OK;
  }
  WaveLayout L;
  L.G = G;
  L.K = K;
  L.d = G * K - q.Q;
  L.layout = layout;
  L.kp = layout_stride(layout, K);
  L.slots = profile_slots(layout, q.rows, G, K);
  // profile rows: one per class of codes with equal scores against the
  // query (q.rep), addressed through q.rowmap when the classes merge codes
  const int A = q.rows;
  const bool sg = q.algo == ISH_ALGO_SEMI_GLOBAL;
  const int ppad = (sg && !(q.ends & ISH_FREE_TARGET_START)) ? -(q.open + q.ext) : 0;
  // semi-global scores carry +2 ext: with frames rising by ext per row and per
  // column, H(i-1, j-1) plus P + 2 ext lands in the frame of (i, j)
  const int pext = sg ? 2 * q.ext : 0;
  auto P = [&](int r, int col) -> int {
    if (col < 0) return ppad + pext;
    return q.M[(size_t)q.rep[r] * q.alphabet + q.q[col]] + pext;
  };
  std::vector<uint8_t> host;
  if (layout == PROF_PAIR) {
    std::vector<uint32_t> w((size_t)A * A * L.slots * L.kp, 0u);
    for (int a = 0; a < A; ++a)
      for (int b = 0; b < A; ++b)
        for (int t = 0; t < L.slots; ++t)
          for (int j = 0; j < K; ++j) {
            const int col = (t & (G - 1)) * K + j - L.d;
            w[((size_t)(a * A + b) * L.slots + t) * L.kp + j] =
                sg ? ((uint32_t)P(b, col) << 16) + (uint32_t)P(a, col)
                   : ((uint32_t)P(a, col) & 0xffffu) | ((uint32_t)P(b, col) << 16);
          }
    host.resize(w.size() * 4);
    memcpy(host.data(), w.data(), host.size());
  } else if (layout == PROF_S32) {
    std::vector<uint32_t> w((size_t)A * L.slots * L.kp, 0u);
    for (int a = 0; a < A; ++a)
      for (int t = 0; t < L.slots; ++t)
        for (int j = 0; j < K; ++j) {
          const uint32_t v = (uint32_t)P(a, (t & (G - 1)) * K + j - L.d);
          w[((size_t)a * L.slots + t) * L.kp + j] = sg ? v : v & 0xffffu;
        }
    host.resize(w.size() * 4);
    memcpy(host.data(), w.data(), host.size());
  } else {
    std::vector<int16_t> w((size_t)A * L.slots * L.kp, 0);
    for (int a = 0; a < A; ++a)
      for (int t = 0; t < L.slots; ++t)
        for (int j = 0; j < K; ++j)
          w[((size_t)a * L.slots + t) * L.kp + j] = (int16_t)P(a, (t & (G - 1)) * K + j - L.d);
    host.resize(w.size() * 2);
    memcpy(host.data(), w.data(), host.size());
  }
  L.prof_bytes = (uint32_t)((host.size() + 15) & ~(size_t)15);
  host.resize(L.prof_bytes, 0);
  if (q.rows < q.alphabet) {
    L.remap_off = L.prof_bytes;
    host.insert(host.end(), q.rowmap.begin(), q.rowmap.end());
    L.prof_bytes += 256;
  }
  CU(L.prof.ensure(L.prof_bytes));
  CU(upload(L.prof.p, host.data(), L.prof_bytes));
  auto res = q.layouts.emplace(key, std::move(L));
  *out = &res.first->second;
  return ISH_OK;
}

int build_plain(ish_ctx *ctx, Query &q) {
  if (q.plain_ready) return ISH_OK;
  const int A = q.alphabet;
  std::vector<int16_t> prof((size_t)A * q.Q + 8, 0);
  for (int c = 0; c < A; ++c)
    for (int col = 0; col < q.Q; ++col) prof[(size_t)c * q.Q + col] = q.M[(size_t)c * A + q.q[col]];
  std::vector<int16_t> hin(q.Q + 1, 0);
  if (q.algo == ISH_ALGO_SEMI_GLOBAL && !(q.ends & ISH_FREE_QUERY_START))
    for (int col = 0; col < q.Q; ++col) hin[col] = (int16_t)(-q.open - q.ext * col);
  CU(q.plain_prof.ensure(prof.size() * 2));
  CU(q.plain_hinit.ensure(hin.size() * 2));
  CU(upload(q.plain_prof.p, prof.data(), prof.size() * 2));
  CU(upload(q.plain_hinit.p, hin.data(), hin.size() * 2));
  q.plain_ready = true;
  return ISH_OK;
}

// Byte -> code tables of ish's encodings (convert_ascii_to_encoding,
// ishlib/matcher/alignment/scoring_matrix.mojo:9-27 AA_TO_NUM, 131-149
// NT_TO_NUM): ascii is the identity; actgn / actgn0 map A/a C/c G/g T/t/U/u to
// 0-3 and everything else to 4 (N); blosum62 maps the 23 letters of its
// residue order (either case) to their index and everything else to 23 ('*').
void encoding_table(int kind, uint8_t t[256]) {
  if (kind == ISH_MATRIX_ASCII) {
    for (int i = 0; i < 256; ++i) t[i] = (uint8_t)i;
  } else if (kind == ISH_MATRIX_ACTGN || kind == ISH_MATRIX_ACTGN0) {
    memset(t, 4, 256);
    const char *groups[4] = {"Aa", "Cc", "Gg", "TtUu"};
    for (int code = 0; code < 4; ++code)
      for (const char *c = groups[code]; *c; ++c) t[(uint8_t)*c] = (uint8_t)code;
  } else {
    memset(t, 23, 256);
    const char *order = "ARNDCQEGHILKMFPSTWYVBZX*";
    for (int code = 0; order[code]; ++code) {
      const uint8_t c = (uint8_t)order[code];
      if (c >= 'A' && c <= 'Z') {
        t[c] = (uint8_t)code;
        t[c + 32] = (uint8_t)code;
      }
    }
  }
}

// Device copy of the encoding table of a matrix kind (nullptr: records are
// already encoded).
int device_encoding(ish_ctx *ctx, int kind, const uint8_t **out) {
  if (kind < ISH_MATRIX_ASCII || kind > ISH_MATRIX_BLOSUM62) return fail(ctx, ISH_EINVAL, "unknown matrix kind %d", kind);
  if (!ctx->enc_tables.p) {
    uint8_t t[4 * 256];
    for (int k = 0; k < 4; ++k) encoding_table(k, t + 256 * k);
    CU(ctx->enc_tables.ensure(sizeof t));
    CU(upload(ctx->enc_tables.p, t, sizeof t));
  }
  *out = ctx->enc_tables.as<uint8_t>() + 256 * kind;
  return ISH_OK;
}

// Device phases of the last load for ish_gpu_last_load_ms: upload (with the
// splitting of a text load) and packing.  When the records' bytes travelled on
// the copy stream, the packing kernels that need only the offsets ran during
// the upload, and packing counts from the end of the upload.
void load_phase_times(ish_ctx *ctx) {
  float a = 0.f, b = 0.f;
  cudaEvent_t mid = ctx->raw_overlapped ? ctx->raw_ev : ctx->load_ev[1];
  if (cudaEventElapsedTime(&a, ctx->load_ev[0], mid) == cudaSuccess) ctx->last_load_ms[0] = a;
  if (cudaEventElapsedTime(&b, mid, ctx->load_ev[2]) == cudaSuccess) ctx->last_load_ms[1] = b;
  (void)cudaGetLastError();
  ctx->load_times_due = false;
}

// Lanes per record of k_pack: the power of two nearest above the average
// 16-byte chunks per record, 4 to 32.
static uint32_t pack_group(uint32_t n, uint64_t total) {
  uint32_t gw = 4;
  while (gw < 32 && (uint64_t)gw * 16 * n < total) gw <<= 1;
  return gw;
}
// Its blocks: one group per record, or a block per 64 KB for sets of long records.
static uint32_t pack_blocks(const ish_ctx *ctx, uint32_t n, uint64_t total) {
  return (uint32_t)std::min<uint64_t>(
      std::max<uint64_t>(ceil_div((uint64_t)n * pack_group(n, total), 256), (total >> 16) + 1),
      (uint64_t)ctx->num_sms * 3);
}
static cudaError_t ensure_codes(ish_ctx *ctx, RecordSet &rs, size_t bytes);

// Sort and pack n records held in ctx->raw (raw_bytes bytes): record i is
// raw[off_in[i] .. end[i]) with `end` on the device, or raw[off_in[i] ..
// off_in[i + 1]) without; `enc` (device, may be null) encodes bytes on the way
// (see k_lengths .. k_pack in kernels.cu).  rs.total must hold the residue
// count.  The kernels run on s; with raw_pending the records' bytes are still
// on their way on the copy stream and only k_pack waits for them (raw_ev).
// With defer the host summary is copied into pinned staging and read when the
// set is first used (finish_pending_load).
int pack_set(ish_ctx *ctx, uint32_t n, uint64_t raw_bytes, const uint64_t *end, const uint8_t *enc, RecordSet &rs,
             cudaStream_t s, bool defer, bool raw_pending) {
  if (!s) s = ctx->stream;
  rs.n = n;
  const uint32_t tiles = ceil_div(n, SCAN_TILE);
  if (tiles > SCAN_TILE) return fail(ctx, ISH_EINVAL, "too many records in one set (%u)", n);
  CU(grow(ctx, ctx->len_tmp, (size_t)n * 4));
  CU(grow(ctx, ctx->poff_tmp, (size_t)n * 8));
  CU(grow(ctx, ctx->scan_tmp, (size_t)tiles * 8));
  // counts [NBUCKETS], descending cursors [NBUCKETS], the largest bucket and
  // the pack's long-record counter
  CU(grow(ctx, ctx->hist, (size_t)NBUCKETS * 4 * 2 + 16));
  uint32_t *counts = ctx->hist.as<uint32_t>(), *cursor = counts + NBUCKETS, *max_bucket = cursor + NBUCKETS;
  // what the host reads back: largest code, largest bucket, counts
  CU(grow(ctx, ctx->summary, (size_t)(2 + NBUCKETS) * 4));
  uint32_t *summary = ctx->summary.as<uint32_t>();
  CU(cudaEventRecord(ctx->load_ev[1], s));
  if (ctx->pack_dirty) {  // first load, or the last one stopped before k_scatter cleared the accumulators
    k_zero2<<<64, 1024, 0, s>>>(counts, NBUCKETS, max_bucket, 2);
    ++ctx->launches;
  }
  ctx->pack_dirty = true;
  uint64_t *tile_sum = ctx->scan_tmp.as<uint64_t>();
  k_lengths<<<tiles, 1024, 0, s>>>(ctx->off_in.as<uint64_t>(), end, n, ctx->len_tmp.as<uint32_t>(), tile_sum, counts,
                                   max_bucket, summary);
  ++ctx->launches;
  k_scan_slots<<<tiles, 1024, 0, s>>>(ctx->len_tmp.as<uint32_t>(), n, tile_sum, ctx->poff_tmp.as<uint64_t>());
  ++ctx->launches;
  k_bucket_cursors<<<BUCKET_BLOCKS, 1024, 0, s>>>(counts, max_bucket, cursor, summary);
  ++ctx->launches;
  const uint64_t packed = rs.total + 16ull * n + 16;
  take_spare_set(ctx, rs, packed);
  CU(grow(ctx, rs.len_s, (size_t)n * 4));
  CU(grow(ctx, rs.off_s, (size_t)n * 8));
  CU(grow(ctx, rs.orig_s, (size_t)n * 4));
  k_scatter<<<ceil_div(n, 1024), 1024, 0, s>>>(ctx->len_tmp.as<uint32_t>(), ctx->poff_tmp.as<uint64_t>(), n, cursor,
                                               rs.len_s.as<uint32_t>(), rs.off_s.as<uint64_t>(),
                                               rs.orig_s.as<uint32_t>(), counts, max_bucket, summary);
  ++ctx->launches;
  CU(cudaGetLastError());
  ctx->pack_dirty = false;
  CU(ensure_codes(ctx, rs, packed));
  const uint32_t gw = pack_group(n, rs.total);
  ctx->raw_overlapped = raw_pending;
  if (raw_pending) CU(cudaStreamWaitEvent(s, ctx->raw_ev, 0));  // the records' bytes are on the device
  const uint32_t pb = pack_blocks(ctx, n, rs.total);
  pack_fn(false)<<<pb, 256, 0, s>>>(ctx->raw.as<uint8_t>(), raw_bytes, ctx->off_in.as<uint64_t>(), end,
                            ctx->poff_tmp.as<uint64_t>(), n, rs.len_s.as<uint32_t>(), rs.orig_s.as<uint32_t>(),
                            max_bucket + 1, enc, rs.codes.as<uint8_t>(), summary, gw, 0);
  ++ctx->launches;
  CU(cudaGetLastError());
  CU(cudaEventRecord(ctx->load_ev[2], s));
  if (defer) {
    // the summary the host needs, read back when the set is first used
    CU(cudaMemcpyAsync(ctx->h_summary, summary, (size_t)(2 + NBUCKETS) * 4, cudaMemcpyDeviceToHost, s));
    CU(cudaEventRecord(ctx->load_done, s));
    rs.pending = true;
    return ISH_OK;
  }
  // host copy of the summary: the largest code and bucket and the counts of
  // the buckets of lengths below HIST_HEAD in one round trip, the rest (long
  // records only) after it
  constexpr uint32_t HIST_HEAD = 8192;
  uint32_t *h = ctx->h_summary;
  CU(cudaMemcpyAsync(h, summary, (size_t)(2 + HIST_HEAD) * 4, cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  const uint32_t maxb = std::min<uint32_t>(h[1], NBUCKETS - 1);
  if (maxb >= HIST_HEAD) {
    CU(cudaMemcpyAsync(h + 2 + HIST_HEAD, summary + 2 + HIST_HEAD, (size_t)(maxb + 1 - HIST_HEAD) * 4,
                       cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
  }
  set_summary(rs, h);
  load_phase_times(ctx);
  return ISH_OK;
}

static void set_lengths(RecordSet &rs);

// A set's host-side summary from the device's {largest code, largest bucket,
// counts}; counts above the largest bucket are not read (they are zero).
void set_summary(RecordSet &rs, const uint32_t *h) {
  rs.max_code = h[0];
  const uint32_t maxb = std::min<uint32_t>(h[1], NBUCKETS - 1);
  rs.hist.assign(h + 2, h + 2 + maxb + 1);
  set_lengths(rs);
}

// What follows from the histogram.
static void set_lengths(RecordSet &rs) {
  const uint32_t maxb = top_bucket(rs);
  rs.n_empty = rs.hist[0];
  rs.max_len = maxb < 32768 ? maxb : (uint32_t)(32768 + ((uint64_t)(maxb - 32768) << 5) + 31);
}

// The length bucket of a record, as the device counts it (len_bucket).
static uint32_t length_bucket(uint64_t len) {
  if (len < 32768) return (uint32_t)len;
  return (uint32_t)std::min<uint64_t>(32768 + ((len - 32768) >> 5), NBUCKETS - 1);
}

// Allocates the codes of a set, giving the cached buffers of freed sets back too
// when memory is short.
static cudaError_t ensure_codes(ish_ctx *ctx, RecordSet &rs, size_t bytes) {
  cudaError_t e = grow(ctx, rs.codes, bytes);
  if (e == cudaErrorMemoryAllocation && !ctx->spare_sets.empty()) {
    (void)cudaGetLastError();
    for (RecordSet &sp : ctx->spare_sets) release_set(sp);
    ctx->spare_sets.clear();
    e = rs.codes.ensure(bytes);
  }
  return e;
}

// Upload and pack a set of at most SORT_SMALL records: two kernels, and the
// histogram from the caller's offsets (which have to ascend: their differences
// index it), so that of the set's summary only the largest code comes from the
// device.  With `limit` (the alphabet of the query
// that is scored next) the call does not wait for it: codes outside the alphabet
// are stored as 0, and the caller reads the largest code, at ctx->summary, with
// its results.
static int load_small(ish_ctx *ctx, const uint8_t *records, const uint64_t *offsets, uint32_t n, RecordSet &rs,
                      const uint8_t *enc, cudaStream_t s, bool defer, uint32_t limit) {
  const uint64_t base = offsets[0], bytes = offsets[n] - base;
  uint32_t top = 0;
  for (uint32_t i = 0; i < n; ++i) {
    if (offsets[i + 1] < offsets[i]) return fail(ctx, ISH_EINVAL, "offsets are not monotone");
    top = std::max(top, length_bucket(offsets[i + 1] - offsets[i]));
  }
  rs.hist.assign(top + 1, 0);
  for (uint32_t i = 0; i < n; ++i) ++rs.hist[length_bucket(offsets[i + 1] - offsets[i])];
  set_lengths(rs);
  rs.n = n;
  rs.max_code = 0;
  const uint64_t packed = bytes + 16ull * n + 16;
  take_spare_set(ctx, rs, packed);
  CU(grow(ctx, ctx->raw, bytes + 32));
  CU(grow(ctx, ctx->off_in, (size_t)(n + 1) * 8));
  CU(grow(ctx, ctx->poff_tmp, (size_t)n * 8));
  CU(grow(ctx, ctx->hist, (size_t)NBUCKETS * 4 * 2 + 16));
  CU(grow(ctx, ctx->summary, (size_t)(2 + NBUCKETS) * 4));
  CU(grow(ctx, rs.len_s, (size_t)n * 4));
  CU(grow(ctx, rs.off_s, (size_t)n * 8));
  CU(grow(ctx, rs.orig_s, (size_t)n * 4));
  CU(ensure_codes(ctx, rs, packed));
  uint32_t *long_counter = ctx->hist.as<uint32_t>() + 2 * NBUCKETS + 1, *max_code = ctx->summary.as<uint32_t>();
  CU(cudaEventRecord(ctx->load_ev[0], s));
  CU(cudaMemcpyAsync(ctx->off_in.p, offsets, (size_t)(n + 1) * 8, cudaMemcpyHostToDevice, s));
  if (bytes) CU(cudaMemcpyAsync(ctx->raw.p, records + base, bytes, cudaMemcpyHostToDevice, s));
  ctx->raw_overlapped = false;
  CU(cudaEventRecord(ctx->load_ev[1], s));
  uint32_t threads = 32;
  while (threads * 4 < n) threads *= 2;
  k_sort_small<<<1, threads, 0, s>>>(ctx->off_in.as<uint64_t>(), n, base, ctx->poff_tmp.as<uint64_t>(),
                                     rs.len_s.as<uint32_t>(), rs.off_s.as<uint64_t>(), rs.orig_s.as<uint32_t>(),
                                     long_counter, max_code);
  ++ctx->launches;
  pack_fn(limit != 0)<<<pack_blocks(ctx, n, bytes), 256, 0, s>>>(
      ctx->raw.as<uint8_t>(), bytes, ctx->off_in.as<uint64_t>(), nullptr, ctx->poff_tmp.as<uint64_t>(), n,
      rs.len_s.as<uint32_t>(), rs.orig_s.as<uint32_t>(), long_counter, enc, rs.codes.as<uint8_t>(), max_code,
      pack_group(n, bytes), limit);
  ++ctx->launches;
  CU(cudaGetLastError());
  CU(cudaEventRecord(ctx->load_ev[2], s));
  ctx->load_times_due = true;
  if (limit) return ISH_OK;
  CU(cudaMemcpyAsync(ctx->h_summary, max_code, 4, cudaMemcpyDeviceToHost, s));
  if (defer) {
    CU(cudaEventRecord(ctx->load_done, s));
    rs.pending = true;
    return ISH_OK;
  }
  CU(cudaStreamSynchronize(s));
  rs.max_code = ctx->h_summary[0];
  return ISH_OK;
}

// Upload and pack a record set given as concatenated records + n+1 offsets.
// limit: see load_small (0: wait for the set's summary).
int load_records(ish_ctx *ctx, const uint8_t *records, const uint64_t *offsets, uint32_t n, RecordSet &rs,
                 const uint8_t *enc, cudaStream_t stream, bool defer, uint32_t limit) {
  if (n == 0) {
    rs.n = 0;
    rs.total = 0;
    return ISH_OK;
  }
  if (!offsets) return fail(ctx, ISH_EINVAL, "offsets is NULL");
  const uint64_t base = offsets[0], end = offsets[n];
  if (end < base) return fail(ctx, ISH_EINVAL, "offsets are not monotone");
  const uint64_t bytes = end - base;
  if (bytes && !records) return fail(ctx, ISH_EINVAL, "records is NULL");
  rs.total = bytes;
  cudaStream_t s = stream ? stream : ctx->stream;
  if (n <= SORT_SMALL) {
    const int rc = load_small(ctx, records, offsets, n, rs, enc, s, defer, limit);
    if (rc) cudaStreamSynchronize(s);  // the caller's buffers are free again on return
    return rc;
  }
  // The offsets go first on s; the records' bytes (+16 slack for the
  // realigning pack loads) follow on the copy stream once the offsets are in
  // (everything before this load on s, which includes the previous pack's
  // reads of the same buffer, is before that point too), while s computes
  // lengths, packed offsets and sorted positions.
  CU(grow(ctx, ctx->raw, bytes + 32));
  CU(grow(ctx, ctx->off_in, (size_t)(n + 1) * 8));
  CU(cudaEventRecord(ctx->load_ev[0], s));
  std::vector<uint64_t> rebased;
  if (base) {
    rebased.assign(offsets, offsets + n + 1);
    for (auto &v : rebased) v -= base;
  }
  CU(cudaMemcpyAsync(ctx->off_in.p, base ? rebased.data() : offsets, (size_t)(n + 1) * 8, cudaMemcpyHostToDevice, s));
  CU(cudaEventRecord(ctx->off_ev, s));
  {
    cudaStream_t c = ctx->copy_stream;
    cudaError_t oe = cudaStreamWaitEvent(c, ctx->off_ev, 0);
    if (oe == cudaSuccess && bytes) oe = cudaMemcpyAsync(ctx->raw.p, records + base, bytes, cudaMemcpyHostToDevice, c);
    if (oe == cudaSuccess) oe = cudaEventRecord(ctx->raw_ev, c);
    if (oe != cudaSuccess) {
      cudaStreamSynchronize(c);  // the caller's buffers are free again on return
      cudaStreamSynchronize(s);
      CU(oe);
    }
  }
  if (base) CU(cudaEventSynchronize(ctx->off_ev));  // the rebased offsets are a temporary
  const int rc = pack_set(ctx, n, bytes, nullptr, enc, rs, s, defer, bytes != 0);
  if (rc) {
    cudaStreamSynchronize(ctx->copy_stream);
    cudaStreamSynchronize(s);
  }
  return rc;
}

// Completes the asynchronous load in flight: waits for its stream's work and
// fills the set's host-side summary from the pinned staging copy.
int finish_pending_load(ish_ctx *ctx) {
  if (!ctx->pending_set) return ISH_OK;
  const int32_t id = ctx->pending_set;
  ctx->pending_set = 0;
  auto it = ctx->sets.find(id);
  const cudaError_t e = cudaEventSynchronize(ctx->load_done);
  if (it == ctx->sets.end()) return ISH_OK;
  RecordSet &rs = it->second;
  rs.pending = false;
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    release_set(rs);
    ctx->sets.erase(it);
    return fail(ctx, ISH_EDEVICE, "asynchronous load of record set %d failed: %s (the set is gone)", id,
                cudaGetErrorString(e));
  }
  if (rs.hist.empty()) set_summary(rs, ctx->h_summary);
  else rs.max_code = ctx->h_summary[0];  // (load_small has counted the lengths)
  load_phase_times(ctx);
  return ISH_OK;
}

RecordSet *use_set(ish_ctx *ctx, int32_t set_id, int *rc) {
  auto it = ctx->sets.find(set_id);
  if (it == ctx->sets.end()) {
    *rc = fail(ctx, ISH_EINVAL, "unknown record set %d", set_id);
    return nullptr;
  }
  if (it->second.pending) {
    *rc = finish_pending_load(ctx);
    if (*rc) return nullptr;
  }
  *rc = ISH_OK;
  return &it->second;
}

// Upload a text buffer, split it into lines on the device and pack the lines
// as records (see k_count_newlines .. k_line_bounds in kernels.cu).
int load_lines(ish_ctx *ctx, const uint8_t *text, uint64_t bytes, RecordSet &rs, const uint8_t *enc, uint32_t *n_out) {
  *n_out = 0;
  rs.n = 0;
  rs.total = 0;
  if (bytes == 0) return ISH_OK;
  if (!text) return fail(ctx, ISH_EINVAL, "text is NULL");
  cudaStream_t s = ctx->stream;
  CU(grow(ctx, ctx->raw, bytes + 32));
  CU(cudaEventRecord(ctx->load_ev[0], s));
  CU(cudaMemcpyAsync(ctx->raw.p, text, bytes, cudaMemcpyHostToDevice, s));
  const uint64_t tiles64 = (bytes + LINE_TILE - 1) / LINE_TILE;
  if (tiles64 > 0x7fffffffull) return fail(ctx, ISH_EINVAL, "text too large");
  const uint32_t tiles = (uint32_t)tiles64;
  CU(grow(ctx, ctx->block_counts, (size_t)tiles * 4 + 8));
  CU(grow(ctx, ctx->nhits, 16));
  k_count_newlines<<<tiles, 1024, 0, s>>>(ctx->raw.as<uint8_t>(), bytes, ctx->block_counts.as<uint32_t>());
  ++ctx->launches;
  k_scan_counts<<<1, 1024, 0, s>>>(ctx->block_counts.as<uint32_t>(), tiles, ctx->nhits.as<uint32_t>());
  ++ctx->launches;
  uint32_t *hs = reinterpret_cast<uint32_t *>(ctx->h_small);
  CU(cudaMemcpyAsync(hs, ctx->nhits.p, 4, cudaMemcpyDeviceToHost, s));
  CU(cudaStreamSynchronize(s));
  const uint32_t n_nl = hs[0];
  const uint8_t last = text[bytes - 1];
  const uint64_t lines = (uint64_t)n_nl + (last != '\n' ? 1 : 0);
  if (lines >= 0xffffffffull) return fail(ctx, ISH_EINVAL, "too many lines (%llu)", (unsigned long long)lines);
  const uint32_t n = (uint32_t)lines;
  CU(grow(ctx, ctx->nl_pos, (size_t)n_nl * 8 + 8));
  CU(grow(ctx, ctx->off_in, (size_t)(n + 1) * 8));
  CU(grow(ctx, ctx->line_end, (size_t)n * 8 + 8));
  write_newlines_fn(false)<<<tiles, 1024, 0, s>>>(ctx->raw.as<uint8_t>(), bytes, ctx->block_counts.as<uint32_t>(),
                                                  ctx->nl_pos.as<uint64_t>(), nullptr);
  ++ctx->launches;
  CU(cudaMemsetAsync(ctx->nhits.p, 0, 16, s));
  k_line_bounds<<<std::max<uint32_t>(1, std::min<uint32_t>(ceil_div(n, 256), (uint32_t)ctx->num_sms * 16)), 256, 0,
                  s>>>(ctx->raw.as<uint8_t>(), bytes, ctx->nl_pos.as<uint64_t>(), n_nl, n, ctx->off_in.as<uint64_t>(),
                       ctx->line_end.as<uint64_t>(), reinterpret_cast<unsigned long long *>(ctx->nhits.p));
  ++ctx->launches;
  CU(cudaGetLastError());
  // residues: the text minus the newlines and the dropped carriage returns;
  // the exact count comes back with the set's summary, packing only needs a
  // bound
  CU(cudaMemcpyAsync(ctx->h_small, ctx->nhits.p, 8, cudaMemcpyDeviceToHost, s));
  rs.total = bytes - n_nl;
  *n_out = n;
  const int rc = pack_set(ctx, n, bytes, ctx->line_end.as<uint64_t>(), enc, rs);
  if (!rc) rs.total = ctx->h_small[0];
  return rc;
}

// Number of records (a prefix of the descending order) whose length bucket
// may exceed `len`.
uint32_t count_longer(const RecordSet &rs, uint64_t len) {
  uint64_t cnt = 0;
  for (uint32_t b = top_bucket(rs); b > 0; --b) {
    const uint64_t lo = b < 32768 ? b : 32768 + ((uint64_t)(b - 32768) << 5);
    const uint64_t hi = b < 32768 ? b : lo + 31;
    if (hi <= len) break;
    (void)lo;
    cnt += rs.hist[b];
  }
  return (uint32_t)cnt;
}

int ensure_outputs(ish_ctx *ctx, uint32_t n) {
  CU(grow(ctx, ctx->out_score, (size_t)n * 4 + 4));
  CU(grow(ctx, ctx->out_qend, (size_t)n * 4 + 4));
  CU(grow(ctx, ctx->out_tend, (size_t)n * 4 + 4));
  CU(grow(ctx, ctx->out_hit, (size_t)n + 16));
  CU(grow(ctx, ctx->counter, 64));
  CU(grow(ctx, ctx->error, 64));
  return ISH_OK;
}

void wave_params(const Query &q, const WaveLayout &L, const RecordSet &rs, OutDev out, int *error, WaveParams *pp) {
  WaveParams &p = *pp;
  p = WaveParams{};
  const int mode = q.algo == ISH_ALGO_LOCAL ? SW : SG;
  p.prof = L.prof.as<const uint4>();
  p.prof_bytes = L.prof_bytes;
  p.Q = q.Q;
  p.G = L.G;
  p.K = L.K;
  p.d = L.d;
  p.kp = L.kp;
  p.alphabet = q.rows;
  p.remap_off = L.remap_off;
  p.layout = L.layout;
  p.lane_mul = 65536u;
  p.open = q.open;
  p.ext = q.ext;
  p.ends = q.ends;
  p.neg_limit = q.neg_limit;
  const bool sg = mode == SG;
  // Semi-global values are unsigned 16-bit: value + bias + row frame + column
  // frame.  With a free target start H(i, j) >= -open - ext * j (a query gap
  // from the left boundary), so with its column frame no H is below
  // bias - open and no E or gap opening below bias - 2 open; a fixed one lowers
  // the left boundary by open + ext per row.  `low` is that depth; the slack
  // above it covers a score (an int8) added to the smallest value, the rows a
  // pair is rounded up by and the floor that stands for minus infinity on the
  // left (ext after its profile step).  At the top: H <= 30000, row frames
  // < 2048 and column frames ext * G * K, where the regime keeps
  // low + ext * (G * K + 3) <= 30000; the sum stays below 65,536.
  const bool ts = q.ends & ISH_FREE_TARGET_START;
  const int low = ts ? 2 * q.open : 3 * q.open + q.ext * (int)std::min<uint64_t>(rs.max_len, 32768);
  // (local alignment: H >= 0, E, F and openings >= -open, H <= 30000)
  p.bias = sg ? low + 8 * q.ext + 256 : q.open + 256;
  p.frame_mask = sg ? frame_rows(q.ext) - 1 : 0x3fffffff;
  p.pk_next = dup16_host(-q.ext);
  p.pk_eopen = dup16_host(q.ext - q.open);
  p.pk_left = sg ? (ts ? (uint32_t)p.bias : (uint32_t)q.open) * 0x10001u : 0u;
  p.pk_left_ext = sg && ts ? (uint32_t)q.ext * 0x10001u : 0u;
  p.pk_drop = sg ? (uint32_t)(-(p.frame_mask + 1) * q.ext) * 0x10001u : 0u;
  p.slots = L.slots;
  p.row_bytes = (uint32_t)(L.slots * L.kp * (L.layout == PROF_S16 ? 2 : 4));
  p.error = error;
  p.rec = RecordsDev{rs.codes.as<const uint8_t>(), rs.off_s.as<const uint64_t>(), rs.len_s.as<const uint32_t>(),
                     rs.orig_s.as<const uint32_t>(), rs.n};
  p.out = out;
  p.dec = Decision{q.max_score, q.thr};
}

// Sets a kernel's dynamic shared memory limit, once per kernel and context.
static cudaError_t allow_smem(ish_ctx *ctx, const void *fn) {
  std::lock_guard<std::mutex> lk(ctx->smem_mu);
  if (ctx->smem_allowed.count(fn)) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WAVE_SMEM_MAX);
  if (e == cudaSuccess) ctx->smem_allowed.insert(fn);
  return e;
}

int launch_wave_range(ish_ctx *ctx, Query &q, RecordSet &rs, uint32_t first, uint32_t count, OutDev out, int G, int K,
                      int layout, cudaStream_t s) {
  if (count == 0) return ISH_OK;
  if (!G || G * K < q.Q + 1) return fail(ctx, ISH_EOVERFLOW, "no wavefront shape for a query of %d residues", q.Q);
  WaveLayout *L = nullptr;
  int rc = build_wave_layout(ctx, q, G, K, layout, &L);
  if (rc) return rc;
  const int mode = q.algo == ISH_ALGO_LOCAL ? SW : SG;
  const int lean = lean_for(ctx, q, G, K, L->layout, &rs, 1);
  WaveFn fn = wave_fn(K, mode, L->layout, lean);
  if (!fn) return fail(ctx, ISH_EOVERFLOW, "no wavefront kernel for K=%d", K);
  {
    const cudaError_t e = allow_smem(ctx, (const void *)fn);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      cudaFuncAttributes a{};
      const cudaError_t ea = cudaFuncGetAttributes(&a, (const void *)fn);
      (void)cudaGetLastError();
      return fail(ctx, ISH_EDEVICE,
                  "wavefront kernel K=%d mode=%d layout=%d: dynamic shared memory %zu bytes refused (%s); kernel "
                  "attributes (%s): static %zu, max dynamic %d, %d registers",
                  K, mode, L->layout, WAVE_SMEM_MAX, cudaGetErrorString(e), cudaGetErrorString(ea), a.sharedSizeBytes,
                  a.maxDynamicSharedSizeBytes, a.numRegs);
    }
  }
  // One block per SM with as many warps as the SM holds, or as the range's
  // record pairs need when spread over all SMs.
  const size_t prof_area = (L->prof_bytes + 15) & ~15u;
  int most = wave_fit_threads(prof_area, K, mode, lean);
  if (most < 32) return fail(ctx, ISH_EOVERFLOW, "wavefront kernel K=%d does not fit (profile %zu)", K, prof_area);
  if (ctx->force_blocks) most = std::min(most, ctx->force_blocks * (K <= 32 ? 256 : 128));
  const uint32_t pairs = (count + 1) / 2;
  const uint32_t warps = ceil_div((uint64_t)pairs * G, 32);
  const int threads = (int)std::min<uint32_t>(most, 32 * ceil_div(warps, ctx->num_sms));
  const uint32_t grid = std::min<uint32_t>(ctx->num_sms, ceil_div(warps, threads / 32));
  const size_t smem = wave_smem(prof_area, threads, K, mode);
  CU(ctx->counter.ensure(64));
  WaveParams p;
  wave_params(q, *L, rs, out, ctx->error.as<int>(), &p);
  p.first = first;
  p.count = count;
  p.dealt = grid * (uint32_t)threads / (uint32_t)G;
  p.counter = ctx->counter.as<uint32_t>();
  p.max_steps = ctx->step_budget ? ctx->step_budget : rs.total + 2ull * count + 1024;
  CU(cudaMemsetAsync(ctx->counter.p, 0, 4, s));
  fn<<<grid, threads, smem, s>>>(p);
  ++ctx->launches;
  CU(cudaGetLastError());
  return ISH_OK;
}

// Blocks of a persistent batched launch: the size among 128 and 256 threads and
// all of an SM's that keeps most threads resident, the smaller one where equal
// (a block waits for its slowest pair at every query switch; small blocks of an
// SM switch at different times).
int batch_launch(ish_ctx *ctx, BatchFn fn, int K, int mode, int lean, size_t prof_area, BatchLaunch *out) {
  CU(allow_smem(ctx, (const void *)fn));
  const int all = wave_sm_threads(K, lean);
  int best = 0;
  for (int t : {128, 256, wave_fit_threads(prof_area, K, mode, lean)}) {
    if (t < 32 || t > all) continue;
    const size_t smem = wave_smem(prof_area, t, K, mode);
    if (smem > WAVE_SMEM_MAX) continue;
    int per_sm = std::min<int>(all / t, (int)((228 * 1024) / (smem + 2048)));
    if (ctx->force_blocks) per_sm = std::min(per_sm, ctx->force_blocks);
    if (per_sm * t > best) {
      best = per_sm * t;
      *out = BatchLaunch{t, (uint32_t)(std::max(per_sm, 1) * ctx->num_sms), smem};
    }
  }
  return best ? ISH_OK : fail(ctx, ISH_EOVERFLOW, "batch kernel K=%d does not fit (profile %zu)", K, prof_area);
}

int launch_plain(ish_ctx *ctx, Query &q, RecordSet &rs, uint32_t first, uint32_t count, OutDev out) {
  if (count == 0) return ISH_OK;
  int rc = build_plain(ctx, q);
  if (rc) return rc;
  // the int16 form (the reference kernel's per-thread arrays and launch shape)
  // when asked for and the query fits its largest array; else int32 columns
  int qmax = 0;
  if (ctx->kernel == ISH_KERNEL_PLAIN16 && q.Q <= PLAIN16_QMAX)
    for (qmax = 64; qmax < q.Q; qmax <<= 1) {
    }
  const int threads = qmax ? 32 : 128;
  const uint32_t blocks =
      qmax ? ceil_div(PLAIN16_THREADS, threads)
           : std::max<uint32_t>(1, std::min<uint32_t>(ceil_div(count, threads), (uint32_t)ctx->num_sms * 4));
  const uint32_t nth = qmax ? PLAIN16_THREADS : blocks * threads;
  if (!qmax) CU(ctx->plain_scratch.ensure((size_t)2 * q.Q * nth * 4 + 16));
  PlainParams p{};
  p.prof = q.plain_prof.as<const int16_t>();
  p.prof_bytes = (uint32_t)(((size_t)q.alphabet * q.Q * 2 + 15) & ~(size_t)15);
  p.use_smem = p.prof_bytes <= 96 * 1024;
  p.Q = q.Q;
  p.alphabet = q.alphabet;
  p.open = q.open;
  p.ext = q.ext;
  p.ends = q.ends;
  p.neg_limit = q.neg_limit;
  p.hinit = q.plain_hinit.as<const int16_t>();
  p.scratch = ctx->plain_scratch.as<int32_t>();
  p.nthreads = nth;
  p.first = first;
  p.count = count;
  p.error = ctx->error.as<int>();
  p.rec = RecordsDev{rs.codes.as<const uint8_t>(), rs.off_s.as<const uint64_t>(), rs.len_s.as<const uint32_t>(),
                     rs.orig_s.as<const uint32_t>(), rs.n};
  p.out = out;
  p.dec = Decision{q.max_score, q.thr};
  const size_t smem = p.use_smem ? p.prof_bytes : 0;
  PlainFn fn = plain_fn(q.algo == ISH_ALGO_LOCAL ? SW : SG, qmax);
  CU(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max<size_t>(smem, 1)));
  fn<<<blocks, threads, smem, ctx->stream>>>(p);
  ++ctx->launches;
  CU(cudaGetLastError());
  return ISH_OK;
}

int fast_check(const Query &q, const RecordSet &rs, int G, int K, char *msg, size_t len) {
  Regime r = regime(q, G ? G * K : q.Q + 64);
  if (!r.fast) {
    snprintf(msg, len,
             "parameters outside the exact-integer fast regime (gap_open must exceed gap_extend and scores must stay "
             "within int16)");
    return ISH_EINVAL;
  }
  const uint32_t nonempty = rs.n - rs.n_empty;
  const uint32_t n_long = r.max_safe_len == ~0ull ? 0 : std::min(count_longer(rs, r.max_safe_len), nonempty);
  if (n_long) {
    snprintf(msg, len, "%u records are longer than %llu residues with a non-free target start", n_long,
             (unsigned long long)r.max_safe_len);
    return ISH_EINVAL;
  }
  if (rs.max_code >= (uint32_t)q.alphabet) {
    snprintf(msg, len, "a record contains code %u >= the alphabet size %d of the query", rs.max_code, q.alphabet);
    return ISH_EINVAL;
  }
  if (!G || G * K < q.Q + 1) {
    snprintf(msg, len, "no wavefront shape for a query of %d residues", q.Q);
    return ISH_EOVERFLOW;
  }
  return ISH_OK;
}

bool fast_regime(ish_ctx *ctx, const Query &q, const RecordSet &rs) {
  int G, K, layout;
  pick_shape(ctx, q, &G, &K, &layout, &rs);
  char msg[256];
  return fast_check(q, rs, G, K, msg, sizeof msg) == ISH_OK;
}

// Whether the wavefront kernel's shared memory (profile, code -> row table,
// slots, saved rows) fits in a block for this shape and layout.
bool wave_fits(const Query &q, int G, int K, int layout) {
  if (!G) return false;
  const int mode = q.algo == ISH_ALGO_LOCAL ? SW : SG;
  size_t prof = (layout_bytes(layout, q.rows, G, K) + 15) & ~(size_t)15;
  if (q.rows < q.alphabet) prof += 256;
  return wave_smem(prof, 128, K, mode) <= WAVE_SMEM_MAX;
}

// The wavefront kernel, or the plain kernel when the wavefront profile does
// not fit in shared memory (long queries over large alphabets) or the plain
// kernel was asked for.
int launch_range(ish_ctx *ctx, Query &q, RecordSet &rs, uint32_t first, uint32_t count, OutDev out, cudaStream_t s) {
  int G, K, layout;
  pick_shape(ctx, q, &G, &K, &layout, &rs);
  if (ctx->kernel == ISH_KERNEL_PLAIN || ctx->kernel == ISH_KERNEL_PLAIN16 || !wave_fits(q, G, K, layout)) {
    if (s != ctx->stream) return fail(ctx, ISH_EINVAL, "the plain kernel runs on the context stream only");
    return launch_plain(ctx, q, rs, first, count, out);
  }
  return launch_wave_range(ctx, q, rs, first, count, out, G, K, layout, s);
}

// Score query q against set rs into the context's device output buffers.
int run_scoring(ish_ctx *ctx, Query &q, RecordSet &rs) {
  const uint32_t n = rs.n;
  int rc = ensure_outputs(ctx, n);
  if (rc) return rc;
  cudaStream_t s = ctx->stream;
  CU(cudaMemsetAsync(ctx->error.p, 0, 4, s));
  OutDev out{ctx->out_score.as<int32_t>(), ctx->out_qend.as<int32_t>(), ctx->out_tend.as<int32_t>(),
             ctx->out_hit.as<uint8_t>()};
  const int mode = q.algo == ISH_ALGO_LOCAL ? SW : SG;
  const uint32_t n_empty = (q.Q == 0) ? n : rs.n_empty;
  const uint32_t nonempty = n - n_empty;
  CU(cudaEventRecord(ctx->ev0, s));
  if (n_empty) {
    k_trivial<<<std::max<uint32_t>(1, std::min<uint32_t>(ceil_div(n_empty, 256), 1024)), 256, 0, s>>>(
        RecordsDev{rs.codes.as<const uint8_t>(), rs.off_s.as<const uint64_t>(), rs.len_s.as<const uint32_t>(),
                   rs.orig_s.as<const uint32_t>(), rs.n},
        nonempty, n_empty, mode, q.Q, out, Decision{q.max_score, q.thr});
    ++ctx->launches;
    CU(cudaGetLastError());
  }
  if (nonempty) {
    if (rs.max_code >= (uint32_t)q.alphabet)
      return fail(ctx, ISH_EINVAL, "a record contains code %u >= the alphabet size %d of the query", rs.max_code,
                  q.alphabet);
    if (ctx->kernel == ISH_KERNEL_EXACT || !fast_regime(ctx, q, rs)) {
      rc = launch_exact(ctx, q, rs, 0, nonempty, out, s);
    } else {
      bool windowed = false;
      ctx->last_windows = 0;
      rc = launch_windows(ctx, q, rs, nonempty, out, s, &windowed);
      if (!rc && !windowed) rc = launch_range(ctx, q, rs, 0, nonempty, out, s);
    }
    if (rc) return rc;
  }
  return ISH_OK;
}

// max_code: the set's largest code where the host has not seen it yet (load_small
// with a limit), checked against the query's alphabet before any output is
// written: such a call's results are staged whether it wants the hits or not.
// NULL else.
int fetch_outputs(ish_ctx *ctx, uint32_t n, int32_t *score, int32_t *qend, int32_t *tend, uint8_t *hit,
                  uint32_t *hit_idx, uint32_t *n_hits, const uint32_t *max_code = nullptr, int alphabet = 0) {
  cudaStream_t s = ctx->stream;
  const bool compact = (hit_idx || n_hits || max_code) && n, staged = compact && n <= SORT_SMALL;
  CU(grow(ctx, ctx->nhits, 16));
  uint32_t *out3 = ctx->nhits.as<uint32_t>();  // hits, error flags, largest code
  if (compact) {
    const uint32_t nb = ceil_div(n, HIT_TILE);
    CU(grow(ctx, ctx->hit_idx, (size_t)n * 4 + 4));
    const uint8_t *flags = ctx->out_hit.as<uint8_t>();
    if (n <= COMPACT_ONE) {
      StageOut stage;
      if (staged) {
        stage.to = ctx->h_stage;
        stage.hit = hit != nullptr;
        if (score) stage.from[0] = ctx->out_score.as<int32_t>();
        if (qend) stage.from[1] = ctx->out_qend.as<int32_t>();
        if (tend) stage.from[2] = ctx->out_tend.as<int32_t>();
      }
      k_compact_one<<<1, 1024, 0, s>>>(flags, n, ctx->hit_idx.as<uint32_t>(), ctx->error.as<int>(), max_code, out3,
                                       stage);
      ++ctx->launches;
    } else {
      CU(grow(ctx, ctx->block_counts, (size_t)nb * 4 + 8));
      uint32_t *counts = ctx->block_counts.as<uint32_t>();
      k_count_hits<<<nb, 1024, 0, s>>>(flags, n, counts);
      ++ctx->launches;
      if (nb <= 1024) {
        k_write_hits_sum<<<nb, 1024, 0, s>>>(flags, n, counts, ctx->hit_idx.as<uint32_t>(), ctx->error.as<int>(), out3);
      } else {
        k_scan_counts<<<1, 1024, 0, s>>>(counts, nb, out3);
        ++ctx->launches;
        k_write_hits<<<nb, 1024, 0, s>>>(flags, n, counts, ctx->hit_idx.as<uint32_t>());
      }
      ++ctx->launches;
    }
    CU(cudaGetLastError());
  }
  CU(cudaEventRecord(ctx->ev1, s));
  // Results of a small call were written to pinned memory by the compaction;
  // those of a larger one are copied: hit count and error flags go into pinned
  // staging too, so that every copy stays asynchronous until the one
  // synchronisation, and the first hit indices travel with the count (hit_idx
  // holds n entries, so the prefix fits whatever the count).
  uint32_t *hs = staged ? ctx->h_stage : reinterpret_cast<uint32_t *>(ctx->h_small);
  constexpr uint32_t HIT_PREFIX = 4096;
  const uint32_t prefix = std::min<uint32_t>(n, HIT_PREFIX);
  if (!staged) {
    if (n && score) CU(cudaMemcpyAsync(score, ctx->out_score.p, (size_t)n * 4, cudaMemcpyDeviceToHost, s));
    if (n && qend) CU(cudaMemcpyAsync(qend, ctx->out_qend.p, (size_t)n * 4, cudaMemcpyDeviceToHost, s));
    if (n && tend) CU(cudaMemcpyAsync(tend, ctx->out_tend.p, (size_t)n * 4, cudaMemcpyDeviceToHost, s));
    if (n && hit) CU(cudaMemcpyAsync(hit, ctx->out_hit.p, (size_t)n, cudaMemcpyDeviceToHost, s));
    hs[0] = hs[1] = hs[2] = 0;
    if (compact) CU(cudaMemcpyAsync(hs, out3, 12, cudaMemcpyDeviceToHost, s));
    if (!compact || ceil_div(n, HIT_TILE) > 1024)
      CU(cudaMemcpyAsync(hs + 1, ctx->error.p, 4, cudaMemcpyDeviceToHost, s));
    if (hit_idx && compact) CU(cudaMemcpyAsync(hit_idx, ctx->hit_idx.p, (size_t)prefix * 4, cudaMemcpyDeviceToHost, s));
  }
  CU(cudaStreamSynchronize(s));
  const int herr = (int)hs[1];
  const uint32_t total = hs[0];
  if (max_code && hs[2] >= (uint32_t)alphabet)
    return fail(ctx, ISH_EINVAL, "a record contains code %u >= the alphabet size %d of the query", hs[2], alphabet);
  if (staged) {
    const uint32_t *v = hs + STAGE_HEAD;
    if (score) memcpy(score, v, (size_t)n * 4);
    if (qend) memcpy(qend, v + SORT_SMALL, (size_t)n * 4);
    if (tend) memcpy(tend, v + 2 * SORT_SMALL, (size_t)n * 4);
    if (hit_idx) memcpy(hit_idx, v + 3 * SORT_SMALL, (size_t)total * 4);
    if (hit) memcpy(hit, v + 4 * SORT_SMALL, n);
  } else if (hit_idx && total > prefix) {
    CU(cudaMemcpyAsync(hit_idx + prefix, ctx->hit_idx.as<uint32_t>() + prefix, (size_t)(total - prefix) * 4,
                       cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
  }
  if (n_hits) *n_hits = total;
  float ms = 0.f;
  if (cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1) == cudaSuccess) ctx->last_ms = ms;
  if (herr & 2) return fail(ctx, ISH_ETIMEDOUT, "wavefront kernel exceeded its step budget (internal error)");
  if (herr) return fail(ctx, ISH_EINVAL, "a record contains a code >= the alphabet size of the query");
  return ISH_OK;
}

}  // namespace host
}  // namespace ish

extern "C" {

int ish_gpu_abi_version(void) { return ISH_GPU_ABI_VERSION; }

int ish_gpu_open(int device, ish_ctx **out) {
  if (!out) return fail(nullptr, ISH_EINVAL, "out is NULL");
  *out = nullptr;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0)
    return fail(nullptr, ISH_ENODEV, "no CUDA device: %s", e == cudaSuccess ? "count is 0" : cudaGetErrorString(e));
  if (device < 0 || device >= ndev) return fail(nullptr, ISH_EINVAL, "device %d out of range (%d devices)", device, ndev);
  ish_ctx *ctx = new ish_ctx();
  ctx->device = device;
  auto bail = [&](cudaError_t err, const char *what) {
    g_open_error = std::string(what) + ": " + cudaGetErrorString(err);
    delete ctx;
    return ISH_EDEVICE;
  };
  if ((e = cudaSetDevice(device)) != cudaSuccess) return bail(e, "cudaSetDevice");
  if ((e = cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess)
    return bail(e, "cudaDeviceGetAttribute");
  {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) ctx->mem_total = total_b;
    (void)cudaGetLastError();
  }
  if ((e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking)) != cudaSuccess)
    return bail(e, "cudaStreamCreate");
  if ((e = cudaEventCreate(&ctx->ev0)) != cudaSuccess) return bail(e, "cudaEventCreate");
  if ((e = cudaEventCreate(&ctx->ev1)) != cudaSuccess) return bail(e, "cudaEventCreate");
  for (cudaEvent_t &ev : ctx->load_ev)
    if ((e = cudaEventCreate(&ev)) != cudaSuccess) return bail(e, "cudaEventCreate");
  if ((e = cudaStreamCreateWithFlags(&ctx->load_stream, cudaStreamNonBlocking)) != cudaSuccess)
    return bail(e, "cudaStreamCreate");
  if ((e = cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking)) != cudaSuccess)
    return bail(e, "cudaStreamCreate");
  if ((e = cudaEventCreate(&ctx->raw_ev)) != cudaSuccess) return bail(e, "cudaEventCreate");
  if ((e = cudaEventCreateWithFlags(&ctx->off_ev, cudaEventDisableTiming)) != cudaSuccess)
    return bail(e, "cudaEventCreate");
  if ((e = cudaEventCreateWithFlags(&ctx->load_done, cudaEventDisableTiming)) != cudaSuccess)
    return bail(e, "cudaEventCreate");
  if ((e = cudaHostAlloc((void **)&ctx->h_summary, (size_t)(2 + NBUCKETS) * 4, cudaHostAllocDefault)) != cudaSuccess)
    return bail(e, "cudaHostAlloc");
  if ((e = cudaHostAlloc((void **)&ctx->h_small, 64 * 8, cudaHostAllocDefault)) != cudaSuccess)
    return bail(e, "cudaHostAlloc");
  if ((e = cudaHostAlloc((void **)&ctx->h_stage, STAGE_WORDS * 4, cudaHostAllocDefault)) != cudaSuccess)
    return bail(e, "cudaHostAlloc");
  *out = ctx;
  return ISH_OK;
}

void ish_gpu_close(ish_ctx *ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  stop_server(ctx);
  (void)finish_pending_load(ctx);
  cudaStreamSynchronize(ctx->stream);
  free_plans(ctx);
  for (auto &kv : ctx->queries) release_query(kv.second);
  for (auto &kv : ctx->sets) release_set(kv.second);
  for (RecordSet &sp : ctx->spare_sets) release_set(sp);
  DevBuf *bufs[] = {&ctx->raw, &ctx->off_in, &ctx->len_tmp, &ctx->poff_tmp, &ctx->hist, &ctx->summary,
                    &ctx->scan_tmp, &ctx->counter, &ctx->error, &ctx->out_score, &ctx->out_qend, &ctx->out_tend,
                    &ctx->out_hit, &ctx->hit_idx, &ctx->block_counts, &ctx->nhits, &ctx->plain_scratch,
                    &ctx->enc_tables, &ctx->nl_pos, &ctx->line_end, &ctx->starts_ws, &ctx->starts_codes};
  for (DevBuf *b : bufs) b->release();
  ctx->exact.release();
  ctx->window_out.release();
  ctx->starts_windows.release();
  ctx->fastx.release();
  cudaEventDestroy(ctx->ev0);
  cudaEventDestroy(ctx->ev1);
  cudaEventDestroy(ctx->load_done);
  cudaStreamDestroy(ctx->load_stream);
  if (ctx->raw_ev) cudaEventDestroy(ctx->raw_ev);
  if (ctx->off_ev) cudaEventDestroy(ctx->off_ev);
  if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
  cudaFreeHost(ctx->h_summary);
  if (ctx->h_small) cudaFreeHost(ctx->h_small);
  if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
  for (cudaEvent_t ev : ctx->load_ev) cudaEventDestroy(ev);
  cudaStreamDestroy(ctx->stream);
  delete ctx;
}

const char *ish_gpu_last_error(const ish_ctx *ctx) { return ctx ? ctx->err.c_str() : g_open_error.c_str(); }

int ish_gpu_set_option(ish_ctx *ctx, int option, int64_t value) {
  if (!ctx) return ISH_EINVAL;
  // the serving thread reads the options for every step
  if (ctx->server) return fail(ctx, ISH_EINVAL, "options cannot change while the serving loop runs");
  switch (option) {
  case ISH_OPT_KERNEL:
    if (value < ISH_KERNEL_AUTO || value > ISH_KERNEL_PLAIN16)
      return fail(ctx, ISH_EINVAL, "bad kernel %lld", (long long)value);
    ctx->kernel = (int)value;
    return ISH_OK;
  case ISH_OPT_SG_LANES:
  case ISH_OPT_SW_U8_LANES:
  case ISH_OPT_SW_U16_LANES:
    if (value < 1 || value > 64) return fail(ctx, ISH_EINVAL, "lane count must be in 1..64");
    (option == ISH_OPT_SG_LANES ? ctx->sg_lanes : option == ISH_OPT_SW_U8_LANES ? ctx->sw_u8_lanes : ctx->sw_u16_lanes) =
        (int)value;
    return ISH_OK;
  case ISH_OPT_WAVE_GROUP:
    if (value != 0 && (value < 1 || value > 32 || (value & (value - 1))))
      return fail(ctx, ISH_EINVAL, "group size must be 0 or a power of two <= 32");
    ctx->force_G = (int)value;
    drop_plans(ctx, 0, 0);
    return ISH_OK;
  case ISH_OPT_PROFILE_LAYOUT:
    if (value < -1 || value > PROF_S32) return fail(ctx, ISH_EINVAL, "profile layout must be -1, 0, 1 or 2");
    ctx->force_layout = (int)value;
    drop_plans(ctx, 0, 0);
    return ISH_OK;
  case ISH_OPT_WAVE_K:
    if (value != 0 && !wave_k_available((int)value))
      return fail(ctx, ISH_EINVAL, "K must be 0, 1..32 or even up to %d", WAVE_KMAX);
    ctx->force_K = (int)value;
    drop_plans(ctx, 0, 0);
    return ISH_OK;
  case ISH_OPT_WINDOWS:
    if (value != 0 && value != 1) return fail(ctx, ISH_EINVAL, "windows must be 0 or 1");
    if (ctx->windows_on != (int)value) free_plans(ctx);  // batched plans window the set or not
    ctx->windows_on = (int)value;
    return ISH_OK;
  case ISH_OPT_WAVE_LEAN:
    if (value < -1 || value > 1) return fail(ctx, ISH_EINVAL, "lean variant must be -1, 0 or 1");
    ctx->force_lean = (int)value;
    drop_plans(ctx, 0, 0);
    return ISH_OK;
  case ISH_OPT_STEP_BUDGET:
    if (value < 0) return fail(ctx, ISH_EINVAL, "step budget must be >= 0");
    ctx->step_budget = (uint64_t)value;
    drop_plans(ctx, 0, 0);
    return ISH_OK;
  case ISH_OPT_SERVE_STEP_CELLS:
    if (value < 0) return fail(ctx, ISH_EINVAL, "serving step cells must be >= 0");
    ctx->serve_step_cells = (double)value;
    return ISH_OK;
  case ISH_OPT_FAULT_ALLOC:
    if (value < -1) return fail(ctx, ISH_EINVAL, "allocation fault countdown must be >= -1");
    g_alloc_fault.store(value);
    return ISH_OK;
  case ISH_OPT_WAVE_BLOCKS:
    if (value < 0 || value > 32) return fail(ctx, ISH_EINVAL, "blocks per SM must be in 0..32");
    ctx->force_blocks = (int)value;
    drop_plans(ctx, 0, 0);
    return ISH_OK;
  default:
    return fail(ctx, ISH_EINVAL, "unknown option %d", option);
  }
}

int ish_gpu_set_query(ish_ctx *ctx, const uint8_t *enc_query, uint32_t qlen, int matrix_kind, const int8_t *matrix,
                      uint32_t alphabet, int algo, uint32_t gap_open, uint32_t gap_ext, uint32_t ends_free,
                      int32_t max_score, float threshold, int32_t *query_id) {
  if (!ctx || !query_id) return ctx ? fail(ctx, ISH_EINVAL, "query_id is NULL") : ISH_EINVAL;
  if (algo != ISH_ALGO_SEMI_GLOBAL && algo != ISH_ALGO_LOCAL) return fail(ctx, ISH_EINVAL, "unknown algorithm %d", algo);
  if (matrix_kind < ISH_MATRIX_ASCII || matrix_kind > ISH_MATRIX_BLOSUM62)
    return fail(ctx, ISH_EINVAL, "unknown matrix kind %d", matrix_kind);
  if (!matrix || !matrix_alphabet_ok(alphabet)) return fail(ctx, ISH_EINVAL, "matrix must be alphabet^2 int8, alphabet 1..256");
  if (qlen && !enc_query) return fail(ctx, ISH_EINVAL, "enc_query is NULL");
  if (qlen > 32767) return fail(ctx, ISH_EOVERFLOW, "query of %u residues is longer than 32767", qlen);
  if (ends_free > 15) return fail(ctx, ISH_EINVAL, "ends_free has bits above ISH_FREE_TARGET_END");
  Query q;
  q.algo = algo;
  q.kind = matrix_kind;
  q.alphabet = (int)alphabet;
  q.Q = (int)qlen;
  // The matchers hand UInt penalties to lanes of the pass type: int16 for the
  // semi-global pass (striped_semi_global_matcher.mojo:232-245), uint8 for
  // ssw_align (local_aln/striped.mojo:151-152).
  if (algo == ISH_ALGO_SEMI_GLOBAL) {
    q.open = (int16_t)gap_open;
    q.ext = (int16_t)gap_ext;
  } else {
    q.open = (uint8_t)gap_open;
    q.ext = (uint8_t)gap_ext;
  }
  q.ends = algo == ISH_ALGO_SEMI_GLOBAL ? (int)ends_free : 0;
  q.max_score = max_score;
  q.thr = threshold;
  q.M.assign(matrix, matrix + (size_t)alphabet * alphabet);
  q.q.assign(enc_query, enc_query + qlen);
  for (uint32_t i = 0; i < qlen; ++i)
    if (q.q[i] >= alphabet) return fail(ctx, ISH_EINVAL, "query code %u at %u >= alphabet %u", q.q[i], i, alphabet);
  q.mmin = 0;
  q.mmax = 0;
  for (int8_t v : q.M) {
    q.mmin = std::min<int>(q.mmin, v);
    q.mmax = std::max<int>(q.mmax, v);
  }
  q.neg_limit = neg_limit_of(q.open, q.mmin);
  {
    std::vector<int> hi(alphabet, 0), lo(alphabet, 0);  // per query code, over the record codes
    for (uint32_t c = 0; c < alphabet; ++c)
      for (uint32_t j = 0; j < alphabet; ++j) {
        hi[j] = std::max<int>(hi[j], q.M[(size_t)c * alphabet + j]);
        lo[j] = std::min<int>(lo[j], q.M[(size_t)c * alphabet + j]);
      }
    for (uint8_t c : q.q) {
      q.col_max_sum += hi[c];
      q.col_min_sum += lo[c];
    }
  }
  compute_rows(q);
  cudaSetDevice(ctx->device);
  const int32_t id = ctx->next_query++;
  ctx->queries.emplace(id, std::move(q));
  *query_id = id;
  return ISH_OK;
}

int ish_gpu_free_query(ish_ctx *ctx, int32_t query_id) {
  if (!ctx) return ISH_EINVAL;
  auto it = ctx->queries.find(query_id);
  if (it == ctx->queries.end()) return fail(ctx, ISH_EINVAL, "unknown query %d", query_id);
  cudaStreamSynchronize(ctx->stream);
  drop_plans(ctx, query_id, 0);
  release_query(it->second);
  ctx->queries.erase(it);
  return ISH_OK;
}

int ish_gpu_records_load(ish_ctx *ctx, const uint8_t *records, const uint64_t *offsets, uint32_t n, int32_t *set_id) {
  if (!ctx || !set_id) return ctx ? fail(ctx, ISH_EINVAL, "set_id is NULL") : ISH_EINVAL;
  if (int rc0 = finish_pending_load(ctx)) return rc0;
  LoadTimer timer(ctx);
  cudaSetDevice(ctx->device);
  RecordSet rs;
  int rc = load_records(ctx, records, offsets, n, rs, nullptr);
  if (rc) {
    release_set(rs);
    return rc;
  }
  const int32_t id = ctx->next_set++;
  ctx->sets.emplace(id, std::move(rs));
  *set_id = id;
  return ISH_OK;
}

int ish_gpu_records_load_async(ish_ctx *ctx, const uint8_t *records, const uint64_t *offsets, uint32_t n,
                               int32_t *set_id) {
  if (!ctx || !set_id) return ctx ? fail(ctx, ISH_EINVAL, "set_id is NULL") : ISH_EINVAL;
  // one load in flight: the previous one completes first (its scratch is reused)
  if (int rc0 = finish_pending_load(ctx)) return rc0;
  LoadTimer timer(ctx);
  cudaSetDevice(ctx->device);
  RecordSet rs;
  if (ctx->load_times_due) load_phase_times(ctx);  // before its events are used again
  // the load stream starts after the work already queued on the context's
  // stream (a set freed just before may still be read there)
  CU(cudaEventRecord(ctx->load_ev[0], ctx->stream));
  CU(cudaStreamWaitEvent(ctx->load_stream, ctx->load_ev[0], 0));
  int rc = load_records(ctx, records, offsets, n, rs, nullptr, ctx->load_stream, true);
  if (rc) {
    cudaStreamSynchronize(ctx->load_stream);
    release_set(rs);
    return rc;
  }
  const int32_t id = ctx->next_set++;
  const bool pending = rs.pending;
  ctx->sets.emplace(id, std::move(rs));
  if (pending) ctx->pending_set = id;
  *set_id = id;
  return ISH_OK;
}

int ish_gpu_records_load_raw(ish_ctx *ctx, const uint8_t *raw, const uint64_t *offsets, uint32_t n, int matrix_kind,
                             int32_t *set_id) {
  if (!ctx || !set_id) return ctx ? fail(ctx, ISH_EINVAL, "set_id is NULL") : ISH_EINVAL;
  if (int rc0 = finish_pending_load(ctx)) return rc0;
  LoadTimer timer(ctx);
  cudaSetDevice(ctx->device);
  const uint8_t *enc = nullptr;
  int rc = device_encoding(ctx, matrix_kind, &enc);
  if (rc) return rc;
  RecordSet rs;
  rc = load_records(ctx, raw, offsets, n, rs, enc);
  if (rc) {
    release_set(rs);
    return rc;
  }
  const int32_t id = ctx->next_set++;
  ctx->sets.emplace(id, std::move(rs));
  *set_id = id;
  return ISH_OK;
}

int ish_gpu_records_load_lines(ish_ctx *ctx, const uint8_t *text, uint64_t bytes, int matrix_kind, int32_t *set_id,
                               uint32_t *n_records) {
  if (!ctx || !set_id) return ctx ? fail(ctx, ISH_EINVAL, "set_id is NULL") : ISH_EINVAL;
  if (int rc0 = finish_pending_load(ctx)) return rc0;
  LoadTimer timer(ctx);
  cudaSetDevice(ctx->device);
  const uint8_t *enc = nullptr;
  int rc = device_encoding(ctx, matrix_kind, &enc);
  if (rc) return rc;
  RecordSet rs;
  uint32_t n = 0;
  rc = load_lines(ctx, text, bytes, rs, enc, &n);
  if (rc) {
    release_set(rs);
    return rc;
  }
  const int32_t id = ctx->next_set++;
  ctx->sets.emplace(id, std::move(rs));
  *set_id = id;
  if (n_records) *n_records = n;
  return ISH_OK;
}

int ish_gpu_records_free(ish_ctx *ctx, int32_t set_id) {
  if (!ctx) return ISH_EINVAL;
  int urc = ISH_OK;
  RecordSet *it_set = use_set(ctx, set_id, &urc);
  if (!it_set) return urc;
  if (server_uses_set(ctx, set_id)) return fail(ctx, ISH_EINVAL, "record set %d is used by the serving loop", set_id);
  auto it = ctx->sets.find(set_id);
  cudaStreamSynchronize(ctx->stream);
  drop_plans(ctx, 0, set_id);
  recycle_set(ctx, it->second);
  ctx->sets.erase(it);
  return ISH_OK;
}

int ish_gpu_records_info(ish_ctx *ctx, int32_t set_id, uint32_t *n, uint64_t *total_bytes) {
  if (!ctx) return ISH_EINVAL;
  int urc = ISH_OK;
  RecordSet *it_set = use_set(ctx, set_id, &urc);
  if (!it_set) return urc;
  if (n) *n = it_set->n;
  if (total_bytes) *total_bytes = it_set->total;
  return ISH_OK;
}

int ish_gpu_score_set(ish_ctx *ctx, int32_t query_id, int32_t set_id, int32_t *score, int32_t *query_end,
                      int32_t *target_end, uint8_t *hit, uint32_t *hit_idx, uint32_t *n_hits) {
  if (!ctx) return ISH_EINVAL;
  auto qi = ctx->queries.find(query_id);
  if (qi == ctx->queries.end()) return fail(ctx, ISH_EINVAL, "unknown query %d", query_id);
  int urc = ISH_OK;
  RecordSet *si_set = use_set(ctx, set_id, &urc);
  if (!si_set) return urc;
  cudaSetDevice(ctx->device);
  int rc = run_scoring(ctx, qi->second, *si_set);
  if (rc) {
    cudaStreamSynchronize(ctx->stream);
    return rc;
  }
  return fetch_outputs(ctx, si_set->n, score, query_end, target_end, hit, hit_idx, n_hits);
}

int ish_gpu_score(ish_ctx *ctx, int32_t query_id, const uint8_t *records, const uint64_t *offsets, uint32_t n,
                  int32_t *score, int32_t *query_end, int32_t *target_end, uint8_t *hit, uint32_t *hit_idx,
                  uint32_t *n_hits) {
  if (!ctx) return ISH_EINVAL;
  auto qi = ctx->queries.find(query_id);
  if (qi == ctx->queries.end()) return fail(ctx, ISH_EINVAL, "unknown query %d", query_id);
  cudaSetDevice(ctx->device);
  if (int rc0 = finish_pending_load(ctx)) return rc0;
  RecordSet rs;
  const int alphabet = qi->second.alphabet;
  const uint32_t limit = n && n <= SORT_SMALL && alphabet < 256 ? (uint32_t)alphabet : 0;
  int rc = load_records(ctx, records, offsets, n, rs, nullptr, nullptr, false, limit);
  if (!rc) rc = run_scoring(ctx, qi->second, rs);
  if (!rc)
    rc = fetch_outputs(ctx, n, score, query_end, target_end, hit, hit_idx, n_hits,
                       limit && qi->second.Q ? ctx->summary.as<uint32_t>() : nullptr, alphabet);
  cudaStreamSynchronize(ctx->stream);
  recycle_set(ctx, rs);  // the next call's set takes these buffers
  return rc;
}

int ish_gpu_calibrate(ish_ctx *ctx, double *dpx_ops_per_s) {
  if (!ctx || !dpx_ops_per_s) return ISH_EINVAL;
  cudaSetDevice(ctx->device);
  CU(ctx->counter.ensure(64));
  const int blocks = ctx->num_sms * 8, threads = 256, iters = 8192;
  cudaStream_t s = ctx->stream;
  k_dpx_peak<<<blocks, threads, 0, s>>>(ctx->counter.as<uint32_t>(), 256, 0x00010001u, 0xfffbfffbu);  // warm-up
  CU(cudaEventRecord(ctx->ev0, s));
  ++ctx->launches;
  k_dpx_peak<<<blocks, threads, 0, s>>>(ctx->counter.as<uint32_t>(), iters, 0x00010001u, 0xfffbfffbu);
  ++ctx->launches;
  CU(cudaEventRecord(ctx->ev1, s));
  CU(cudaGetLastError());
  CU(cudaStreamSynchronize(s));
  float ms = 0.f;
  CU(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  *dpx_ops_per_s = (double)blocks * threads * iters * 8 / (ms * 1e-3);
  return ISH_OK;
}

int ish_gpu_calibrate_lanes(ish_ctx *ctx, double *s16x2_cells_per_s, double *u8x4_cells_per_s) {
  if (!ctx) return ISH_EINVAL;
  if (!s16x2_cells_per_s || !u8x4_cells_per_s) return fail(ctx, ISH_EINVAL, "NULL output");
  cudaSetDevice(ctx->device);
  CU(ctx->counter.ensure(64));
  const int blocks = ctx->num_sms * 8, threads = 256, rows = 4096;
  cudaStream_t s = ctx->stream;
  for (int u8 = 0; u8 < 2; ++u8) {
    const LaneFn fn = lane_rows_fn(u8 != 0);
    const uint32_t open = u8 ? 0x0a0a0a0au : 10u, ext = u8 ? 0x01010101u : 1u;
    fn<<<blocks, threads, 0, s>>>(ctx->counter.as<uint32_t>(), 64, 0x03020104u, open, ext, 0x04040404u);  // warm-up
    CU(cudaEventRecord(ctx->ev0, s));
    fn<<<blocks, threads, 0, s>>>(ctx->counter.as<uint32_t>(), rows, 0x03020104u, open, ext, 0x04040404u);
    CU(cudaEventRecord(ctx->ev1, s));
    ctx->launches += 2;
    CU(cudaGetLastError());
    CU(cudaStreamSynchronize(s));
    float ms = 0.f;
    CU(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    // 16 words per thread and row, 2 or 4 cells per word
    const double cells = (double)blocks * threads * rows * 16 * (u8 ? 4 : 2);
    (u8 ? *u8x4_cells_per_s : *s16x2_cells_per_s) = cells / (ms * 1e-3);
  }
  return ISH_OK;
}

int ish_gpu_launch_count(ish_ctx *ctx, uint64_t *count) {
  if (!ctx || !count) return ISH_EINVAL;
  *count = ctx->launches.load();
  return ISH_OK;
}

int ish_gpu_last_windows(ish_ctx *ctx, uint32_t *windows) {
  if (!ctx || !windows) return ISH_EINVAL;
  *windows = ctx->last_windows;
  return ISH_OK;
}

int ish_gpu_last_kernel_ms(ish_ctx *ctx, double *ms) {
  if (!ctx || !ms) return ISH_EINVAL;
  *ms = ctx->last_ms;
  return ISH_OK;
}

int ish_gpu_last_load_ms(ish_ctx *ctx, double *upload_ms, double *pack_ms, double *wall_ms) {
  if (!ctx) return ISH_EINVAL;
  if (ctx->load_times_due) load_phase_times(ctx);
  if (upload_ms) *upload_ms = ctx->last_load_ms[0];
  if (pack_ms) *pack_ms = ctx->last_load_ms[1];
  if (wall_ms) *wall_ms = ctx->last_load_ms[2];
  return ISH_OK;
}

}  // extern "C"

// Dispatch over the instantiation files.
namespace ish {
WaveFn wave_fn_a(int, int, int);
WaveFn wave_fn_b(int, int, int);
WaveFn wave_fn_c(int, int, int);
WaveFn wave_fn_d(int, int, int);
WaveFn wave_fn_e(int, int, int);
WaveFn wave_fn_f(int, int, int);
WaveFn wave_fn_g(int, int, int);
BatchFn batch_fn_g(int, int, int);
WaveFn wave_fn_h(int, int, int);
BatchFn batch_fn_h(int, int, int);
WaveFn wave_fn(int K, int mode, int layout, int lean) {
  if (K < 1) return nullptr;
  if (lean && wave_has_lean(K)) return K <= 32 ? wave_fn_h(K, mode, layout) : wave_fn_g(K, mode, layout);
  if (K <= 8) return wave_fn_a(K, mode, layout);
  if (K <= 16) return wave_fn_b(K, mode, layout);
  if (K <= 24) return wave_fn_c(K, mode, layout);
  if (K <= 32) return wave_fn_d(K, mode, layout);
  if (K <= 48) return wave_fn_e(K, mode, layout);
  return wave_fn_f(K, mode, layout);
}
BatchFn batch_fn_a(int, int, int);
BatchFn batch_fn_b(int, int, int);
BatchFn batch_fn_c(int, int, int);
BatchFn batch_fn_d(int, int, int);
BatchFn batch_fn_e(int, int, int);
BatchFn batch_fn_f(int, int, int);
BatchFn batch_fn(int K, int mode, int layout, int lean) {
  if (K < 1) return nullptr;
  if (lean && wave_has_lean(K)) return K <= 32 ? batch_fn_h(K, mode, layout) : batch_fn_g(K, mode, layout);
  if (K <= 8) return batch_fn_a(K, mode, layout);
  if (K <= 16) return batch_fn_b(K, mode, layout);
  if (K <= 24) return batch_fn_c(K, mode, layout);
  if (K <= 32) return batch_fn_d(K, mode, layout);
  if (K <= 48) return batch_fn_e(K, mode, layout);
  return batch_fn_f(K, mode, layout);
}
}  // namespace ish
