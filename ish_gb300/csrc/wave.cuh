// wave.cuh -- the wavefront scoring kernel.
//
// A group of G threads (G = 1, 2, ..., 32; a sub-warp) scores a PAIR of
// records at once: the low and high 16-bit halves of every register belong to
// record A and record B of the pair.  Thread t of the group owns K consecutive
// query columns [t*K - d, (t+1)*K - d); the query is padded at the front with
// d >= 1 columns whose profile and boundary values make them transparent (see
// build_wave_layout in ish_gpu.cu), so the last query column is always the
// last register of thread G-1.  Rows flow through the group as a software
// pipeline: thread t processes row i of the pair one step after thread t-1
// did, receiving H(i, first column - 1) and F(i, first column) through
// __shfl_up_sync.  G = 1 is "one thread per record pair with packed 16-bit
// lanes" for short queries; G = 32 is a warp-wide anti-diagonal wavefront for
// long queries.
//
// The packed values are unsigned 16-bit, raised by a bias, and a row is one
// pass over the thread's columns that updates H and E in place.  E and F open
// from H.  The DPX add-max and three-input maximum share one pipe (16 lanes per
// clock and sub-partition), which bounds the row, so whatever can be a plain
// 32-bit add of both halves -- the bias keeps the low half from borrowing from
// the high one -- runs beside it on the integer multiply-add pipe.
//
// Local alignment, four DPX instructions and two adds per cell and record pair
// (two cells), the first of which assembles the pair's profile word P:
//   T = max(Hdiag + P, floor);  H = max3(T, E, F);  u = H - open
//   E = max(E - ext, u);  F = max(F - ext, u)
// with the floor at score 0 and half a three-input maximum per column for the
// row's best.  (The five-instruction form that floors H - open instead, and one
// in which max3(Hdiag + P, E, floor) leaves the F chain one instruction long,
// measured 5 % and 3 % slower at 38 columns.)
//
// Semi-global, three DPX instructions and an add (two with the 32-bit profile):
//   T = Hdiag + P;  H = max3(T, E, F);  E = max(H + c, E);  F = max(H + c, F)
// The values are also raised by frames that rise by ext per row and per column:
// a gap extension then costs nothing, so both gap updates are one add-max with
// the same c = ext - open, and the profile carries +2 ext for the diagonal
// step.  Rows drop back to frame 0 every R rows
// (R * ext <= 2048); the column frame runs over the whole padded query.  P is
// the pair's scores as ONE signed integer b * 65536 + a.  wave_params() in
// ish_gpu.cu derives the bias and shows that every value fits 16 bits.
// (Local alignment cannot use frames: its floor would move with them.)
// Measured on GB300 (row loops alone, 38 columns per thread): 9.3 clocks per
// column and warp with the 32-bit profile, where the shared-memory loads bound
// it (8.4), 8.0 with the pair profile, against 11.8 for four DPX per cell pair.
// The 16-bit profile is joined by a PRMT per column, whose halves cannot be
// added as one integer; it keeps T = max(Hdiag + P, E), H = max(T, F).
//
// End coordinates follow the reference exactly:
//   semi-global, target end free: first row where H(i, Q-1) strictly beats the
//     running maximum (ishlib/matcher/alignment/semi_global_aln/striped.mojo:436-450);
//   semi-global, query end free: smallest query column of the maximum of the
//     last row, with the tie rule of striped.mojo:453-468;
//   local: first row whose column maximum strictly beats every earlier cell,
//     smallest query column of that maximum in that row
//     (ishlib/matcher/alignment/local_aln/striped.mojo:395-428).
#pragma once

#include "kernels.cuh"

namespace ish {

// Scores sorted entries [p.first, p.first + p.count) of the record set: the
// groups of the calling block take record pairs from *counter until none are
// left.  With DEAL (the launch's blocks all start on this range) a group's first
// pair is dealt instead: the longest pairs to the first warp of every block, the
// next to the second, and the counter hands out what is left.  When the groups
// took them from the counter the first blocks got all the longest pairs, and a
// set of little more than a pair per group was bound by those blocks (100,000
// lines 215 -> 205 us, 3,000 proteins with match starts 887 -> 860).  `prof` is
// the profile in shared memory; `slots_all` holds one word per thread (a group's
// G pair indices in flight), `save_all` wave_save_words(K) words per thread
// (local alignment only).
template <int K, int MODE, int LAYOUT, bool DEAL>
__device__ __forceinline__ void wave_rows(const WaveParams &p, const unsigned char *prof, uint32_t *slots_all,
                                          uint32_t *save_all, uint32_t *counter) {
  constexpr int RPS = (MODE == SG) ? WAVE_RPS_SG : WAVE_RPS_SW;
  static_assert(RPS == 2 || RPS == 4, "rows per step: 2 or 4");
  const int tid = threadIdx.x;
  const int G = p.G;
  const int lane = tid & 31;
  const int t = lane & (G - 1);
  const bool t0 = t == 0;
  // pair indices in flight in the group, by sequence number modulo G: a pair
  // is in at most G consecutive steps' threads, so thread 0 rewrites its slot
  // only after thread G-1 has left it
  uint32_t *slots = slots_all + (tid & ~(G - 1));
  // local alignment: per thread, the H row of the last improvement of each lane
  constexpr int KP8 = (K + 7) & ~7;
  uint16_t *saveA = reinterpret_cast<uint16_t *>(save_all + tid * wave_save_words(K));
  uint16_t *saveB = saveA + KP8;

  const unsigned FULL = 0xffffffffu;
  // local: score 0, and -open in both halves as one integer
  const uint32_t FLOOR = (uint32_t)p.bias * 0x10001u, NOPEN_SUM = (uint32_t)(-p.open) * 0x10001u;
  const uint32_t NEXT = p.pk_next;
  // semi-global: a gap opens from H at ext - open in the frames
  const uint32_t EOPEN = p.pk_eopen;
  const uint32_t EOPEN_SUM = (uint32_t)(p.ext - p.open) * 0x10001u;  // ... as one integer for both halves
  const bool te = (MODE == SG) && (p.ends & 8);
  const bool qe = (MODE == SG) && (p.ends & 2);
  // record pairs of the range: every pair_stride-th from pair_phase
  const uint32_t pstride = p.pair_stride ? p.pair_stride : 1u, pphase = p.pair_stride ? p.pair_phase : 0u;
  const uint32_t npairs_all = (p.count + 1) >> 1;
  const uint32_t npairs = npairs_all > pphase ? (npairs_all - pphase + pstride - 1) / pstride : 0u;
  const int col0 = t * K - p.d;  // query column of register 0
  // parameters read every step, held in registers (the batched kernel's
  // parameters live in shared memory)
  const int kp = p.kp, alpha = p.alphabet, fmask = p.frame_mask, ext = p.ext;
  const uint32_t remap_off = p.remap_off, lane_mul = p.lane_mul;
  // the frame of a row (always 0 for local alignment)
  auto frame_of = [&](int r) { return (MODE == SG) ? (r & fmask) * ext : 0; };
  // semi-global: H entering the padding from the left at row r is
  // left0 + frame(r) / ext * left_ext (left_ext 0: a floor below every value)
  const uint32_t LEFT0 = (MODE == SG) ? p.pk_left : 0u;
  const uint32_t LEFT_EXT = (MODE == SG) ? p.pk_left_ext : 0u;
  // this thread's part of every profile row, and the bytes between the rows
  // of consecutive codes: a row's address is one multiply-add
  const unsigned char *prof_t = prof + (uint32_t)((lane & (p.slots - 1)) * kp) * (LAYOUT == PROF_S16 ? 2u : 4u);
  const uint32_t row_bytes = p.row_bytes;

  uint32_t H[K], E[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    H[j] = 0;
    E[j] = 0;
  }
  uint32_t prevH = 0;  // H(row above the step's first row, column col0 - 1)
  // passed to thread t+1: per row of the step, H of the last column and F
  // leaving it; local alignment: the best of this thread's and all earlier
  // columns up to the step's last row, which the next thread uses a step later
  uint32_t outH[RPS], outF[RPS], outB = 0, left_best = 0;
  // local alignment: the best of all later columns in the rows that the next
  // thread, a step behind, had left when this step began
  uint32_t right_best = 0;
#pragma unroll
  for (int k = 0; k < RPS; ++k) outH[k] = outF[k] = 0;
  uint32_t outC = CTL_IDLE;
  int q4 = 0, lenA = 0, lenB = 0;  // q4: row of the step's first row
  // the next q4 at which this thread has anything beside its rows to do, and
  // (thread 0) the q4 at which its pair has no rows left
  int wake = t0 ? RPS : 0x7fffffff, end_q = t0 ? RPS : -1;
  // this thread's record streams: 4 codes per 32-bit word, one word ahead
  const uint8_t *pa = nullptr, *pb = nullptr;
  uint32_t wA = 0, wB = 0, nA = 0, nB = 0;
  // tracking
  // SG: lane-wise running max of H(i, Q-1), at thread G-1 (the other threads
  // hold the largest value, so that none of their rows count); SW: of this
  // thread's cells
  uint32_t best = 0;
  int rowA = -1, rowB = -1;  // first row of the lane's maximum
  // last-row partials for thread t+1: semi-global in registers, local alignment
  // in the padding behind the thread's saved row: scores and columns of A and B
  // (16 bits each), then their rows
  uint32_t oR0 = 0, oR1 = 0;
  constexpr int save_stride = wave_save_words(K) / 4;
  uint4 *partial = reinterpret_cast<uint4 *>(save_all + tid * wave_save_words(K) + KP8);
  bool ended = false;  // a record of the warp ended in the last step
  const bool remap = remap_off != 0;
  // whether the ends of records matter to this thread: with the query end
  // fixed, only the last column (thread G-1) gives a semi-global result
  const bool ends_here = MODE == SW || qe || t == G - 1;
  // thread 0 of the group holds the next pair's number: it is taken CLAIM rows
  // before the current pair ends, late enough that a group with a long pair
  // leaves the next ones to the others, and early enough that neither the
  // counter nor the new pair's lengths and codes are waited for
  uint32_t f_next = 0;
  // The pairs dealt come before the counter's.  (Semi-global computes their number,
  // local alignment takes it from the parameters: the other way round the register
  // allocation at 38 columns costs each 0.7 to 1 %.)
  const auto claim = [&]() -> uint32_t {
    const uint32_t dealt = MODE == SG ? (gridDim.x * blockDim.x) >> __popc(G - 1) : p.dealt;
    return atomicAdd(counter, 1u) + (DEAL ? dealt : 0u);
  };
  const int lgG = __popc(G - 1);
  if (t0) f_next = DEAL ? ((tid >> 5) * gridDim.x + blockIdx.x) * (32u >> lgG) + (lane >> lgG) : claim();
  constexpr int CHK = 8 / RPS;  // steps between termination checks
  constexpr int CLAIM = 32, LOOK_META = 20, LOOK_CODES = 8;  // rows before a pair's end (see below)
  uint32_t step = 0;

  // One row of the pair with record codes cA, cB: `diag` is H of the row above
  // at column col0 - 1, `fs` is F entering column col0.  Updates H and E in
  // place, column by column from the left (each profile word is used as it
  // arrives, which keeps few of them in registers), and returns F leaving the
  // last column.
  auto row_step = [&](uint32_t cA, uint32_t cB, uint32_t diag, uint32_t fs) -> uint32_t {
    // one column: `dp` is the pair's scores, semi-global (but for PROF_S16)
    // with H of the row above one column to the left added
    auto cell = [&](int j, uint32_t dp) {
      uint32_t &h = H[j], &e = E[j];
      if (MODE == SG && LAYOUT != PROF_S16) {
        diag = h;
        h = __vimax3_u16x2(dp, e, fs);
        e = __viaddmax_u16x2(h, EOPEN, e);
        fs = __viaddmax_u16x2(h, EOPEN, fs);
      } else if (MODE == SG) {
        const uint32_t T = __viaddmax_u16x2(diag, dp, e);
        diag = h;
        h = __vmaxu2(T, fs);
        e = __viaddmax_u16x2(T, EOPEN, e);
        fs = __viaddmax_u16x2(T, EOPEN, fs);
      } else {
        const uint32_t T = __viaddmax_u16x2(diag, dp, FLOOR);
        diag = h;
        h = __vimax3_u16x2(T, e, fs);
        const uint32_t u = h + NOPEN_SUM;
        e = __viaddmax_u16x2(e, NEXT, u);
        fs = __viaddmax_u16x2(fs, NEXT, u);
      }
    };
    if (LAYOUT == PROF_PAIR) {
      const uint4 *r4 = reinterpret_cast<const uint4 *>(prof_t + (cA * alpha + cB) * row_bytes);
#pragma unroll
      for (int v = 0; v < (K + 3) / 4; ++v) {
        const uint4 w = r4[v];
        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (4 * v + m < K) cell(4 * v + m, MODE == SG ? ww[m] + diag : ww[m]);
      }
    } else if (LAYOUT == PROF_S32) {
      // a 32-bit word per code; the packed pair is b * 65536 + a, one integer
      // multiply-add (the multiplier is a runtime value, so this stays an IMAD
      // on the FMA pipe, which the DPX recurrence on the ALU pipe leaves idle)
      const uint4 *ra = reinterpret_cast<const uint4 *>(prof_t + cA * row_bytes);
      const uint4 *rb = reinterpret_cast<const uint4 *>(prof_t + cB * row_bytes);
      const uint32_t mul = lane_mul;
#pragma unroll
      for (int v = 0; v < (K + 3) / 4; ++v) {
        const uint4 a = ra[v], b = rb[v];
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (4 * v + m < K) cell(4 * v + m, MODE == SG ? aw[m] + (bw[m] * mul + diag) : bw[m] * mul + aw[m]);
      }
    } else {
      // 16-bit words (profiles too large for the 32-bit layout): one PRMT
      // per packed pair
      const uint4 *ra = reinterpret_cast<const uint4 *>(prof_t + cA * row_bytes);
      const uint4 *rb = reinterpret_cast<const uint4 *>(prof_t + cB * row_bytes);
#pragma unroll
      for (int v = 0; v < (K + 7) / 8; ++v) {
        const uint4 a = ra[v], b = rb[v];
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          if (8 * v + 2 * m < K) cell(8 * v + 2 * m, __byte_perm(aw[m], bw[m], 0x5410));
          if (8 * v + 2 * m + 1 < K) cell(8 * v + 2 * m + 1, __byte_perm(aw[m], bw[m], 0x7632));
        }
      }
    }
    return fs;
  };

  // Local alignment, after row `row` (`live`: the halves of the lanes whose
  // record holds that row): a row maximum that does not beat every cell so far
  // in this thread, in the columns to its left AND in earlier rows of those to
  // its right can never be the first row of the record's maximum at its smallest
  // column (it is smaller, or equal in a later row or a larger column), so only
  // the others are recorded.  `thr` is that bar: this thread's rows up to the
  // last, the left columns' rows up to the last step (a later row of theirs may
  // tie without winning), and the rows the right columns have reached (they run
  // behind).
  auto sw_track = [&](int row, uint32_t &thr, uint32_t live) {
    uint32_t cm = H[0];
#pragma unroll
    for (int j = 1; j + 1 < K; j += 2) cm = __vimax3_u16x2(cm, H[j], H[j + 1]);
    if ((K & 1) == 0 && K > 1) cm = __vmaxu2(cm, H[K - 1]);
    cm &= live;
    const uint32_t nb = __vmaxu2(thr, cm);
    if (nb != thr) {
      // keep this row (shared-memory stores only); the column of the maximum
      // is looked up once, at the record's last row
      const bool upA = ulo16(cm) > ulo16(thr), upB = uhi16(cm) > uhi16(thr);
      // the improving lane's halves of the row: one PRMT per two columns
#define ISH_H(j) ((j) < K ? H[(j) < K ? (j) : 0] : 0u)
      if (upA) {
#pragma unroll
        for (int v = 0; v < KP8 / 8; ++v)
          reinterpret_cast<uint4 *>(saveA)[v] =
              make_uint4(__byte_perm(ISH_H(8 * v), ISH_H(8 * v + 1), 0x5410),
                         __byte_perm(ISH_H(8 * v + 2), ISH_H(8 * v + 3), 0x5410),
                         __byte_perm(ISH_H(8 * v + 4), ISH_H(8 * v + 5), 0x5410),
                         __byte_perm(ISH_H(8 * v + 6), ISH_H(8 * v + 7), 0x5410));
      }
      if (upB) {
#pragma unroll
        for (int v = 0; v < KP8 / 8; ++v)
          reinterpret_cast<uint4 *>(saveB)[v] =
              make_uint4(__byte_perm(ISH_H(8 * v), ISH_H(8 * v + 1), 0x7632),
                         __byte_perm(ISH_H(8 * v + 2), ISH_H(8 * v + 3), 0x7632),
                         __byte_perm(ISH_H(8 * v + 4), ISH_H(8 * v + 5), 0x7632),
                         __byte_perm(ISH_H(8 * v + 6), ISH_H(8 * v + 7), 0x7632));
      }
#undef ISH_H
      if (upA) rowA = row;
      if (upB) rowB = row;
      best = ((upA ? cm : best) & 0xffffu) | ((upB ? cm : best) & 0xffff0000u);
      thr = nb;
    }
  };

  // Semi-global, target end free, one row: the running max of column Q-1
  // (register K-1 of thread G-1); a strict improvement records the row, so
  // the FIRST row of the maximum wins.
  auto te_row = [&](int row) {
    const uint32_t nb = __viaddmax_u16x2(H[K - 1], dup16(-frame_of(row)), best);
    if (nb != best) {
      if (lo16(nb) != lo16(best)) rowA = row;
      if (hi16(nb) != hi16(best)) rowB = row;
      best = nb;
    }
  };

  // o takes v's 16-bit half of each lane whose record ends now
  auto put_lanes = [](uint32_t &o, uint32_t v, bool a, bool b) {
    o = (a ? (v & 0xffffu) : (o & 0xffffu)) | (b ? (v & 0xffff0000u) : (o & 0xffff0000u));
  };

  // Outputs of the pair's record x (0: A, 1: B), written by thread G-1.
  auto put_out = [&](int x, uint32_t pr, int score, int eq, int er) {
    const uint32_t orig = p.rec.orig[p.first + 2 * pr + x];
    if (p.out.score) p.out.score[orig] = score;
    if (p.out.qend) p.out.qend[orig] = eq;
    if (p.out.tend) p.out.tend[orig] = er;
    if (p.out.hit) p.out.hit[orig] = decide(MODE, score, eq, er, p.dec);
  };
  const int last_off = (MODE == SG) ? p.bias + G * K * ext : 0;  // bias and frame of the last column

  // Semi-global with a free query end, at the last row of one or both records
  // (H holds it): fold the maximum of the last row left to right -- thread
  // t-1's partial arrived as iR at the start of this step, this thread's leaves
  // as oR at the next.
  auto qe_event = [&](int row, uint32_t ctl, uint32_t iR0, uint32_t iR1) {
    const bool lastA = row == lenA - 1, lastB = row == lenB - 1;
    int bA = 0, bB = 0, qA = 0x7fff, qB = 0x7fff;  // H + bias + row frame, above 0
    uint32_t row_h[K];  // staged: the loop indexes it
#pragma unroll
    for (int j = 0; j < K; ++j) row_h[j] = H[j];
#pragma unroll 1
    for (int j = 0; j < K; ++j) {
      if (col0 + j >= 0) {
        const int cf = (t * K + j + 1) * ext;
        const int a = ulo16(row_h[j]) - cf, b = uhi16(row_h[j]) - cf;
        if (a > bA) {
          bA = a;
          qA = col0 + j;
        }
        if (b > bB) {
          bB = b;
          qB = col0 + j;
        }
      }
    }
    if (t > 0) {  // columns to the left win ties
      if (!(bA > ulo16(iR0))) {
        bA = ulo16(iR0);
        qA = (int)(iR1 & 0xffffu);
      }
      if (!(bB > uhi16(iR0))) {
        bB = uhi16(iR0);
        qB = (int)(iR1 >> 16);
      }
    }
    if (t < G - 1) {
      put_lanes(oR0, (uint32_t)(bA & 0xffff) | ((uint32_t)bB << 16), lastA, lastB);
      put_lanes(oR1, (uint32_t)qA | ((uint32_t)qB << 16), lastA, lastB);
      return;
    }
    const uint32_t pr = slots[(ctl >> CTL_SEQ_SHIFT) & (G - 1)];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      if (!(x == 0 ? lastA : lastB)) continue;
      const int T = x == 0 ? lenA : lenB;
      int score = te ? (x == 0 ? ulo16(best) : uhi16(best)) - last_off : p.neg_limit;
      int er = x == 0 ? rowA : rowB, eq = p.Q - 1;
      const int s1 = (x == 0 ? bA : bB) - frame_of(row) - p.bias, t1 = x == 0 ? qA : qB;
      if (s1 > score) {
        score = s1;
        er = T - 1;
        eq = t1;
      } else if (s1 == score && er == T - 1 && t1 < eq) {
        eq = t1;
      }
      put_out(x, pr, score, eq, er);
    }
  };

  // Local alignment, after the step in which one or both records end: fold the
  // partial results left to right, as above.  Columns to the left win ties, so
  // the saved row is searched for its column only where this thread's best
  // beats the partial that came in.
  auto sw_event = [&](uint32_t ctl, uint32_t iR0, uint32_t iR1, uint32_t iR2, uint32_t iR3) {
    const bool lastA = (unsigned)(lenA - 1 - q4) < (unsigned)RPS, lastB = (unsigned)(lenB - 1 - q4) < (unsigned)RPS;
    int bA = lo16(iR0), bB = hi16(iR0), rA = (int)iR2, rB = (int)iR3;
    int qA = (int)(int16_t)(iR1 & 0xffffu), qB = (int)(int16_t)(iR1 >> 16);
    if (t == 0) {
      bA = bB = 0;
      rA = rB = -1;
      qA = qB = 0x7fff;
    }
    const int mA = ulo16(best) - p.bias, mB = uhi16(best) - p.bias;
    const bool ownA = lastA && (mA > bA || (mA == bA && mA > 0 && rowA < rA));
    const bool ownB = lastB && (mB > bB || (mB == bB && mB > 0 && rowB < rB));
    if (ownA) {
      bA = mA;
      rA = rowA;
    }
    if (ownB) {
      bB = mB;
      rB = rowB;
    }
    if (ownA || ownB) {  // smallest column of this thread's maximum in its first row
      const int sA = bA + p.bias, sB = bB + p.bias;
      const uint32_t *wa = reinterpret_cast<const uint32_t *>(saveA), *wb = reinterpret_cast<const uint32_t *>(saveB);
#pragma unroll 1
      for (int v = (K + 1) / 2 - 1; v >= 0; --v) {
        const uint32_t a = wa[v], b = wb[v];
        if (ownA && 2 * v + 1 < K && uhi16(a) == sA) qA = col0 + 2 * v + 1;
        if (ownA && ulo16(a) == sA) qA = col0 + 2 * v;
        if (ownB && 2 * v + 1 < K && uhi16(b) == sB) qB = col0 + 2 * v + 1;
        if (ownB && ulo16(b) == sB) qB = col0 + 2 * v;
      }
    }
    if (t < G - 1) {
      uint16_t *h = reinterpret_cast<uint16_t *>(partial);
      int *r = reinterpret_cast<int *>(partial);
      if (lastA) {
        h[0] = (uint16_t)bA;
        h[2] = (uint16_t)qA;
        r[2] = rA;
      }
      if (lastB) {
        h[1] = (uint16_t)bB;
        h[3] = (uint16_t)qB;
        r[3] = rB;
      }
      return;
    }
    const uint32_t pr = slots[(ctl >> CTL_SEQ_SHIFT) & (G - 1)];
    if (lastA) put_out(0, pr, bA, bA ? qA : 0, bA ? rA : -1);
    if (lastB) put_out(1, pr, bB, bB ? qB : 0, bB ? rB : -1);
  };

  // Every thread of the warp computes every step: an idle one (no record pair
  // in its pipeline slot) works on what its last pair left, whose lanes are
  // final, and a new pair resets all of its state.
  while (true) {
    __syncwarp();
    uint32_t msgH[RPS], msgF[RPS], msgB = 0, msgR = 0;
#pragma unroll
    for (int k = 0; k < RPS; ++k) {
      msgH[k] = __shfl_up_sync(FULL, outH[k], 1, G);
      msgF[k] = __shfl_up_sync(FULL, outF[k], 1, G);
    }
    if (MODE == SW) {
      msgB = __shfl_up_sync(FULL, outB, 1, G);
      msgR = __shfl_down_sync(FULL, __vmaxu2(best, right_best), 1, G);
    }
    uint32_t msgC = __shfl_up_sync(FULL, outC, 1, G);
    if (t0) msgC &= ~CTL_NEW;  // its own last control word
    // partial results of records that ended in thread t-1's previous step
    uint32_t iR0 = 0, iR1 = 0, iR2 = 0, iR3 = 0;
    if (MODE == SW) {
      if (ended) {
        if (t > 0) {
          const uint4 v = *(partial - save_stride);
          iR0 = v.x;
          iR1 = v.y;
          iR2 = v.z;
          iR3 = v.w;
        }
        __syncwarp();  // read before this step's ends rewrite them
      }
    } else if (qe && ended) {
      iR0 = __shfl_up_sync(FULL, oR0, 1, G);
      iR1 = __shfl_up_sync(FULL, oR1, 1, G);
    }
    q4 += RPS;
    // Everything beside the rows -- new pairs, frame resets, the look-ahead,
    // record ends -- happens in steps that some thread of the warp waits for,
    // so the others pay one comparison and one vote for all of it.
    bool endA = false, endB = false, ends = false;
    if (__any_sync(FULL, (msgC & CTL_NEW) || q4 == wake)) {
      if (t0 && q4 == end_q) {  // thread 0 of the group takes the next pair
        const uint32_t seq = (outC + (1u << CTL_SEQ_SHIFT)) & (31u << CTL_SEQ_SHIFT);
        msgC = seq | (f_next < npairs ? CTL_NEW : CTL_IDLE);
      }
      const bool fresh = msgC & CTL_NEW;
      if (fresh) q4 = 0;
      const auto at = [&](int r) { return (unsigned)(max(lenA, lenB) - q4 - r) < (unsigned)RPS; };
      if (fresh) {
        uint32_t pr = f_next * pstride + pphase;  // the pair's index in the range
        if (t0) {
          slots[(msgC >> CTL_SEQ_SHIFT) & (G - 1)] = pr;
        } else {
          pr = slots[(msgC >> CTL_SEQ_SHIFT) & (G - 1)];
        }
        const uint32_t sA = p.first + 2 * pr;
        lenA = (int)p.rec.len[sA];
        pa = p.rec.codes + p.rec.off[sA];
        if (2 * pr + 1 < p.count) {
          lenB = (int)p.rec.len[sA + 1];
          pb = p.rec.codes + p.rec.off[sA + 1];
        } else {
          lenB = 0;
          pb = pa;
        }
        if (t0) {
          end_q = (max(max(lenA, lenB), 1) + RPS - 1) & ~(RPS - 1);
          if (max(lenA, lenB) < CLAIM + RPS) f_next = claim();
        }
        nA = __ldg(reinterpret_cast<const uint32_t *>(pa));
        nB = lenB ? __ldg(reinterpret_cast<const uint32_t *>(pb)) : 0u;
        // row -1: H(-1, c) is 0 in the padding and with a free query start,
        // -open - ext * q else; with its frame c * ext (column frame less one
        // row's) that is bias + c * ext, or one value for all of the query
        if (MODE == SG) {
          const bool qs = p.ends & 1;
          const uint32_t step = qs ? (uint32_t)ext * 0x10001u : 0u;
          const uint32_t h0 = (uint32_t)(qs ? p.bias + t * K * ext : p.bias + p.d * ext - p.open) * 0x10001u;
#pragma unroll
          for (int j = 0; j < K; ++j) {
            H[j] = h0 + (uint32_t)j * step;
            E[j] = H[j] + EOPEN_SUM;  // row 0's frame is one ext above row -1's
          }
          prevH = h0 - step;
          if (!qs && t * K <= p.d) {  // (the padding is this thread's, or ends at its left)
#pragma unroll
            for (int j = -1; j < K; ++j) {
              const int c = t * K + j;
              if (c < p.d) {
                const uint32_t v = (uint32_t)(p.bias + c * ext) * 0x10001u;
                if (j < 0) {
                  prevH = v;
                } else {
                  H[j > 0 ? j : 0] = v;
                  E[j > 0 ? j : 0] = v + EOPEN_SUM;
                }
              }
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < K; ++j) H[j] = E[j] = FLOOR;
          prevH = FLOOR;
        }
        best = (MODE == SW) ? FLOOR : (t != G - 1 ? 0xffffffffu : 0u);
        left_best = FLOOR;
        rowA = rowB = -1;
      } else {
        if (MODE == SG && (q4 & fmask) == 0) {
          // frame R*ext -> 0: lower what this step takes from the row above
          // (values of row q4 - 1 in frame -ext: still non-negative halves)
          const uint32_t FRAME_DROP = p.pk_drop;
#pragma unroll
          for (int j = 0; j < K; ++j) {
            H[j] += FRAME_DROP;
            E[j] += FRAME_DROP;
          }
          prevH += FRAME_DROP;  // (thread 0's is set below)
        }
        // thread 0: the next pair is claimed, and what it needs first is
        // fetched into L1
        if (t0 && at(CLAIM)) f_next = claim();
        if (t0 && (at(LOOK_META) || at(LOOK_CODES)) && f_next < npairs) {
          const uint32_t sA = p.first + 2 * (f_next * pstride + pphase);
          if (at(LOOK_META)) {
            asm volatile("prefetch.global.L1 [%0];" ::"l"(p.rec.len + sA));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(p.rec.off + sA));
          } else {
            asm volatile("prefetch.global.L1 [%0];" ::"l"(p.rec.codes + p.rec.off[sA]));
            if (sA + 1 < p.first + p.count)
              asm volatile("prefetch.global.L1 [%0];" ::"l"(p.rec.codes + p.rec.off[sA + 1]));
          }
        }
      }
      // long records: the codes 256 rows ahead are pulled into L1, so the
      // group's loads hit L1 even when few warps are left to hide latency
      if (t0 && (q4 & 127) == 0) {
        if (q4 + 256 < lenA) asm volatile("prefetch.global.L1 [%0];" ::"l"(pa + q4 + 256));
        if (q4 + 256 < lenB) asm volatile("prefetch.global.L1 [%0];" ::"l"(pb + q4 + 256));
      }
      // whether a record of the warp ends in this step's rows (warp-uniform)
      endA = ends_here && (unsigned)(lenA - 1 - q4) < (unsigned)RPS;
      endB = ends_here && (unsigned)(lenB - 1 - q4) < (unsigned)RPS;
      ends = __any_sync(FULL, endA || endB);
      // the next step to wait for
      wake = 0x7fffffff;
      const auto wait_for = [&](int q) {
        if (q > q4) wake = min(wake, q);
      };
      if (MODE == SG) wait_for((q4 | fmask) + 1);
      if (ends_here) {
        wait_for((lenA - 1) & ~(RPS - 1));
        wait_for((lenB - 1) & ~(RPS - 1));
      }
      if (t0) {
        const int rows = max(lenA, lenB);
        wait_for(end_q);
        wait_for((rows - CLAIM) & ~(RPS - 1));
        wait_for((rows - LOOK_META) & ~(RPS - 1));
        wait_for((rows - LOOK_CODES) & ~(RPS - 1));
        if ((q4 | 127) + 256 < rows) wait_for((q4 | 127) + 1);
      }
    }
    ended = ends;
    outC = msgC;
    // ---- record codes of this step ----
    // Codes were checked against the alphabet when the set was loaded and
    // every record slot is zero-padded to 16 bytes.  Past a record's end the
    // last word repeats: those rows only feed a lane whose result is final.
    if (RPS == 4 || (q4 & 3) == 0) {
      wA = nA;
      wB = nB;
      if (q4 + 4 < lenA) nA = __ldg(reinterpret_cast<const uint32_t *>(pa + q4 + 4));
      if (q4 + 4 < lenB) nB = __ldg(reinterpret_cast<const uint32_t *>(pb + q4 + 4));
    } else {
      wA >>= 16;
      wB >>= 16;
    }
    // Codes that score alike share a profile row.  Mapped once per step: a test
    // in every row keeps the compiler from starting a row's loads in the row
    // above (38 columns, no mapping, 400,000 proteins: semi-global 6,440 -> 6,280
    // us, local 1 % on top of the wider bar's 1 %).
    if (remap && (RPS == 4 || (q4 & 3) == 0)) {
      const unsigned char *map = prof + remap_off;
      const auto rows_of = [&](uint32_t w) {
        return (uint32_t)map[w & 0xffu] | (uint32_t)map[(w >> 8) & 0xffu] << 8 |
               (uint32_t)map[(w >> 16) & 0xffu] << 16 | (uint32_t)map[w >> 24] << 24;
      };
      wA = rows_of(wA);
      wB = rows_of(wB);
    }
    // thread 0: what enters the padding from the left, H at its boundary (local:
    // the floor) and F below every value
    if (t0) {
      const uint32_t hf = MODE == SG ? LEFT0 + (uint32_t)(q4 & fmask) * LEFT_EXT : FLOOR;
      prevH = MODE == SG ? hf - LEFT_EXT : hf;
#pragma unroll
      for (int k = 0; k < RPS; ++k) {
        msgH[k] = MODE == SG ? hf + (uint32_t)k * LEFT_EXT : hf;
        msgF[k] = MODE == SG ? 0u : FLOOR + NOPEN_SUM;
      }
      msgB = FLOOR;
    }
    if (MODE == SG && qe && ends) {
      // ---- free query end, a record of the warp ends: one row at a time, with
      // the last row's maximum taken after it ----
      uint32_t d = prevH, sA = wA, sB = wB;
#pragma unroll 1
      for (int k = 0; k < RPS; ++k) {
        const int row = q4 + k;
        const uint32_t fs = row_step(sA & 0xffu, sB & 0xffu, d, msgF[0]);
        sA >>= 8;
        sB >>= 8;
        d = msgH[0];
#pragma unroll
        for (int j = 0; j + 1 < RPS; ++j) {
          msgH[j] = msgH[j + 1];
          msgF[j] = msgF[j + 1];
          outH[j] = outH[j + 1];
          outF[j] = outF[j + 1];
        }
        outH[RPS - 1] = H[K - 1];
        outF[RPS - 1] = fs;
        if (te) te_row(row);
        if (row == lenA - 1 || row == lenB - 1) qe_event(row, msgC, iR0, iR1);
      }
      prevH = d;
    } else {
      // ---- the step's rows ----
      // (local alignment; in a pair's first two steps the next thread's word is
      // still of the pair before)
      if (MODE == SW) right_best = t == G - 1 || q4 < 2 * RPS ? 0u : msgR;
      uint32_t thr = MODE == SW ? __vimax3_u16x2(best, left_best, right_best) : 0u;
#pragma unroll
      for (int k = 0; k < RPS; ++k) {
        const uint32_t fs = row_step(__byte_perm(wA, 0u, 0x4440 + k), __byte_perm(wB, 0u, 0x4440 + k),
                                     k == 0 ? prevH : msgH[k - 1], msgF[k]);
        outH[k] = H[K - 1];
        outF[k] = fs;
        if (MODE == SW) {
          uint32_t live = 0xffffffffu;  // a record that ended in this step has no further rows
          if (k > 0 && ends) live = (q4 + k >= lenA ? 0u : 0xffffu) | (q4 + k >= lenB ? 0u : 0xffff0000u);
          sw_track(q4 + k, thr, live);
        }
      }
      prevH = msgH[RPS - 1];
      if (MODE == SW) {
        outB = __vmaxu2(best, msgB);
        left_best = msgB;
        if (endA || endB) sw_event(msgC, iR0, iR1, iR2, iR3);
      } else if (!ends) {
        if (te) {
          // the largest H(., Q-1) of the step's rows without their frames
          // (frame(q4 + k) = frame(q4) + k * ext): m = max_k outH[k] - k * ext
          uint32_t m = outH[RPS - 1];
#pragma unroll
          for (int k = RPS - 2; k >= 0; --k) m = __viaddmax_u16x2(m, NEXT, outH[k]);
          const uint32_t nb = __viaddmax_u16x2(m, dup16(-frame_of(q4)), best);
          if (nb != best) {
            // the first row reaching the new maximum, per improved lane
            bool dA = lo16(nb) == lo16(best), dB = hi16(nb) == hi16(best);
#pragma unroll
            for (int k = 0; k < RPS; ++k) {
              const uint32_t u = __viaddmax_u16x2(outH[k], dup16(-frame_of(q4 + k)), 0u);
              if (!dA && lo16(u) == lo16(nb)) {
                rowA = q4 + k;
                dA = true;
              }
              if (!dB && hi16(u) == hi16(nb)) {
                rowB = q4 + k;
                dB = true;
              }
            }
            best = nb;
          }
        }
      } else if (t == G - 1) {
        // a record of the warp ends: row by row, this thread's records up to
        // their last row, then their outputs
        int sA = 0, sB = 0;
#pragma unroll
        for (int k = 0; k < RPS; ++k) {
          const uint32_t u = __viaddmax_u16x2(outH[k], dup16(-frame_of(q4 + k)), 0u);
          const bool inA = q4 + k < lenA, inB = q4 + k < lenB;
          if (inA) sA = ulo16(u);
          if (inB) sB = uhi16(u);
          if (te && inA && ulo16(u) > ulo16(best)) {
            best = (best & 0xffff0000u) | (u & 0xffffu);
            rowA = q4 + k;
          }
          if (te && inB && uhi16(u) > uhi16(best)) {
            best = (best & 0xffffu) | (u & 0xffff0000u);
            rowB = q4 + k;
          }
        }
        if (endA || endB) {
          const uint32_t pr = slots[(msgC >> CTL_SEQ_SHIFT) & (G - 1)];
          if (endA) put_out(0, pr, (te ? ulo16(best) : sA) - last_off, p.Q - 1, te ? rowA : lenA - 1);
          if (endB) put_out(1, pr, (te ? uhi16(best) : sB) - last_off, p.Q - 1, te ? rowB : lenB - 1);
        }
      }
    }

    // Every step thread 0 starts reaches thread G-1 within G-1 steps, and thread
    // 0 idles only when no pair is left, so the group is done once all of its
    // threads idle.  The step budget
    // (all rows of the range plus the pipeline depth) is a hard stop.
    // (checked every CHK steps; idle extra steps do nothing)
    if ((++step & (CHK - 1)) == 0) {
      if (!__any_sync(FULL, !(outC & CTL_IDLE))) break;
      if (step / CHK > p.max_steps / (CHK * RPS)) {
        if (lane == 0) atomicOr(p.error, 2);
        break;
      }
    }
  }
}

// Rows with the parameters read from a shared-memory copy, as the batched
// kernel does: kept in the parameter bank, the compiler holds them in
// registers across the row loop, which some shapes pay for in spills
// (WAVE_PARAMS_SMEM).  Only the kernels that call this declare the copy.
template <int K, int MODE, int LAYOUT>
__device__ __forceinline__ void wave_rows_smem_params(const WaveParams &p, const unsigned char *prof,
                                                      uint32_t *slots_all, uint32_t *save_all) {
  __shared__ WaveParams sp;
  if (threadIdx.x == 0) sp = p;
  __syncthreads();
  wave_rows<K, MODE, LAYOUT, true>(sp, prof, slots_all, save_all, p.counter);
}

// Copies a query's profile to shared memory (the caller's barrier follows).  All
// of a thread's copies are in flight at once: a one-warp block of a small call
// loads 40 KB in 80 of them, which took longer than its rows when each batch of
// four loads was waited for (500 lines in one call: 126 -> 117 us).
__device__ __forceinline__ void load_profile(unsigned char *smem, const uint4 *src, uint32_t bytes) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
  for (uint32_t i = threadIdx.x; i < bytes >> 4; i += blockDim.x)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 16), "l"(src + i) : "memory");
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Shared memory of a block: the profile, then a slot word per thread, then
// (local alignment) wave_save_words(K) save words per thread.
template <int K, int MODE, int LAYOUT, int LEAN = 0>
__global__ void __launch_bounds__(wave_sm_threads(K, LEAN), 1)
    wave_kernel(const __grid_constant__ WaveParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  load_profile(smem_raw, p.prof, p.prof_bytes);
  uint32_t *slots_all = reinterpret_cast<uint32_t *>(smem_raw + ((p.prof_bytes + 15u) & ~15u));
  uint32_t *save_all = slots_all + blockDim.x;
  if constexpr (WAVE_PARAMS_SMEM(K, MODE, LEAN)) {
    wave_rows_smem_params<K, MODE, LAYOUT>(p, smem_raw, slots_all, save_all);
  } else {
    __syncthreads();
    wave_rows<K, MODE, LAYOUT, true>(p, smem_raw, slots_all, save_all, p.counter);
  }
}

// The batched launch: one persistent kernel for every query of a shape class
// (same K, mode and profile layout; G may differ per query).  Each query's
// record pairs are handed out by its own counter in global memory, in
// descending length order, exactly as in wave_kernel.  A block walks the
// queries of the class starting at its own offset (so the blocks spread over
// the queries) and stays on a query until its counter runs dry; a barrier and
// a profile reload happen only at a query switch, where the pairs left are the
// shortest of the set.  Queries whose counter is already exhausted are skipped.
template <int K, int MODE, int LAYOUT, int LEAN = 0>
__global__ void __launch_bounds__(wave_sm_threads(K, LEAN), 1)
    batch_kernel(const __grid_constant__ BatchParams b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ WaveParams sp;
  __shared__ int s_skip;
  uint32_t *slots_all = reinterpret_cast<uint32_t *>(smem_raw + b.prof_area);
  uint32_t *save_all = slots_all + blockDim.x;
  const uint32_t start = (uint32_t)(((uint64_t)blockIdx.x * b.ntiles) / gridDim.x);
  for (uint32_t it = 0; it < b.ntiles; ++it) {
    uint32_t tile = start + it;
    if (tile >= b.ntiles) tile -= b.ntiles;
    const BatchTile tl = b.tiles[tile];
    const WaveParams *qp = b.queries + tl.q;
    uint32_t *counter = b.tile_counter + tile;
    if (threadIdx.x == 0) {
      const uint32_t taken = *reinterpret_cast<volatile uint32_t *>(counter);
      const uint32_t stride = tl.pairs >> 16, phase = tl.pairs & 0xffffu, all = (tl.count + 1) / 2;
      const uint32_t mine = stride ? (all > phase ? (all - phase + stride - 1) / stride : 0u) : all;
      s_skip = taken >= mine;
      if (!s_skip) {
        sp = *qp;
        sp.first = tl.first;
        sp.count = tl.count;
        sp.pair_stride = stride;
        sp.pair_phase = phase;
        // every group's steps are bounded by all pairs of the range at its
        // longest length (records are sorted, the first is longest to within a
        // bucket; the last bucket holds any length from its own on)
        const uint64_t npairs = (tl.count + 1) / 2, first = qp->rec.len[tl.first];
        const uint64_t most = first < LAST_BUCKET_LEN ? first : 0xffffffffu;
        sp.max_steps = b.step_cap ? b.step_cap : npairs * (most + 2 * 32 + 8) + 1024;
      }
    }
    __syncthreads();
    if (s_skip) {
      __syncthreads();  // s_skip is rewritten next iteration
      continue;
    }
    load_profile(smem_raw, qp->prof, qp->prof_bytes);
    __syncthreads();
    wave_rows<K, MODE, LAYOUT, false>(sp, smem_raw, slots_all, save_all, counter);
    __syncthreads();
  }
}

}  // namespace ish

namespace ish {

// Kernel tables.  Each wave_X.cu instantiates the wavefront and batched
// kernels of one K range (one translation unit per range, so the build
// compiles them in parallel); wave_table / batch_table pick one at run time
// by (K, mode, profile layout).
template <int K, int LEAN>
struct WaveEntry {
  static WaveFn wave(int mode, int layout) {
    static const WaveFn t[2][3] = {
        {wave_kernel<K, SG, PROF_S16, LEAN>, wave_kernel<K, SG, PROF_PAIR, LEAN>, wave_kernel<K, SG, PROF_S32, LEAN>},
        {wave_kernel<K, SW, PROF_S16, LEAN>, wave_kernel<K, SW, PROF_PAIR, LEAN>, wave_kernel<K, SW, PROF_S32, LEAN>}};
    return t[mode == SW][layout];
  }
  static BatchFn batch(int mode, int layout) {
    static const BatchFn t[2][3] = {
        {batch_kernel<K, SG, PROF_S16, LEAN>, batch_kernel<K, SG, PROF_PAIR, LEAN>,
         batch_kernel<K, SG, PROF_S32, LEAN>},
        {batch_kernel<K, SW, PROF_S16, LEAN>, batch_kernel<K, SW, PROF_PAIR, LEAN>,
         batch_kernel<K, SW, PROF_S32, LEAN>}};
    return t[mode == SW][layout];
  }
};

template <int LEAN, int... Ks>
WaveFn wave_table(int K, int mode, int layout) {
  if (layout < PROF_S16 || layout > PROF_S32) return nullptr;
  WaveFn f = nullptr;
  ((K == Ks ? (void)(f = WaveEntry<Ks, LEAN>::wave(mode, layout)) : (void)0), ...);
  return f;
}

template <int LEAN, int... Ks>
BatchFn batch_table(int K, int mode, int layout) {
  if (layout < PROF_S16 || layout > PROF_S32) return nullptr;
  BatchFn f = nullptr;
  ((K == Ks ? (void)(f = WaveEntry<Ks, LEAN>::batch(mode, layout)) : (void)0), ...);
  return f;
}

}  // namespace ish
