// kernels.cuh -- declarations shared by the kernel translation units and the
// host engine.
#pragma once

#include "engine.cuh"

namespace ish {

constexpr uint32_t NBUCKETS = 65536;     // length buckets of the record sort
constexpr uint32_t LAST_BUCKET_LEN = 32768 + 32 * (NBUCKETS - 1 - 32768);  // lengths from here on share one
constexpr uint32_t SCAN_TILE = 4096;     // values per block of k_scan64_block (1024 threads)
constexpr uint32_t HIT_TILE = 8192;      // records per block of the hit compaction
constexpr uint32_t SMEM_BUCKETS = 4096;  // length buckets counted in shared memory by k_lengths / k_scatter

constexpr uint32_t LINE_TILE = 65536;    // text bytes per block of the line splitter
__global__ void k_zero2(uint32_t *a, uint32_t na, uint32_t *b, uint32_t nb);
__global__ void k_lengths(const uint64_t *off, const uint64_t *end, uint32_t n, uint32_t *len, uint64_t *tile_sum,
                          uint32_t *hist, uint32_t *max_bucket, uint32_t *summary);
__global__ void k_scan_slots(const uint32_t *len, uint32_t n, const uint64_t *tile_sum, uint64_t *poff);
constexpr uint32_t BUCKET_BLOCKS = NBUCKETS / 1024;  // blocks of the bucket cursor kernel
__global__ void k_bucket_cursors(const uint32_t *hist, const uint32_t *max_bucket, uint32_t *cursor,
                                 uint32_t *summary);
__global__ void k_scatter(const uint32_t *len, const uint64_t *poff, uint32_t n, uint32_t *cursor, uint32_t *len_s,
                          uint64_t *off_s, uint32_t *orig_s, uint32_t *hist, uint32_t *max_bucket,
                          const uint32_t *summary);
constexpr uint32_t SORT_SMALL = 4096;    // records that k_sort_small takes
__global__ void k_sort_small(uint64_t *off, uint32_t n, uint64_t base, uint64_t *poff, uint32_t *len_s,
                             uint64_t *off_s, uint32_t *orig_s, uint32_t *long_counter, uint32_t *max_code);
typedef void (*PackFn)(const uint8_t *src, uint64_t src_bytes, const uint64_t *off, const uint64_t *end,
                       const uint64_t *poff, uint32_t n, const uint32_t *len_s, const uint32_t *orig_s,
                       uint32_t *long_counter, const uint8_t *enc, uint8_t *dst, uint32_t *max_code, uint32_t gw,
                       uint32_t limit);
PackFn pack_fn(bool limited);
__global__ void k_count_newlines(const uint8_t *text, uint64_t bytes, uint32_t *block_counts);
// k_write_newlines<headers>: with headers, also the first '>' or '@' of every
// line (hc, preset to all ones)
typedef void (*NewlinesFn)(const uint8_t *text, uint64_t bytes, const uint32_t *block_offsets, uint64_t *pos,
                           unsigned long long *hc);
NewlinesFn write_newlines_fn(bool headers);
__global__ void k_line_bounds(const uint8_t *text, uint64_t bytes, const uint64_t *nl, uint32_t n_nl, uint32_t n_lines,
                              uint64_t *start, uint64_t *end, unsigned long long *total);
__global__ void k_scan64_block(const uint64_t *in, uint64_t *out, uint32_t n, uint64_t *block_sums);
__global__ void k_scan64_add(uint64_t *out, uint32_t n, const uint64_t *block_offsets);
__global__ void k_trivial(RecordsDev rec, uint32_t first, uint32_t count, int mode, int qlen, OutDev out, Decision dec);
typedef void (*PlainFn)(const PlainParams);
// plain_kernel<mode, qmax>: qmax 0 (int32 columns in global scratch) or a
// power of two 64..2048 (int16 per-thread columns); nullptr otherwise
PlainFn plain_fn(int mode, int qmax);
constexpr int PLAIN16_QMAX = 2048;     // longest query of the int16 plain kernel
constexpr int PLAIN16_THREADS = 15000; // its launch: 15,000 threads in blocks of 32
__global__ void k_count_hits(const uint8_t *hit, uint32_t n, uint32_t *block_counts);
__global__ void k_scan_counts(uint32_t *counts, uint32_t nb, uint32_t *total);
__global__ void k_dpx_peak(uint32_t *out, int iters, uint32_t b, uint32_t c);
// k_lane_rows<u8>: local-alignment rows on 2 x 16-bit or 4 x 8-bit lanes
// (ish_gpu_calibrate_lanes)
typedef void (*LaneFn)(uint32_t *out, int rows, uint32_t p0, uint32_t popen, uint32_t pext, uint32_t bias);
LaneFn lane_rows_fn(bool u8);
__global__ void k_write_hits(const uint8_t *hit, uint32_t n, const uint32_t *block_offsets, uint32_t *idx);
constexpr uint32_t COMPACT_ONE = 16384;  // records that k_compact_one takes
// The results of a call on up to SORT_SMALL records in pinned host memory: three
// counts of k_compact_one, then scores, query ends, target ends, hit indices
// (SORT_SMALL words each) and hit flags.  The six copies it replaces cost a call
// more than the bytes: 500 lines 116 -> 109 us, 3,000 proteins with match starts
// 825 -> 781 (their arrays are pageable, whose copies the driver stages one by
// one).
struct StageOut {
  uint32_t *to = nullptr;
  const int32_t *from[3] = {nullptr, nullptr, nullptr};  // scores, query ends, target ends on the device (null: not wanted)
  bool hit = false;                                      // the flags are wanted
};
constexpr uint32_t STAGE_HEAD = 4, STAGE_WORDS = STAGE_HEAD + 4 * SORT_SMALL + SORT_SMALL / 4;
__global__ void k_compact_one(const uint8_t *hit, uint32_t n, uint32_t *idx, const int *error,
                              const uint32_t *max_code, uint32_t *out, StageOut stage);
__global__ void k_write_hits_sum(const uint8_t *hit, uint32_t n, const uint32_t *block_counts, uint32_t *idx,
                                 const int *error, uint32_t *out);
__global__ void k_gather_hits(const uint32_t *idx, const uint32_t *count, const int32_t *score, const int32_t *qend,
                              const int32_t *tend, int32_t *hit_score, int32_t *hit_qend, int32_t *hit_tend);

// Rows a wavefront thread computes per pipeline step.  A record's codes arrive
// four to a 32-bit word, and everything beside the recurrence itself -- the
// pipeline shuffles and control word, thread 0's work grab, the code refill,
// the frame reset, the end-of-record test and the target-end maximum -- runs
// once per step instead of once per row.  A pair's rows are rounded up to a
// multiple of the rows per step (the rows past both records' ends feed nothing).
// Semi-global row frames reset only at step boundaries, so the fast regime
// keeps R >= WAVE_RPS_SG rows per frame period (gap_extend <= 512 at 4).
// Four for local alignment too: its carried dominance bar is one word per step,
// so four rows cost no more registers than two (protein, 8 threads x 38
// columns: 5,573 GCUPS against 5,302 with two).
#ifndef WAVE_RPS_SG
#define WAVE_RPS_SG 4
#endif
#ifndef WAVE_RPS_SW
#define WAVE_RPS_SW 4
#endif

// Wavefront kernels are instantiated for K = 1..32 and even K up to WAVE_KMAX
// columns per thread, both modes and the three profile layouts.
constexpr int WAVE_KMAX = 64;
// Threads an SM holds (the register budget): 512 up to K = 32 columns per
// thread (128 registers), 384 up to K = 48 (168), 256 above.  Register-lean
// builds trade warps for registers per thread: 384 threads for 25 <= K <= 32 and
// 256 for 34 <= K <= 48.  Which build runs is chosen per (K, mode) from
// measurements (wave_lean, lean_for).  The launch bound is one block of all of
// them, so the host may launch them as one block that shares one profile
// (launch_wave_range), or as smaller ones (batch_launch).
constexpr int WAVE_LEAN_KMIN = 25, WAVE_LEAN_KMAX = 48;
__host__ __device__ constexpr bool wave_has_lean(int K) { return K >= WAVE_LEAN_KMIN && K <= WAVE_LEAN_KMAX && K != 33; }
__host__ __device__ constexpr int wave_sm_threads(int K, int lean) {
  return lean && wave_has_lean(K) ? (K <= 32 ? 384 : 256) : (K <= 32 ? 512 : K <= 48 ? 384 : 256);
}
// wave_kernel reads its parameters from a shared-memory copy for these (K, mode,
// lean build) (see wave.cuh).  Against the parameter bank, on 200,000 proteins (G =
// 8 and 16) and 200,000 reads of 150 (G = 4 and 8): semi-global 0 to +4 % at K =
// 10..48 with few exceptions (K = 26 with the 32-bit profile +32 %, K = 27 -4 %, K =
// 36 with the pair profile -5 %), -1 to +4 % from K = 58 on, and level or behind on
// reads at the K left out; local -5 to +2 % (K = 38 of the protein search +2 %, the
// mean -1 %), where the copy stays as it was set for rows that needed it.
#ifndef WAVE_PARAMS_SMEM
#define WAVE_PARAMS_SMEM(K, MODE, LEAN)                                              \
  (((MODE) == 0 && (K) >= 9 && (K) <= 32) || ((MODE) == 1 && (K) >= 12 && (K) <= 32) || \
   (!(LEAN) && (K) >= 34 && (K) <= 48) || (K) >= 58 || ((MODE) == 1 && (K) == 50))
#endif
// Local alignment keeps, per thread, the H row of each lane's last
// improvement as 16-bit values: two arrays of K (rounded up to 8) halves,
// strided by an odd number of 16-byte units.
__host__ __device__ constexpr int wave_save_words(int K) { return ((((K + 7) & ~7) / 4) | 1) * 4; }
typedef void (*WaveFn)(const WaveParams);
// Returns the kernel for (K, mode, profile layout, lean variant) or nullptr.
WaveFn wave_fn(int K, int mode, int layout, int lean = 0);
typedef void (*BatchFn)(const BatchParams);
BatchFn batch_fn(int K, int mode, int layout, int lean = 0);  // batch_kernel<K, mode, layout, lean> or nullptr

// The splitting kernels take the text in tiles of LINE_TILE bytes per
// 1024-thread block; warp w of a block covers LINE_WARP consecutive bytes of
// its tile, 512 per step and 16 per lane, all of them loaded before any is
// looked at (they are bound by the loads in flight), and no block-wide barrier
// runs inside a loop.  The text lies in a buffer with at least 15 bytes of slack
// past its end (every 16-byte word that starts inside it can be loaded) and
// starts 16-byte aligned.
constexpr uint32_t LINE_WARP = LINE_TILE / 32, LINE_STEPS = LINE_WARP / 512;

// Bit k set where byte k of the 16 in w is c (four times in c4).
__device__ __forceinline__ uint32_t byte_bits(const uint4 &w, uint32_t c4) {
  const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t t = ww[k] ^ c4;  // a zero byte where equal
    const uint32_t z = ~(((t & 0x7f7f7f7fu) + 0x7f7f7f7fu) | t) & 0x80808080u;
    m |= (((z >> 7) * 0x01020408u) >> 24 & 0xfu) << (4 * k);  // bits 0, 8, 16, 24 to 0..3
  }
  return m;
}
// The bits of the 16 bytes from byte i that lie inside the text.
__device__ __forceinline__ uint32_t inside_bits(uint64_t bytes, uint64_t i) {
  return i >= bytes ? 0u : bytes - i >= 16 ? 0xffffu : (1u << (uint32_t)(bytes - i)) - 1u;
}
// This lane's words of the warp's segment starting at byte w0 (zero past the text).
__device__ __forceinline__ void load_segment(const uint8_t *text, uint64_t bytes, uint64_t w0, uint32_t lane,
                                             uint4 (&w)[LINE_STEPS]) {
#pragma unroll
  for (uint32_t k = 0; k < LINE_STEPS; ++k) {
    const uint64_t i = w0 + k * 512 + lane * 16;
    w[k] = i < bytes ? __ldg(reinterpret_cast<const uint4 *>(text + i)) : make_uint4(0, 0, 0, 0);
  }
}

}  // namespace ish
