// kernels.cu -- record packing, the plain one-thread-per-record kernel and
// the epilogue kernels of the GB300 alignment-scoring engine.
#include "kernels.cuh"

namespace ish {

// ---------------------------------------------------------------------------
// Record packing.  The caller's records arrive as one concatenated byte array
// plus n+1 offsets (what ish's runners accumulate per batch,
// ishlib/parallel_line_search_runner.mojo:84-111).  On the device each record
// is copied to a 16-byte aligned slot (so the wavefront feeder can stream it
// with 16-byte loads) and the records are ordered by descending length, so
// that the two records of a pair have nearly the same length and the longest
// pairs start first.
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t len_bucket(uint64_t len) {
  // exact below 32768, 32-residue resolution above (records up to ~1 Mb)
  if (len < 32768) return (uint32_t)len;
  uint64_t b = 32768 + ((len - 32768) >> 5);
  return b > NBUCKETS - 1 ? NBUCKETS - 1 : (uint32_t)b;
}

// Record i is src[off[i] .. end[i]) when `end` is given, else
// src[off[i] .. off[i + 1]) (one concatenated array).
__device__ __forceinline__ uint64_t rec_len(const uint64_t *off, const uint64_t *end, uint32_t i) {
  return (end ? end[i] : off[i + 1]) - off[i];
}

// The packing kernels below run in this order on one stream: k_lengths,
// k_scan_slots, k_bucket_cursors, k_scatter, k_pack.  The accumulators they
// share between loads -- the length histogram `hist` and the largest length
// bucket `max_bucket` -- are zero when a load starts and are zeroed again by
// k_scatter, their last reader, so a load needs no separate clearing pass;
// what the host reads back goes to `summary` = {largest code, largest
// bucket, per-bucket record counts}.  (The host clears the accumulators with
// k_zero2 after a load that stopped half way.)
__global__ void k_zero2(uint32_t *a, uint32_t na, uint32_t *b, uint32_t nb) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < na + nb; i += gridDim.x * blockDim.x) {
    if (i < na) a[i] = 0;
    else b[i - na] = 0;
  }
}

// Per record: its length; per tile of SCAN_TILE records (one 1024-thread
// block, four consecutive records per thread): the sum of the 16-byte slot
// sizes; and the length histogram.  The buckets below SMEM_BUCKETS are counted
// in shared memory and flushed once per block (a set's lengths crowd into a few
// hundred buckets, and one global atomic per record on those few addresses
// would serialise); longer records go to the global histogram directly.
__global__ void __launch_bounds__(1024) k_lengths(const uint64_t *off, const uint64_t *end, uint32_t n, uint32_t *len,
                                                  uint64_t *tile_sum, uint32_t *hist, uint32_t *max_bucket,
                                                  uint32_t *summary) {
  __shared__ uint32_t sh[SMEM_BUCKETS];
  __shared__ uint64_t wsum[32];
  for (uint32_t k = threadIdx.x; k < SMEM_BUCKETS; k += blockDim.x) sh[k] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) summary[0] = 0;  // largest code, raised by k_pack
  __syncthreads();
  constexpr int PER = SCAN_TILE / 1024;
  uint32_t mb = 0;
  uint64_t slots = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const uint32_t i = blockIdx.x * SCAN_TILE + threadIdx.x * PER + k;
    if (i < n) {
      const uint64_t l = rec_len(off, end, i);
      len[i] = (uint32_t)l;
      slots += (l + 15) & ~(uint64_t)15;
      const uint32_t b = len_bucket(l);
      if (b < SMEM_BUCKETS) atomicAdd(&sh[b], 1u);
      else atomicAdd(&hist[b], 1u);
      mb = max(mb, b);
    }
  }
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) {
    mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    slots += __shfl_xor_sync(0xffffffffu, slots, o);
  }
  if (lane == 0) {
    if (mb) atomicMax(max_bucket, mb);
    wsum[wid] = slots;
  }
  __syncthreads();
  if (wid == 0) {
    uint64_t t = wsum[lane];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) tile_sum[blockIdx.x] = t;
  }
  for (uint32_t k = threadIdx.x; k < SMEM_BUCKETS; k += blockDim.x)
    if (sh[k]) atomicAdd(&hist[k], sh[k]);
}

// Packed offset of every record: the exclusive scan of the 16-byte slot sizes
// in record order.  Block b scans tile b and adds the slots of the tiles
// before it (at most SCAN_TILE tile sums, summed by the block itself), so one
// pass does what a scan of tile sums and an add pass would.
__global__ void __launch_bounds__(1024) k_scan_slots(const uint32_t *len, uint32_t n, const uint64_t *tile_sum,
                                                     uint64_t *poff) {
  __shared__ uint64_t warp_sums[32];
  __shared__ uint64_t before;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // slots of the earlier tiles
  uint64_t e = 0;
  for (uint32_t t = tid; t < blockIdx.x; t += blockDim.x) e += tile_sum[t];
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if (lane == 0) warp_sums[wid] = e;
  __syncthreads();
  if (wid == 0) {
    uint64_t w = warp_sums[lane];
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (lane == 0) before = w;
  }
  __syncthreads();
  constexpr int PER = SCAN_TILE / 1024;
  const uint32_t base = blockIdx.x * SCAN_TILE + tid * PER;
  uint64_t v[PER], sum = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    v[k] = base + k < n ? ((uint64_t)len[base + k] + 15) & ~(uint64_t)15 : 0;
    sum += v[k];
  }
  uint64_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;  // the earlier reads of warp_sums ended at the barrier above
  __syncthreads();
  if (wid == 0) {
    uint64_t w = warp_sums[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  uint64_t run = before + x - sum + (wid > 0 ? warp_sums[wid - 1] : 0);
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    if (base + k < n) poff[base + k] = run;
    run += v[k];
  }
}

// First sorted position of every length bucket, buckets in DESCENDING order
// (longest records first): block b covers the descending positions
// [b*1024, b*1024 + 1024), i.e. buckets NBUCKETS-1-(b*1024+t), so its loads
// are coalesced, and adds the records of the positions before it that can
// hold any (buckets up to the set's largest).  Blocks whose buckets all lie
// above the largest hold no records and stop at once.  The counts and the
// largest bucket are copied to `summary` for the host.
__global__ void __launch_bounds__(1024) k_bucket_cursors(const uint32_t *hist, const uint32_t *max_bucket,
                                                         uint32_t *cursor, uint32_t *summary) {
  __shared__ uint32_t warp_incl[32];
  __shared__ uint32_t base;
  const uint32_t b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t maxb = *max_bucket;
  if (b == 0 && tid == 0) summary[1] = maxb;
  if (NBUCKETS - 1024 * (b + 1) > maxb) return;  // the block's smallest bucket is above the largest used
  // records at the descending positions [lo, b*1024): buckets maxb down to the block's first
  const uint32_t lo = NBUCKETS - 1 - maxb;
  uint32_t e = 0;
  for (uint32_t p = lo + tid; p < b * 1024; p += 1024) e += hist[NBUCKETS - 1 - p];
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if (lane == 0) warp_incl[warp] = e;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = warp_incl[lane];
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (lane == 0) base = w;
  }
  __syncthreads();
  const uint32_t bucket = NBUCKETS - 1 - (b * 1024 + tid);
  const uint32_t c = hist[bucket];
  summary[2 + bucket] = c;
  uint32_t incl = c;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += x;
  }
  if (lane == 31) warp_incl[warp] = incl;  // the reads of warp_incl above ended at the barrier
  __syncthreads();
  if (warp == 0) {
    uint32_t w = warp_incl[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= (uint32_t)o) w += x;
    }
    warp_incl[lane] = w;
  }
  __syncthreads();
  const uint32_t before_warp = warp ? warp_incl[warp - 1] : 0u;
  cursor[bucket] = base + before_warp + incl - c;
}

// Sorted position of every record: record i goes to the next free place of
// its bucket.  Each block takes 1024 records (one per thread, 1024 threads),
// ranks them within their bucket in shared memory, reserves one range per
// used bucket from the global cursor and writes; buckets from SMEM_BUCKETS on
// (long records, few) take one global atomic per record.  The order within a
// bucket is unspecified: the two lanes of a pair are scored independently.
// The kernel also zeroes the histogram (buckets up to the largest, the only
// ones that can be non-zero) and the largest bucket for the next load, and
// the long-record counter that k_pack takes next (max_bucket[1]).
__global__ void __launch_bounds__(1024) k_scatter(const uint32_t *len, const uint64_t *poff, uint32_t n,
                                                  uint32_t *cursor, uint32_t *len_s, uint64_t *off_s,
                                                  uint32_t *orig_s, uint32_t *hist, uint32_t *max_bucket,
                                                  const uint32_t *summary) {
  __shared__ uint32_t sh[SMEM_BUCKETS];  // counts, then the block's first position per bucket
  for (uint32_t k = threadIdx.x; k < SMEM_BUCKETS; k += blockDim.x) sh[k] = 0;
  const uint32_t maxb = summary[1];
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k <= maxb; k += gridDim.x * blockDim.x) hist[k] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    max_bucket[0] = 0;  // for the next load
    max_bucket[1] = 0;  // k_pack's long-record counter, for this load
  }
  __syncthreads();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t l = 0, b = 0, rank = 0;
  if (i < n) {
    l = len[i];
    b = len_bucket(l);
    if (b < SMEM_BUCKETS) rank = atomicAdd(&sh[b], 1u);
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < SMEM_BUCKETS; k += blockDim.x) {
    const uint32_t c = sh[k];
    if (c) sh[k] = atomicAdd(&cursor[k], c);
  }
  __syncthreads();
  if (i < n) {
    const uint32_t pos = b < SMEM_BUCKETS ? sh[b] + rank : atomicAdd(&cursor[b], 1u);
    len_s[pos] = l;
    off_s[pos] = poff[i];
    orig_s[pos] = i;
  }
}

// Sets of at most SORT_SMALL records: lengths, packed offsets and sorted
// positions in one block, where the four kernels above spend most of their time
// being launched; what the host needs to know of the set (its histogram) it has
// counted from its own offsets.  Each thread holds four consecutive keys
// (longest bucket first, then record order) of a bitonic network: steps of 1
// and 2 stay in the thread, of 4 to 64 in the warp, and only those from 128 (15
// of 78 at 4,096 records) meet at a barrier.  The block has a quarter of the
// next power of two in threads.  Rebases off by `base` for k_pack.  (The whole
// load of 500 lines 60 us -> 51 with it and one stream, one synchronisation
// less; a network in shared memory alone took 23 us longer at 3,000 proteins.)
__global__ void __launch_bounds__(1024) k_sort_small(uint64_t *off, uint32_t n, uint64_t base, uint64_t *poff,
                                                     uint32_t *len_s, uint64_t *off_s, uint32_t *orig_s,
                                                     uint32_t *long_counter, uint32_t *max_code) {
  __shared__ uint4 cross[2][SORT_SMALL / 4];
  __shared__ uint64_t warp_sums[32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, e0 = tid * 4;
  if (tid == 0) *long_counter = *max_code = 0;
  uint64_t o[5], sum = 0;
  uint32_t v[4];
#pragma unroll
  for (int k = 0; k < 5; ++k) o[k] = e0 + k <= n ? off[e0 + k] - base : 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint64_t len = e0 + k < n ? o[k + 1] - o[k] : 0;
    v[k] = e0 + k < n ? (NBUCKETS - 1 - len_bucket(len)) * SORT_SMALL + e0 + k : 0xffffffffu;
    sum += (len + 15) & ~(uint64_t)15;
  }
  uint64_t x = sum;
  for (int s = 1; s < 32; s <<= 1) {
    const uint64_t y = __shfl_up_sync(0xffffffffu, x, s);
    if (lane >= (uint32_t)s) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();  // (also: every thread has read its offsets)
  uint64_t before = lane < wid ? warp_sums[lane] : 0;
  for (int s = 16; s > 0; s >>= 1) before += __shfl_xor_sync(0xffffffffu, before, s);
  uint64_t run = before + x - sum;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t i = e0 + k;
    if (i < n) {
      poff[i] = run;
      run += (o[k + 1] - o[k] + 15) & ~(uint64_t)15;
    }
    if (i <= n && base) off[i] = o[k];
  }
  if (base && e0 + 4 == n && tid == blockDim.x - 1) off[n] = o[4];

  auto keep = [&](int k, uint32_t other, bool low) { v[k] = low ? min(v[k], other) : max(v[k], other); };
  int buf = 0;
  for (uint32_t width = 2; width <= blockDim.x * 4; width <<= 1) {
    for (uint32_t step = width >> 1; step >= 128; step >>= 1) {
      cross[buf][tid] = make_uint4(v[0], v[1], v[2], v[3]);
      __syncthreads();
      const uint4 p = cross[buf][tid ^ (step >> 2)];
      const bool low = ((e0 & step) == 0) == ((e0 & width) == 0);
      keep(0, p.x, low), keep(1, p.y, low), keep(2, p.z, low), keep(3, p.w, low);
      buf ^= 1;
    }
    for (uint32_t step = min(width >> 1, 64u); step >= 4; step >>= 1) {
      const bool low = ((e0 & step) == 0) == ((e0 & width) == 0);
#pragma unroll
      for (int k = 0; k < 4; ++k) keep(k, __shfl_xor_sync(0xffffffffu, v[k], step >> 2), low);
    }
    auto order = [&](int a, int b) {
      const bool up = ((e0 + a) & width) == 0;
      const uint32_t lo = min(v[a], v[b]), hi = max(v[a], v[b]);
      v[a] = up ? lo : hi;
      v[b] = up ? hi : lo;
    };
    if (width >= 4) order(0, 2), order(1, 3);
    order(0, 1), order(2, 3);
  }
  __syncthreads();  // the offsets of every record are written
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (e0 + k < n) {
      const uint32_t i = v[k] % SORT_SMALL;
      len_s[e0 + k] = (uint32_t)(off[i + 1] - off[i]);
      off_s[e0 + k] = poff[i];
      orig_s[e0 + k] = i;
    }
  }
}

// Copies every record to dst[poff[i] ..) in 16-byte chunks realigned with
// funnel shifts, optionally encoded through a 256-entry byte table (ish's
// convert_ascii_to_encoding, done per byte on the host by the runners,
// ishlib/parallel_line_search_runner.mojo:90-94); the tail of the 16-byte slot
// is zero-filled, and the largest code of the set is reduced into *max_code,
// so a query's alphabet can be checked once per set.  Records of PACK_LONG
// bytes or more are copied first, each by a whole block, longest first (the
// prefix of the sorted order, taken through *long_counter, which k_scatter
// zeroed): one warp cannot keep enough loads in flight to copy a megabase
// record quickly.  The other records go to groups of `gw` lanes (a power of
// two up to 32, chosen by the host near the set's average 16-byte chunks per
// record, so that short lines do not leave most of a warp idle), PACK_U
// records per group at a time.  With LIMIT, codes from `limit` up are stored as 0
// (after they went into the largest code): a caller that scores before it has
// seen that code reads no profile row outside the alphabet.  (A build of its own:
// tested at run time it took the packing of 400,000 proteins from 178 to 215 us.)
constexpr uint64_t PACK_LONG = 16384;

template <bool LIMIT>
__global__ void __launch_bounds__(256, 3) k_pack(const uint8_t *src, uint64_t src_bytes, const uint64_t *off,
                                                 const uint64_t *end, const uint64_t *poff, uint32_t n,
                                                 const uint32_t *len_s, const uint32_t *orig_s,
                                                 uint32_t *long_counter, const uint8_t *enc, uint8_t *dst,
                                                 uint32_t *max_code, uint32_t gw, uint32_t limit) {
  __shared__ uint8_t table[256];
  __shared__ uint32_t s_item;
  if (enc) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) table[i] = enc[i];
    __syncthreads();
  }
  const uint32_t group = (blockIdx.x * blockDim.x + threadIdx.x) / gw;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t glane = threadIdx.x & (gw - 1);
  const uint32_t ngroups = (gridDim.x * blockDim.x) / gw;
  const uint32_t *src32 = reinterpret_cast<const uint32_t *>(src);
  const uint64_t nwords = (src_bytes + 3) >> 2;
  uint32_t mx = 0;
  // one 16-byte chunk: realign, encode, zero the bytes past the record end,
  // store, and fold into the largest code
  auto emit = [&](uint4 *d, uint64_t c, uint64_t len, uint64_t b, const uint32_t (&w)[5]) {
    const uint32_t sh = (uint32_t)(b & 3) * 8;
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = __funnelshift_r(w[k], w[k + 1], sh);
    if (enc) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t x = o[k];
        o[k] = (uint32_t)table[x & 0xffu] | ((uint32_t)table[(x >> 8) & 0xffu] << 8) |
               ((uint32_t)table[(x >> 16) & 0xffu] << 16) | ((uint32_t)table[x >> 24] << 24);
      }
    }
    const uint64_t rem = len - c * 16;
    if (rem < 16) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int64_t keep = (int64_t)rem - 4 * k;
        if (keep <= 0) o[k] = 0;
        else if (keep < 4) o[k] &= (1u << (8 * keep)) - 1u;
      }
    }
    mx = __vmaxu4(mx, __vmaxu4(__vmaxu4(o[0], o[1]), __vmaxu4(o[2], o[3])));
    if constexpr (LIMIT) {
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k] &= __vcmpltu4(o[k], limit * 0x01010101u);
    }
    d[c] = make_uint4(o[0], o[1], o[2], o[3]);
  };
  auto load = [&](uint64_t b, uint32_t (&w)[5]) {
    const uint64_t w0 = b >> 2;
#pragma unroll
    for (int k = 0; k < 5; ++k) w[k] = (w0 + k < nwords) ? __ldg(src32 + w0 + k) : 0u;
  };
  constexpr int PACK_U = 4, PACK_V = 2;
  // chunks [c0, nchunks) of a record, `step` lanes apart, PACK_V per lane in flight
  auto copy_from = [&](uint4 *d, uint64_t s0, uint64_t len, uint64_t c0, uint64_t step) {
    const uint64_t nchunks = (len + 15) >> 4;
    for (; c0 < nchunks; c0 += (uint64_t)PACK_V * step) {
      uint32_t wc[PACK_V][5];
#pragma unroll
      for (int v = 0; v < PACK_V; ++v) {
        const uint64_t c = c0 + (uint64_t)v * step;
        if (c < nchunks) load(s0 + c * 16, wc[v]);
      }
#pragma unroll
      for (int v = 0; v < PACK_V; ++v) {
        const uint64_t c = c0 + (uint64_t)v * step;
        if (c < nchunks) emit(d, c, len, s0 + c * 16, wc[v]);
      }
    }
  };
  // long records: a whole block each, longest first
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(long_counter, 1u);
    __syncthreads();
    const uint32_t i = s_item;
    __syncthreads();  // every thread has read s_item before it is taken again
    if (i >= n || len_s[i] < PACK_LONG) break;
    const uint32_t r = orig_s[i];
    copy_from(reinterpret_cast<uint4 *>(dst + poff[r]), off[r], len_s[i], threadIdx.x, blockDim.x);
  }
  // the other records: PACK_U per group at a time, their offsets and then the
  // first chunk of each loaded before any is used, so that a group has
  // several records' loads in flight (short records are latency-bound)
  for (uint64_t r0 = group; r0 < n; r0 += (uint64_t)PACK_U * ngroups) {
    uint64_t s0[PACK_U], len[PACK_U], po[PACK_U];
#pragma unroll
    for (int u = 0; u < PACK_U; ++u) {
      const uint64_t r = r0 + (uint64_t)u * ngroups;
      s0[u] = len[u] = po[u] = 0;
      if (r < n) {  // three independent loads; a long record (done above) gets no work
        s0[u] = off[r];
        po[u] = poff[r];
        const uint64_t l = rec_len(off, end, (uint32_t)r);
        len[u] = l < PACK_LONG ? l : 0;
      }
    }
    uint32_t w[PACK_U][5];
#pragma unroll
    for (int u = 0; u < PACK_U; ++u) {
      if ((uint64_t)glane * 16 < len[u]) load(s0[u] + (uint64_t)glane * 16, w[u]);
    }
#pragma unroll
    for (int u = 0; u < PACK_U; ++u) {
      uint4 *d = reinterpret_cast<uint4 *>(dst + po[u]);
      if ((uint64_t)glane * 16 < len[u]) emit(d, glane, len[u], s0[u] + (uint64_t)glane * 16, w[u]);
      copy_from(d, s0[u], len[u], glane + gw, gw);
    }
  }
  uint32_t m = max(max(mx & 0xffu, (mx >> 8) & 0xffu), max((mx >> 16) & 0xffu, mx >> 24));
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0 && m) atomicMax(max_code, m);
}
PackFn pack_fn(bool limited) { return limited ? (PackFn)k_pack<true> : (PackFn)k_pack<false>; }

// ---------------------------------------------------------------------------
// Line splitting: the records of a text buffer are its lines, as ish's line
// reader cuts them (ishlib/vendor/kseq.mojo:270-330, read_until with the
// newline delimiter): lines end at '\n', a trailing '\r' is dropped from lines
// longer than one byte, a final line without '\n' is a record, and a final
// '\n' does not start another one.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_count_newlines(const uint8_t *text, uint64_t bytes, uint32_t *block_counts) {
  __shared__ uint32_t wsum[32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint64_t w0 = (uint64_t)blockIdx.x * LINE_TILE + (uint64_t)wid * LINE_WARP;
  uint4 w[LINE_STEPS];
  load_segment(text, bytes, w0, lane, w);
  uint32_t c = 0;
#pragma unroll
  for (uint32_t k = 0; k < LINE_STEPS; ++k)
    c += __popc(byte_bits(w[k], 0x0a0a0a0au) & inside_bits(bytes, w0 + k * 512 + lane * 16));
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (lane == 0) wsum[wid] = c;
  __syncthreads();
  if (wid == 0) {
    uint32_t v = wsum[lane];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) block_counts[blockIdx.x] = v;
  }
}

// Positions of the newlines, in order (block_offsets: exclusive scan of the
// per-block counts), and with HEADERS the first '>' or '@' of every line.  A
// line's header characters after the first are dropped inside the warp, by the
// ballots of the lanes between them and the line's start, so that a quality
// line full of '@' costs one atomic per warp segment it spans.  Measured on
// 104 MB of FASTQ (1 M lines): 127 + 159 us as two kernels of 4-byte loads that
// read the text twice each, 75 us as this one; counting 63 -> 21 us (4.9 TB/s).
template <bool HEADERS>
__global__ void __launch_bounds__(1024) k_write_newlines(const uint8_t *text, uint64_t bytes,
                                                         const uint32_t *block_offsets, uint64_t *pos,
                                                         unsigned long long *hc) {
  __shared__ uint32_t wsum[32];
  const unsigned FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint64_t w0 = (uint64_t)blockIdx.x * LINE_TILE + (uint64_t)wid * LINE_WARP;
  uint4 w[LINE_STEPS];
  load_segment(text, bytes, w0, lane, w);
  uint32_t nl[LINE_STEPS], c = 0;
#pragma unroll
  for (uint32_t k = 0; k < LINE_STEPS; ++k) {
    nl[k] = byte_bits(w[k], 0x0a0a0a0au) & inside_bits(bytes, w0 + k * 512 + lane * 16);
    c += __popc(nl[k]);
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
  if (lane == 0) wsum[wid] = c;
  __syncthreads();
  uint32_t x = wsum[lane];
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  uint32_t run = block_offsets[blockIdx.x] + __shfl_sync(FULL, x, wid) - c;  // newlines before the warp's segment
  bool carry = false;  // the line open at the step's start has a header character in this segment
#pragma unroll
  for (uint32_t k = 0; k < LINE_STEPS; ++k) {
    const uint64_t i = w0 + k * 512 + lane * 16;
    const uint32_t cnt = __popc(nl[k]);
    uint32_t incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    const uint32_t before = run + incl - cnt;
    if (HEADERS) {
      const uint32_t h = (byte_bits(w[k], 0x3e3e3e3eu) | byte_bits(w[k], 0x40404040u)) & inside_bits(bytes, i);
      // the lane's bytes of the line open at its first byte, and of the line
      // open at its last
      const uint32_t first = nl[k] ? h & ((nl[k] & (0u - nl[k])) - 1u) : h;
      const uint32_t last = nl[k] ? h & ~((2u << (31 - __clz(nl[k]))) - 1u) : h;
      const uint32_t has_nl = __ballot_sync(FULL, nl[k] != 0), has_h = __ballot_sync(FULL, last != 0);
      const uint32_t below = (1u << lane) - 1u, breaks = has_nl & below;
      const uint32_t same = breaks ? below & ~((1u << (31 - __clz(breaks))) - 1u) : below;  // lanes holding this line
      if (first && !(has_h & same) && (breaks || !carry)) atomicMin(hc + before, (unsigned long long)(i + __ffs(first) - 1));
      // lines that start inside the lane's bytes
      uint32_t line = before;
      for (uint32_t rest = nl[k]; rest;) {
        const uint32_t upto = rest & (0u - rest);  // this newline's bit
        rest ^= upto;
        ++line;
        const uint32_t seg = h & ~(upto | (upto - 1u)) & (rest ? (rest & (0u - rest)) - 1u : 0xffffu);
        if (seg) atomicMin(hc + line, (unsigned long long)(i + __ffs(seg) - 1));
      }
      carry = has_nl ? (has_h & ~((1u << (31 - __clz(has_nl))) - 1u)) != 0 : carry || has_h;
    }
    uint32_t p = before;
    for (uint32_t m = nl[k]; m; m &= m - 1) pos[p++] = i + (uint32_t)(__ffs(m) - 1);
    run += __shfl_sync(FULL, incl, 31);
  }
}
NewlinesFn write_newlines_fn(bool headers) {
  return headers ? (NewlinesFn)k_write_newlines<true> : (NewlinesFn)k_write_newlines<false>;
}

// Line i's bounds; *total accumulates the residues of all lines.
__global__ void k_line_bounds(const uint8_t *text, uint64_t bytes, const uint64_t *nl, uint32_t n_nl, uint32_t n_lines,
                              uint64_t *start, uint64_t *end, unsigned long long *total) {
  unsigned long long sum = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_lines; i += gridDim.x * blockDim.x) {
    const uint64_t s = i == 0 ? 0 : nl[i - 1] + 1;
    uint64_t e = i < n_nl ? nl[i] : bytes;
    if (e - s > 1 && text[e - 1] == '\r') --e;
    start[i] = s;
    end[i] = e;
    sum += e - s;
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(total, sum);
}

// Exclusive scan of uint64 values (n <= 1024 * 1024 * 16 per call level).
__global__ void k_scan64_block(const uint64_t *in, uint64_t *out, uint32_t n, uint64_t *block_sums) {
  __shared__ uint64_t warp_sums[32];
  const uint32_t base = blockIdx.x * SCAN_TILE;
  const int tid = threadIdx.x;
  // each thread scans SCAN_TILE / 1024 consecutive values
  constexpr int PER = SCAN_TILE / 1024;
  uint64_t v[PER];
  uint64_t s = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const uint32_t i = base + tid * PER + k;
    v[k] = i < n ? in[i] : 0;
    s += v[k];
  }
  // inclusive warp scan of s
  uint64_t x = s;
  const int lane = tid & 31, wid = tid >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint64_t w = warp_sums[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  uint64_t run = x - s + (wid > 0 ? warp_sums[wid - 1] : 0);
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const uint32_t i = base + tid * PER + k;
    if (i < n) out[i] = run;
    run += v[k];
  }
  if (tid == 1023 && block_sums) block_sums[blockIdx.x] = run;
}

__global__ void k_scan64_add(uint64_t *out, uint32_t n, const uint64_t *block_offsets) {
  const uint32_t b = blockIdx.x;
  const uint64_t add = block_offsets[b];
  for (uint32_t i = b * SCAN_TILE + threadIdx.x; i < min(n, (b + 1) * SCAN_TILE); i += blockDim.x) out[i] += add;
}

// ---------------------------------------------------------------------------
// Empty records: semi_global_aln returns (0, 0, 0) when the record or the
// query is empty (semi_global_aln/striped.mojo:275-276); sw on an empty record
// leaves max 0, end -1 and reports query end 0 (local_aln/striped.mojo:423-428).
// ---------------------------------------------------------------------------
__global__ void k_trivial(RecordsDev rec, uint32_t first, uint32_t count, int mode, int qlen, OutDev out,
                          Decision dec) {
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < count; s += gridDim.x * blockDim.x) {
    const uint32_t orig = rec.orig[first + s];
    int32_t score = 0, qe = 0, te = 0;
    if (mode == SW) {
      te = -1;
      qe = qlen > 0 ? 0 : -1;
    }
    if (out.score) out.score[orig] = score;
    if (out.qend) out.qend[orig] = qe;
    if (out.tend) out.tend[orig] = te;
    if (out.hit) out.hit[orig] = decide(mode, score, qe, te, dec);
  }
}

// ---------------------------------------------------------------------------
// The plain kernels: one thread per record, scalar Gotoh with the query on the
// inner loop -- the design of the reference's GPU kernel
// (ishlib/gpu/kernels/semi_global.mojo:20-115 with
// ishlib/matcher/alignment/semi_global_aln/basic.mojo:242-425) made exact:
// they apply the end rules of the striped CPU matchers.  Two storage forms of
// the H and E columns:
//   QMAX = 0:  int32 columns in a global scratch buffer, interleaved by thread
//              for coalescing, 128-thread blocks (any query length);
//   QMAX > 0:  int16 per-thread arrays sized for queries up to QMAX residues,
//              as the reference keeps InlineArray[NUM, max_query_length]
//              (basic.mojo:305-306), launched as 15,000 threads in blocks of 32
//              like the reference's default (ishlib/gpu/searcher_device.mojo:
//              477-497).  Exact in the fast regime, where every value fits int16.
// They are the one-query-per-launch comparison for the wavefront kernel.
// ---------------------------------------------------------------------------
template <int MODE, int QMAX>
__global__ void __launch_bounds__(QMAX ? 32 : 128) plain_kernel(const PlainParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int16_t *prof = p.prof;
  if (p.use_smem) {
    uint4 *dst = reinterpret_cast<uint4 *>(smem_raw);
    const uint4 *src = reinterpret_cast<const uint4 *>(p.prof);
    for (uint32_t i = threadIdx.x; i < p.prof_bytes / 16; i += blockDim.x) dst[i] = src[i];
    __syncthreads();
    prof = reinterpret_cast<const int16_t *>(smem_raw);
  }
  const uint32_t nth = p.nthreads;
  const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x;
  if (gt >= nth) return;
  const int Q = p.Q, open = p.open, ext = p.ext;
  const bool ts = p.ends & 4, te = p.ends & 8, qe = p.ends & 2;
  int32_t *Hc = p.scratch + gt;
  int32_t *Ec = p.scratch + (size_t)Q * nth + gt;
  int16_t Hl[QMAX ? QMAX : 1], El[QMAX ? QMAX : 1];
  auto ldH = [&](int q) -> int {
    if constexpr (QMAX > 0) return Hl[q];
    else return Hc[(size_t)q * nth];
  };
  auto ldE = [&](int q) -> int {
    if constexpr (QMAX > 0) return El[q];
    else return Ec[(size_t)q * nth];
  };
  auto stH = [&](int q, int v) {
    if constexpr (QMAX > 0) Hl[q] = (int16_t)v;
    else Hc[(size_t)q * nth] = v;
  };
  auto stE = [&](int q, int v) {
    if constexpr (QMAX > 0) El[q] = (int16_t)v;
    else Ec[(size_t)q * nth] = v;
  };
  for (uint32_t s = gt; s < p.count; s += nth) {
    const uint32_t idx = p.first + s;
    const int T = (int)p.rec.len[idx];
    const uint8_t *codes = p.rec.codes + p.rec.off[idx];
    const uint32_t orig = p.rec.orig[idx];
    for (int q = 0; q < Q; ++q) {
      const int h0 = p.hinit[q];
      stH(q, h0);
      stE(q, MODE == SW ? 0 : h0 - open);
    }
    int best = MODE == SW ? 0 : p.neg_limit, er = -1, eq = MODE == SW ? 0 : Q - 1;
    int hlast = 0;
    for (int i = 0; i < T; ++i) {
      uint32_t c = codes[i];
      if (c >= (uint32_t)p.alphabet) {
        atomicOr(p.error, 1);
        c = 0;
      }
      const int16_t *prow = prof + (size_t)c * Q;
      int hdiag, F;
      if (MODE == SW) {
        hdiag = 0;
        F = 0;
      } else {
        hdiag = (i == 0 || ts) ? 0 : -open - ext * (i - 1);  // boundary[i]
        F = (ts ? 0 : -open - ext * i) - open;                // boundary[i+1] - open
      }
      int colmax = 0, colq = 0;
      int h = 0;
      for (int q = 0; q < Q; ++q) {
        const int e = ldE(q);
        const int hold = ldH(q);
        h = max(hdiag + prow[q], max(e, F));
        hdiag = hold;
        stH(q, h);
        int v = h - open;
        if (MODE == SW) v = max(v, 0);
        stE(q, max(e - ext, v));
        F = max(F - ext, v);
        if (MODE == SW && h > colmax) {
          colmax = h;
          colq = q;
        }
      }
      if (MODE == SW) {
        if (colmax > best) {
          best = colmax;
          er = i;
          eq = colq;
        }
      } else {
        if (h > best) {
          best = h;
          er = i;
        }
        hlast = h;
      }
    }
    int score, tend, qend;
    if (MODE == SW) {
      score = best;
      tend = best == 0 ? -1 : er;
      qend = best == 0 ? 0 : eq;
    } else if (!te && !qe) {
      score = hlast;
      tend = T - 1;
      qend = Q - 1;
    } else {
      score = te ? best : p.neg_limit;
      tend = er;
      qend = Q - 1;
      if (qe) {
        for (int q = 0; q < Q; ++q) {
          const int v = ldH(q);
          if (v > score) {
            score = v;
            qend = q;
            tend = T - 1;
          } else if (v == score && tend == T - 1 && q < qend) {
            qend = q;
          }
        }
      }
    }
    if (p.out.score) p.out.score[orig] = score;
    if (p.out.qend) p.out.qend[orig] = qend;
    if (p.out.tend) p.out.tend[orig] = tend;
    if (p.out.hit) p.out.hit[orig] = decide(MODE, score, qend, tend, p.dec);
  }
}

PlainFn plain_fn(int mode, int qmax) {
  switch (qmax) {
#define ISH_PLAIN(QM) \
  case QM:            \
    return mode == SW ? (PlainFn)plain_kernel<SW, QM> : (PlainFn)plain_kernel<SG, QM>;
    ISH_PLAIN(0)
    ISH_PLAIN(64)
    ISH_PLAIN(128)
    ISH_PLAIN(256)
    ISH_PLAIN(512)
    ISH_PLAIN(1024)
    ISH_PLAIN(2048)
#undef ISH_PLAIN
    default:
      return nullptr;
  }
}

// ---------------------------------------------------------------------------
// Hit compaction: indices of hit[i] != 0 in ascending order.
// ---------------------------------------------------------------------------
// Hit compaction.  blockIdx.y selects one of several query-major flag arrays
// of n entries (batched launches); counts and offsets are laid out [y][x], so
// one exclusive scan over them concatenates the per-query hit lists.
// Hit compaction in tiles of HIT_TILE records per 1024-thread block: warp w
// of a block covers HIT_TILE / 32 consecutive records of the tile, 32 per
// ballot, so neither pass needs a block-wide barrier inside its loop.
// blockIdx.y selects one of several hit arrays of n records laid end to end.
constexpr uint32_t HIT_WARP = HIT_TILE / 32;

__global__ void __launch_bounds__(1024) k_count_hits(const uint8_t *hit, uint32_t n, uint32_t *block_counts) {
  __shared__ uint32_t wsum[32];
  hit += (size_t)blockIdx.y * n;
  block_counts += (size_t)blockIdx.y * gridDim.x;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint64_t w0 = (uint64_t)blockIdx.x * HIT_TILE + wid * HIT_WARP;
  uint32_t c = 0;
#pragma unroll
  for (uint32_t k = 0; k < HIT_WARP; k += 32) {
    const uint64_t i = w0 + k + lane;
    c += __popc(__ballot_sync(0xffffffffu, i < n && hit[i]));
  }
  if (lane == 0) wsum[wid] = c;
  __syncthreads();
  if (wid == 0) {
    uint32_t v = wsum[lane];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) block_counts[blockIdx.x] = v;
  }
}

__global__ void k_scan_counts(uint32_t *counts, uint32_t nb, uint32_t *total) {
  // single block, sequential chunks of 1024
  __shared__ uint32_t part[1024];
  uint32_t carry = 0;
  for (uint32_t base = 0; base < nb; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < nb ? counts[i] : 0;
    part[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      const uint32_t y = threadIdx.x >= (unsigned)o ? part[threadIdx.x - o] : 0;
      __syncthreads();
      part[threadIdx.x] += y;
      __syncthreads();
    }
    if (i < nb) counts[i] = carry + part[threadIdx.x] - v;
    const uint32_t tot = part[1023];
    __syncthreads();
    carry += tot;
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(1024) k_write_hits(const uint8_t *hit, uint32_t n, const uint32_t *block_offsets,
                                                     uint32_t *idx) {
  __shared__ uint32_t wsum[32];
  hit += (size_t)blockIdx.y * n;
  block_offsets += (size_t)blockIdx.y * gridDim.x;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint64_t w0 = (uint64_t)blockIdx.x * HIT_TILE + wid * HIT_WARP;
  uint32_t c = 0;
#pragma unroll
  for (uint32_t k = 0; k < HIT_WARP; k += 32) {
    const uint64_t i = w0 + k + lane;
    c += __popc(__ballot_sync(0xffffffffu, i < n && hit[i]));
  }
  if (lane == 0) wsum[wid] = c;
  __syncthreads();
  // hits of the tile's earlier warps (exclusive scan over the 32 warp counts)
  uint32_t x = wsum[lane];
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  uint32_t run = block_offsets[blockIdx.x] + __shfl_sync(0xffffffffu, x, wid) - c;
  if (!c) return;
  const uint32_t below = (1u << lane) - 1u;
  for (uint32_t k = 0; k < HIT_WARP; k += 32) {
    const uint64_t i = w0 + k + lane;
    const bool h = i < n && hit[i];
    const uint32_t m = __ballot_sync(0xffffffffu, h);
    if (h) idx[run + __popc(m & below)] = (uint32_t)i;
    run += __popc(m);
  }
}

// The whole compaction of up to COMPACT_ONE records in one block: out = {hits,
// *error, *max_code or 0}, which the host reads back together.  (One launch
// and one copy instead of three and two: scoring 500 resident lines 87 us -> 81.)
// With stage.to, pinned host memory, the results asked for are written there as
// well (see StageOut), and the call makes no copies at all.
__global__ void __launch_bounds__(1024) k_compact_one(const uint8_t *hit, uint32_t n, uint32_t *idx, const int *error,
                                                      const uint32_t *max_code, uint32_t *out, StageOut stage) {
  if (stage.to) {
    out = stage.to;
    idx = stage.to + STAGE_HEAD + 3 * SORT_SMALL;
    for (uint32_t i = threadIdx.x; i < n; i += 1024) {
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (stage.from[k]) stage.to[STAGE_HEAD + k * SORT_SMALL + i] = (uint32_t)stage.from[k][i];
      if (stage.hit) reinterpret_cast<uint8_t *>(stage.to + STAGE_HEAD + 4 * SORT_SMALL)[i] = hit[i];
    }
  }
  __shared__ uint32_t wsum[32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t per = ((n + 1023) / 1024) * 32, w0 = wid * per;  // consecutive records of each warp
  uint32_t c = 0;
#pragma unroll 4
  for (uint32_t k = 0; k < per; k += 32) {
    const uint32_t i = w0 + k + lane;
    c += __popc(__ballot_sync(0xffffffffu, i < n && hit[i]));
  }
  if (lane == 0) wsum[wid] = c;
  __syncthreads();
  uint32_t x = wsum[lane];
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  uint32_t run = __shfl_sync(0xffffffffu, x, wid) - c;
  if (threadIdx.x == 31) {
    out[0] = x;
    out[1] = (uint32_t)*error;
    out[2] = max_code ? *max_code : 0u;
  }
  if (!c) return;
  const uint32_t below = (1u << lane) - 1u;
  for (uint32_t k = 0; k < per; k += 32) {
    const uint32_t i = w0 + k + lane;
    const bool h = i < n && hit[i];
    const uint32_t m = __ballot_sync(0xffffffffu, h);
    if (h) idx[run + __popc(m & below)] = i;
    run += __popc(m);
  }
}

// k_write_hits without the scan between it and k_count_hits: every block adds
// the counts of the tiles before its own, at most 1,024 of them, and the last
// writes out = {hits, *error, 0}.  (100,000 resident lines 122 us -> 118.)
__global__ void __launch_bounds__(1024) k_write_hits_sum(const uint8_t *hit, uint32_t n, const uint32_t *block_counts,
                                                         uint32_t *idx, const int *error, uint32_t *out) {
  __shared__ uint32_t wsum[32], bsum[32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t before = threadIdx.x < blockIdx.x ? block_counts[threadIdx.x] : 0u;
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  const uint64_t w0 = (uint64_t)blockIdx.x * HIT_TILE + wid * HIT_WARP;
  uint32_t c = 0;
#pragma unroll
  for (uint32_t k = 0; k < HIT_WARP; k += 32) {
    const uint64_t i = w0 + k + lane;
    c += __popc(__ballot_sync(0xffffffffu, i < n && hit[i]));
  }
  if (lane == 0) {
    wsum[wid] = c;
    bsum[wid] = before;
  }
  __syncthreads();
  uint32_t x = wsum[lane], b = bsum[lane];
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
  uint32_t run = b + __shfl_sync(0xffffffffu, x, wid) - c;
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 31) {
    out[0] = b + x;
    out[1] = (uint32_t)*error;
    out[2] = 0;
  }
  if (!c) return;
  const uint32_t below = (1u << lane) - 1u;
  for (uint32_t k = 0; k < HIT_WARP; k += 32) {
    const uint64_t i = w0 + k + lane;
    const bool h = i < n && hit[i];
    const uint32_t m = __ballot_sync(0xffffffffu, h);
    if (h) idx[run + __popc(m & below)] = (uint32_t)i;
    run += __popc(m);
  }
}

// Scores and end coordinates of the compacted hits (the hit count is read on
// the device, so no host round trip is needed before the gather).
__global__ void k_gather_hits(const uint32_t *idx, const uint32_t *count, const int32_t *score, const int32_t *qend,
                              const int32_t *tend, int32_t *hit_score, int32_t *hit_qend, int32_t *hit_tend) {
  const uint32_t nh = *count;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x) {
    const uint32_t r = idx[i];
    hit_score[i] = score[r];
    hit_qend[i] = qend[r];
    hit_tend[i] = tend[r];
  }
}

// ---------------------------------------------------------------------------
// Calibration: throughput of the packed 16-bit DPX add-max instruction the
// cell recurrence is built from.  Eight independent dependency chains per
// thread keep the pipe busy; the result is folded so nothing is dead code.
// ---------------------------------------------------------------------------
__global__ void k_dpx_peak(uint32_t *out, int iters, uint32_t b, uint32_t c) {
  uint32_t a[8], cc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    a[k] = threadIdx.x * 0x00010001u + k;
    cc[k] = c + k * 0x00030005u;
  }
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = __viaddmax_s16x2(a[k], b, cc[k]);
  }
  uint32_t x = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) x ^= a[k];
  if (x == 0x12345678u) out[0] = x;
}

// Local-alignment cell updates on packed lanes, for the lane-width choice of
// the wavefront kernel.  U8 = false: two 16-bit lanes per word and five DPX
// add-max per word (the wavefront kernel needs four).  U8 = true: four 8-bit lanes
// per word with a biased unsigned byte profile, as the reference's u8 pass
// keeps it (local_aln/striped.mojo:78-139), through the saturating SIMD byte
// intrinsics (add, subtract, max: ten per word).  Sixteen words of columns
// per thread in registers and no memory traffic in the loop; the row's
// boundary changes every row, so nothing is hoisted out of it.
template <bool U8>
__global__ void k_lane_rows(uint32_t *out, int rows, uint32_t p0, uint32_t popen, uint32_t pext, uint32_t bias) {
  constexpr int K = 16;
  uint32_t H[K], E[K], P[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    H[j] = 0;
    E[j] = 0;
    P[j] = (p0 + (uint32_t)j * 0x01030107u) ^ (threadIdx.x * 0x00010001u);
  }
  // 16-bit lanes add the negated penalties; 8-bit lanes subtract them
  const uint32_t n16o = (0u - popen) & 0xffffu, n16e = (0u - pext) & 0xffffu;
  const uint32_t OPEN = U8 ? popen : (n16o | (n16o << 16));
  const uint32_t EXT = U8 ? pext : (n16e | (n16e << 16));
  for (int r = 0; r < rows; ++r) {
    const uint32_t diag = (uint32_t)r * 0x00050005u;
#pragma unroll
    for (int j = K - 1; j >= 0; --j) {
      const uint32_t hd = j ? H[j - 1] : diag;
      uint32_t T;
      if (U8) {
        T = __vmaxu4(__vsubus4(__vaddus4(hd, P[j]), bias), E[j]);
        E[j] = __vmaxu4(__vsubus4(E[j], EXT), __vsubus4(T, OPEN));
      } else {
        T = __viaddmax_s16x2(hd, P[j], E[j]);
        E[j] = __viaddmax_s16x2(E[j], EXT, __viaddmax_s16x2(T, OPEN, 0u));
      }
      H[j] = T;
    }
    uint32_t fs = OPEN;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint32_t T = H[j];
      if (U8) {
        H[j] = __vmaxu4(__vsubus4(fs, OPEN), T);
        fs = __vmaxu4(__vsubus4(fs, EXT), T);
      } else {
        H[j] = __viaddmax_s16x2(fs, OPEN, T);
        fs = __viaddmax_s16x2(fs, EXT, T);
      }
    }
  }
  uint32_t x = 0;
#pragma unroll
  for (int j = 0; j < K; ++j) x ^= H[j] ^ E[j];
  if (x == 0x12345678u) out[0] = x;
}
LaneFn lane_rows_fn(bool u8) { return u8 ? (LaneFn)k_lane_rows<true> : (LaneFn)k_lane_rows<false>; }

}  // namespace ish
