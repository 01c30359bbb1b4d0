// starts.cu -- match starts on the device (ish_gpu_match_starts): the reverse
// pass that the CPU matchers run for every hit.
//
//   semi-global: semi_global_aln_start_end runs semi_global_aln again on the
//     reversed prefix record[0 : target_end + 1] with the reversed query and
//     swapped free ends; start = len(prefix) - reverse.reference - 1
//     (ishlib/matcher/alignment/semi_global_aln/striped.mojo:160-191, and the
//     matcher's find_start, striped_semi_global_matcher.mojo:259-276);
//   local: ssw_align runs sw over record[0 : ref_end + 1] backwards with the
//     reversed query; ref_begin = the record index of that pass's best
//     (ishlib/matcher/alignment/local_aln/striped.mojo:232-259).
//
// Both are the forward pass on reversed inputs, so the device builds the
// reversed prefixes of all hits as a packed record set, scores it with the
// wavefront kernel and the reversed query, and turns the reverse end row j
// into start = len(prefix) - 1 - j.
#include <algorithm>
#include <cstring>
#include <vector>

#include "host.h"

namespace ish {

__global__ void k_invert(const uint32_t *orig_s, uint32_t n, uint32_t *inv) {
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) inv[orig_s[s]] = s;
}

// Prefix length and 16-byte slot of every hit (the slot keeps at least one
// zero byte past the prefix and is never empty).  No prefix is longer than
// `most`, for which the host has made room.
__global__ void k_rev_lengths(const uint32_t *hits, const int32_t *tend, uint32_t nh, const uint32_t *inv,
                              const uint32_t *len_s, uint32_t n, uint32_t *rlen, uint64_t *slot, uint32_t *orig,
                              int32_t *rev_end, int *error, uint64_t most) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x) {
    const uint32_t h = hits[i];
    uint32_t r = 0;
    if (h < n) {
      const int64_t T = len_s[inv[h]];
      int64_t e = (int64_t)tend[i] + 1;
      e = e < 0 ? 0 : e;
      r = (uint32_t)(e < T ? e : T);
      if (r > most) {
        r = 0;
        atomicOr(error, 4);
      }
    } else {
      atomicOr(error, 4);
    }
    rlen[i] = r;
    slot[i] = ((uint64_t)r + 16) & ~(uint64_t)15;
    orig[i] = i;
    rev_end[i] = 0;
  }
}

// One warp per hit: reversed prefix, zero padded to the slot end.
__global__ void k_rev_pack(const uint32_t *hits, uint32_t nh, uint32_t n, const uint32_t *inv, const uint8_t *codes,
                           const uint64_t *off_s, const uint32_t *rlen, const uint64_t *poff, const uint64_t *slot,
                           uint8_t *dst) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nh; i += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t h = hits[i];
    const uint32_t r = rlen[i];
    const uint8_t *src = h < n ? codes + off_s[inv[h]] : codes;
    uint8_t *d = dst + poff[i];
    const uint64_t sz = slot[i];
    for (uint64_t j = lane; j < sz; j += 32) d[j] = j < r ? src[r - 1 - j] : 0;
  }
}

// (start may be pinned host memory, as error_out always is)
__global__ void k_starts(const uint32_t *rlen, const int32_t *rev_end, uint32_t nh, int64_t *start, const int *error,
                         uint32_t *error_out) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *error_out = (uint32_t)*error;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x)
    start[i] = (int64_t)rlen[i] - 1 - rev_end[i];
}

namespace host {
namespace {

// Reversed prefixes of up to this many bytes are allocated for by their bound and
// kept for the next call.
constexpr uint64_t STARTS_KEEP = uint64_t(256) << 20;

// The reversed query: sequence reversed, free query/target start and end
// swapped (semi_global_aln_start_end, striped.mojo:165-183).
Query &reverse_of(Query &q) {
  if (!q.reverse) {
    q.reverse.reset(new Query());
    Query &r = *q.reverse;
    clone_params(q, r);
    std::reverse(r.q.begin(), r.q.end());
    if (q.algo == ISH_ALGO_SEMI_GLOBAL) {
      const int e = q.ends;
      r.ends = ((e & ISH_FREE_QUERY_END) ? ISH_FREE_QUERY_START : 0) |
               ((e & ISH_FREE_QUERY_START) ? ISH_FREE_QUERY_END : 0) |
               ((e & ISH_FREE_TARGET_END) ? ISH_FREE_TARGET_START : 0) |
               ((e & ISH_FREE_TARGET_START) ? ISH_FREE_TARGET_END : 0);
    }
  }
  return *q.reverse;
}

}  // namespace
}  // namespace host
}  // namespace ish

using namespace ish;
using namespace ish::host;

extern "C" int ish_gpu_match_starts(ish_ctx *ctx, int32_t query_id, int32_t set_id, const uint32_t *hit_idx,
                                    const int32_t *target_end, uint32_t n_hits, int64_t *start) {
  if (!ctx) return ISH_EINVAL;
  auto qi = ctx->queries.find(query_id);
  if (qi == ctx->queries.end()) return fail(ctx, ISH_EINVAL, "unknown query %d", query_id);
  int urc = ISH_OK;
  RecordSet *si_set = use_set(ctx, set_id, &urc);
  if (!si_set) return urc;
  if (n_hits == 0) return ISH_OK;
  if (!hit_idx || !target_end || !start) return fail(ctx, ISH_EINVAL, "hit_idx, target_end and start are required");
  cudaSetDevice(ctx->device);
  Query &q = qi->second;
  RecordSet &rs = *si_set;
  const uint32_t n = rs.n;
  // Bounds of the reversed prefixes' rows and bytes, from the ends alone (a row
  // count is also at most its record's, which the device knows; the host knows
  // the longest record's, or, where the last length bucket holds some, the set's).
  const uint64_t most = top_bucket(rs) == NBUCKETS - 1 ? std::min<uint64_t>(rs.total, 0xffffffffu) : rs.max_len;
  uint64_t bound = 0;
  uint32_t longest = 0;
  for (uint32_t i = 0; i < n_hits; ++i) {
    if (hit_idx[i] >= n) return fail(ctx, ISH_EINVAL, "hit index %u >= %u records", hit_idx[i], n);
    const uint32_t r = (uint32_t)std::min<int64_t>(std::max<int64_t>((int64_t)target_end[i] + 1, 0), (int64_t)most);
    longest = std::max(longest, r);
    bound += ((uint64_t)r + 16) & ~(uint64_t)15;
  }
  Query &rq = reverse_of(q);
  // the reverse pass runs where the forward pass ran: the wavefront kernels
  // in their exact regime, else the lane-exact emulation (exact.cu)
  bool fast = rq.Q > 0 && ctx->kernel != ISH_KERNEL_EXACT;
  if (fast) {
    int G, K, layout;
    pick_shape(ctx, rq, &G, &K, &layout);
    Regime r = regime(rq, G ? G * K : rq.Q + 64);
    fast = r.fast && G && G * K >= rq.Q + 1 && (r.max_safe_len == ~0ull || rs.max_len <= r.max_safe_len);
  }
  if (rq.Q > 0 && rs.max_code >= (uint32_t)rq.alphabet)
    return fail(ctx, ISH_EINVAL, "a record contains code %u >= the alphabet size %d of the query", rs.max_code,
                rq.alphabet);
  cudaStream_t s = ctx->stream;
  const uint32_t nb = std::max<uint32_t>(1, std::min<uint32_t>(ceil_div(n, 256), (uint32_t)ctx->num_sms * 8));
  if (!rs.inv_ready) {
    CU(rs.inv.ensure((size_t)n * 4));
    k_invert<<<nb, 256, 0, s>>>(rs.orig_s.as<uint32_t>(), n, rs.inv.as<uint32_t>());
    ++ctx->launches;
    CU(cudaGetLastError());
    rs.inv_ready = true;
  }
  // The context keeps the call's buffers (unless large): allocating and freeing
  // ten of them and waiting for lengths in between took 245 of the 375 us of
  // 2,205 hits in reads.
  RecordSet rev;
  rev.windows = ctx->starts_windows;
  ctx->starts_windows = WindowView{};
  auto cleanup = [&] {
    rev.windows.clear();
    ctx->starts_windows = rev.windows;
    if (ctx->starts_ws.cap > (size_t(64) << 20)) ctx->starts_ws.release();
    if (ctx->starts_codes.cap > STARTS_KEEP) ctx->starts_codes.release();
  };
  int rc = ISH_OK;
  do {
    const uint32_t tiles = ceil_div(n_hits, SCAN_TILE);
    if (tiles > SCAN_TILE) {
      rc = fail(ctx, ISH_EINVAL, "too many hits in one call (%u)", n_hits);
      break;
    }
#define SCU(call)                                                                                  \
  {                                                                                                \
    cudaError_t _e = (call);                                                                       \
    if (_e != cudaSuccess) {                                                                       \
      (void)cudaGetLastError();                                                                    \
      rc = fail(ctx, _e == cudaErrorMemoryAllocation ? ISH_ENOMEM : ISH_EDEVICE, "%s: %s", #call,  \
                cudaGetErrorString(_e));                                                           \
      break;                                                                                       \
    }                                                                                              \
  }
    // per hit: slot, packed offset, start; hit, end, rows, order, reverse end
    const size_t nh = ((size_t)n_hits + 3) & ~(size_t)3;
    SCU(ctx->starts_ws.ensure(nh * 44 + (size_t)(tiles + 1) * 16 + 16));
    uint64_t *slot = ctx->starts_ws.as<uint64_t>(), *poff = slot + nh, *bsum = poff + nh + 2;
    uint64_t *boff = bsum + tiles + 1;
    int64_t *d_start = reinterpret_cast<int64_t *>(boff + tiles + 1);
    uint32_t *d_hits = reinterpret_cast<uint32_t *>(d_start + nh), *rlen = d_hits + 2 * nh, *orig = rlen + nh;
    int32_t *d_tend = reinterpret_cast<int32_t *>(d_hits + nh), *rev_end = reinterpret_cast<int32_t *>(orig + nh);
    SCU(ctx->error.ensure(64));
    SCU(cudaMemsetAsync(ctx->error.p, 0, 4, s));
    // few hits: both arrays in one copy from pinned memory, the starts written back there
    const bool staged = nh * 8 + 16 <= STAGE_WORDS * 4;
    if (staged) {
      memcpy(ctx->h_stage, hit_idx, (size_t)n_hits * 4);
      memcpy(ctx->h_stage + nh, target_end, (size_t)n_hits * 4);
      SCU(cudaMemcpyAsync(d_hits, ctx->h_stage, nh * 8, cudaMemcpyHostToDevice, s));
    } else {
      SCU(cudaMemcpyAsync(d_hits, hit_idx, (size_t)n_hits * 4, cudaMemcpyHostToDevice, s));
      SCU(cudaMemcpyAsync(d_tend, target_end, (size_t)n_hits * 4, cudaMemcpyHostToDevice, s));
    }
    const uint32_t hb = std::max<uint32_t>(1, std::min<uint32_t>(ceil_div(n_hits, 256), (uint32_t)ctx->num_sms * 8));
    k_rev_lengths<<<hb, 256, 0, s>>>(d_hits, d_tend, n_hits, rs.inv.as<uint32_t>(), rs.len_s.as<uint32_t>(), n, rlen,
                                     slot, orig, rev_end, ctx->error.as<int>(), most);
    ++ctx->launches;
    k_scan64_block<<<tiles, 1024, 0, s>>>(slot, poff, n_hits, bsum);
    ++ctx->launches;
    if (tiles > 1) {
      k_scan64_block<<<1, 1024, 0, s>>>(bsum, boff, tiles, nullptr);
      ++ctx->launches;
      k_scan64_add<<<tiles, 1024, 0, s>>>(poff, n_hits, boff);
      ++ctx->launches;
    }
    SCU(cudaGetLastError());
    // (ends far past their records make the bounds too large to allocate for)
    if (bound > STARTS_KEEP) {
      uint64_t last[2] = {0, 0};
      SCU(cudaMemcpyAsync(&last[0], poff + n_hits - 1, 8, cudaMemcpyDeviceToHost, s));
      SCU(cudaMemcpyAsync(&last[1], slot + n_hits - 1, 8, cudaMemcpyDeviceToHost, s));
      std::vector<uint32_t> hl(n_hits);
      SCU(cudaMemcpyAsync(hl.data(), rlen, (size_t)n_hits * 4, cudaMemcpyDeviceToHost, s));
      SCU(cudaStreamSynchronize(s));
      bound = last[0] + last[1];
      longest = *std::max_element(hl.begin(), hl.end());
    }
    SCU(ctx->starts_codes.ensure(bound + 16));
    rev.codes = ctx->starts_codes;  // (borrowed, like the arrays below)
    k_rev_pack<<<std::max<uint32_t>(1, std::min<uint32_t>(ceil_div((uint64_t)n_hits * 32, 256),
                                                          (uint32_t)ctx->num_sms * 16)),
                 256, 0, s>>>(d_hits, n_hits, n, rs.inv.as<uint32_t>(), rs.codes.as<uint8_t>(), rs.off_s.as<uint64_t>(),
                              rlen, poff, slot, rev.codes.as<uint8_t>());
    ++ctx->launches;
    SCU(cudaGetLastError());
    // the reversed prefixes as a record set in hit order (empty prefixes keep
    // reverse end 0, i.e. start -1, as semi_global_aln gives for an empty
    // record)
    rev.n = n_hits;
    rev.total = bound;
    rev.off_s.p = poff;
    rev.len_s.p = rlen;
    rev.orig_s.p = orig;
    OutDev out{nullptr, nullptr, rev_end, nullptr};
    if (rq.Q > 0 && fast) {
      // long prefixes (hits in long records) go through the window view like
      // a forward pass; it needs the longest prefix
      rev.max_len = longest;
      bool windowed = false;
      rc = launch_windows(ctx, rq, rev, n_hits, out, s, &windowed);
      if (!rc && !windowed) rc = launch_range(ctx, rq, rev, 0, n_hits, out, s);
    } else if (rq.Q > 0) {
      rc = launch_exact(ctx, rq, rev, 0, n_hits, out, s);
    }
    if (rc) break;
    int64_t *to = staged ? reinterpret_cast<int64_t *>(ctx->h_stage + 4) : d_start;
    k_starts<<<hb, 256, 0, s>>>(rlen, rev_end, n_hits, to, ctx->error.as<int>(), ctx->h_stage);
    ++ctx->launches;
    SCU(cudaGetLastError());
    if (!staged) SCU(cudaMemcpyAsync(start, d_start, (size_t)n_hits * 8, cudaMemcpyDeviceToHost, s));
    SCU(cudaStreamSynchronize(s));
    if (staged) memcpy(start, to, (size_t)n_hits * 8);
    const uint32_t herr = ctx->h_stage[0];
    if (herr & 2) rc = fail(ctx, ISH_ETIMEDOUT, "wavefront kernel exceeded its step budget (internal error)");
    else if (herr) rc = fail(ctx, ISH_EINVAL, "bad hit index or record code");
#undef SCU
  } while (0);
  cudaStreamSynchronize(s);
  cleanup();
  return rc;
}
