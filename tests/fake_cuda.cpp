// A CUDA runtime without a device, linked with the library's own objects: device
// memory is host memory, streams run every call at once and the kernels listed
// in launch() are written out here (the others do nothing).  It checks what a
// device would not report:
//   - what a blocking upload from pageable memory or a memset leaves on its way, in
//     the order of the legacy stream alone, has been waited for when another stream
//     launches a kernel;
//   - the source of an asynchronous upload from pageable memory stays readable
//     and unchanged until its stream has been waited for;
//   - what the kernels written out here touch lies inside one allocation.
#include <cuda_runtime.h>
#include <malloc.h>
#include <sys/uio.h>
#include <unistd.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <string>
#include <thread>
#include <vector>

namespace {

std::recursive_mutex mu;
std::map<const void *, std::string> kernels;          // host stub -> device name
std::map<const char *, size_t> device, pinned;        // allocation -> bytes
struct Upload {
  cudaStream_t stream;
  const char *src;
  std::string bytes;  // the source when the copy was asked for
};
std::vector<Upload> uploads;  // not waited for yet
std::string report, wave;             // wave: the last wavefront kernel launched
std::vector<std::string> contents;  // of the asynchronous uploads from pageable memory
bool on_its_way = false;  // a legacy-stream upload or memset that nothing has waited for
bool refuse_func_attributes = false, refuse_other_threads = false;
std::thread::id caller;  // where refuse_other_threads was set
int copies_to_go = -1;  // asynchronous copies that still succeed before one is refused (-1: all)
dim3 grid_, block_;
size_t shared_;
cudaStream_t stream_;

const auto perturb = mallopt(M_PERTURB, 0xa5);  // freed memory does not keep its contents

// Bytes from p to the end of the allocation it lies in (0: in none).
size_t room(const std::map<const char *, size_t> &m, const void *p) {
  auto it = m.upper_bound((const char *)p);
  if (it == m.begin()) return 0;
  --it;
  const size_t at = (const char *)p - it->first;
  return at < it->second ? it->second - at : 0;
}

void touch(const char *what, const void *p, size_t bytes) {
  if (bytes && room(device, p) < bytes)
    report += std::string(what) + ": " + std::to_string(bytes) + " bytes, room for " + std::to_string(room(device, p)) + "\n";
}

void waited(cudaStream_t s) {
  for (size_t i = 0; i < uploads.size();) {
    if (uploads[i].stream != s) {
      ++i;
      continue;
    }
    std::string now(uploads[i].bytes.size(), 0);
    iovec to{&now[0], now.size()}, from{(void *)uploads[i].src, now.size()};
    if (process_vm_readv(getpid(), &to, 1, &from, 1, 0) != (ssize_t)now.size() || now != uploads[i].bytes)
      report += "an upload's source was gone before its stream was waited for\n";
    uploads.erase(uploads.begin() + i);
  }
}

template <class T>
T arg(void **a, int i) {
  return *(T *)a[i];
}

uint64_t bucket(uint64_t len) { return len < 32768 ? len : std::min<uint64_t>(32768 + ((len - 32768) >> 5), 65535); }

// The longest first, equal lengths in record order.
void sort_records(const uint32_t *len, const uint64_t *pos, uint32_t n, uint32_t *len_s, uint64_t *off_s, uint32_t *orig_s) {
  std::iota(orig_s, orig_s + n, 0u);
  std::stable_sort(orig_s, orig_s + n, [&](uint32_t x, uint32_t y) { return bucket(len[x]) > bucket(len[y]); });
  for (uint32_t e = 0; e < n; ++e) {
    len_s[e] = len[orig_s[e]];
    off_s[e] = pos[orig_s[e]];
  }
}

void launch(const std::string &name, void **a) {
  auto is = [&](const char *k) { return name.find(k) != std::string::npos; };
  if (is("wave_kernel") || is("batch_kernel")) wave = name;
  if (is("k_sort_small")) {
    const uint64_t *off = arg<uint64_t *>(a, 0);
    const uint32_t n = arg<uint32_t>(a, 1);
    std::vector<uint32_t> len(n);
    std::vector<uint64_t> pos(n);
    for (uint32_t i = 0; i < n; ++i) len[i] = (uint32_t)(off[i + 1] - off[i]);
    for (uint32_t i = 1; i < n; ++i) pos[i] = pos[i - 1] + ((len[i - 1] + 15) & ~15ull);
    sort_records(len.data(), pos.data(), n, arg<uint32_t *>(a, 4), arg<uint64_t *>(a, 5), arg<uint32_t *>(a, 6));
  } else if (is("k_lengths")) {
    const uint64_t *off = arg<uint64_t *>(a, 0), *end = arg<uint64_t *>(a, 1);
    for (uint32_t i = 0; i < arg<uint32_t>(a, 2); ++i)
      arg<uint32_t *>(a, 3)[i] = (uint32_t)((end ? end[i] : off[i + 1]) - off[i]);
    arg<uint32_t *>(a, 7)[0] = 0;
  } else if (is("k_scan_slots")) {
    uint64_t sum = 0;
    for (uint32_t i = 0; i < arg<uint32_t>(a, 1); ++i) {
      arg<uint64_t *>(a, 3)[i] = sum;
      sum += (arg<uint32_t *>(a, 0)[i] + 15) & ~15ull;
    }
  } else if (is("k_scatter")) {
    const uint32_t n = arg<uint32_t>(a, 2);
    uint32_t *len_s = arg<uint32_t *>(a, 4), *summary = arg<uint32_t *>(a, 9);
    sort_records(arg<uint32_t *>(a, 0), arg<uint64_t *>(a, 1), n, len_s, arg<uint64_t *>(a, 5), arg<uint32_t *>(a, 6));
    std::fill(summary + 2, summary + 2 + 65536, 0u);
    for (uint32_t e = 0; e < n; ++e) ++summary[2 + bucket(len_s[e])];
    summary[1] = (uint32_t)bucket(len_s[0]);
  } else if (is("k_pack")) {  // the largest code alone
    for (uint64_t i = 0; i < arg<uint64_t>(a, 1); ++i)
      *arg<uint32_t *>(a, 11) = std::max<uint32_t>(*arg<uint32_t *>(a, 11), arg<uint8_t *>(a, 0)[i]);
  } else if (is("k_compact_one")) {  // the head of its results alone
    uint32_t *out = *(uint32_t **)a[6] ? *(uint32_t **)a[6] : arg<uint32_t *>(a, 5);
    out[0] = 0;
    out[1] = *arg<uint32_t *>(a, 3);
    out[2] = arg<uint32_t *>(a, 4) ? *arg<uint32_t *>(a, 4) : 0;
  } else if (is("k_invert")) {
    for (uint32_t e = 0; e < arg<uint32_t>(a, 1); ++e) arg<uint32_t *>(a, 2)[arg<uint32_t *>(a, 0)[e]] = e;
  } else if (is("k_rev_lengths")) {
    for (uint32_t i = 0; i < arg<uint32_t>(a, 2); ++i) {
      const int64_t rows = (int64_t)arg<int32_t *>(a, 1)[i] + 1;
      const uint32_t len = arg<uint32_t *>(a, 4)[arg<uint32_t *>(a, 3)[arg<uint32_t *>(a, 0)[i]]];
      const uint32_t r = (uint32_t)std::max<int64_t>(0, std::min<int64_t>(rows, len));
      arg<uint32_t *>(a, 6)[i] = r;
      arg<uint64_t *>(a, 7)[i] = ((uint64_t)r + 16) & ~15ull;
    }
  } else if (is("k_scan64_block")) {
    uint64_t sum = 0;
    for (uint32_t i = 0; i < arg<uint32_t>(a, 2); ++i) {
      arg<uint64_t *>(a, 1)[i] = sum;
      sum += arg<uint64_t *>(a, 0)[i];
    }
  } else if (is("k_rev_pack")) {
    const uint32_t n = arg<uint32_t>(a, 1);
    if (n) touch("reversed prefixes", arg<uint8_t *>(a, 9), arg<uint64_t *>(a, 7)[n - 1] + arg<uint64_t *>(a, 8)[n - 1]);
  }
}

cudaError_t alloc(std::map<const char *, size_t> &m, void **p, size_t bytes) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (refuse_other_threads && std::this_thread::get_id() != caller) return cudaErrorMemoryAllocation;
  *p = calloc(1, bytes);
  m[(const char *)*p] = bytes;
  return cudaSuccess;
}
cudaError_t release(std::map<const char *, size_t> &m, void *p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  m.erase((const char *)p);
  free(p);
  return cudaSuccess;
}
template <class T>
cudaError_t handle(T *p) {
  static char next[1 << 16];
  static size_t k = 0;
  std::lock_guard<std::recursive_mutex> lk(mu);
  *p = (T)&next[++k];
  return cudaSuccess;
}

}  // namespace

extern "C" {

__attribute__((visibility("default"))) const char *fake_report() { return report.c_str(); }
__attribute__((visibility("default"))) const char *fake_last_wave() { return wave.c_str(); }
// Bytes of upload i from the last (0), to `to` if given.
__attribute__((visibility("default"))) size_t fake_upload(size_t i, char *to) {
  const std::string &c = contents[contents.size() - 1 - i];
  if (to) memcpy(to, c.data(), c.size());
  return c.size();
}
__attribute__((visibility("default"))) void fake_refuse_func_attributes(int on) { refuse_func_attributes = on; }
__attribute__((visibility("default"))) void fake_refuse_memory_to_other_threads(int on) {
  refuse_other_threads = on;
  caller = std::this_thread::get_id();
}
__attribute__((visibility("default"))) void fake_refuse_copy_after(int n) { copies_to_go = n; }
__attribute__((visibility("default"))) int fake_unread_uploads() { return (int)uploads.size(); }

void **__cudaRegisterFatBinary(void *) { return (void **)&perturb; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  kernels[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, CUstream_st *st) {
  mu.lock();  // (until the launch has taken them)
  grid_ = g, block_ = b, shared_ = s, stream_ = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
  *g = grid_, *b = block_, *s = shared_, *(cudaStream_t *)st = stream_;
  mu.unlock();
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **a, size_t, cudaStream_t) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (on_its_way) report += kernels[(const void *)k] + " launched while an upload was on its way\n";
  launch(kernels[(const void *)k], a);
  return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { return *f = *t = size_t(4) << 30, cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "refused"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *, const void *) { return cudaErrorInvalidValue; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) {
  return refuse_func_attributes ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorInvalidValue; }

cudaError_t cudaMalloc(void **p, size_t bytes) { return alloc(device, p, bytes); }
cudaError_t cudaFree(void *p) { return release(device, p); }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { return alloc(pinned, p, bytes); }
cudaError_t cudaMallocHost(void **p, size_t bytes) { return alloc(pinned, p, bytes); }
cudaError_t cudaFreeHost(void *p) { return release(pinned, p); }

cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t bytes, cudaMemcpyKind kind, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (copies_to_go >= 0 && copies_to_go-- == 0) return cudaErrorInvalidValue;
  if (kind != cudaMemcpyDeviceToHost) touch("copy to the device", to, bytes);
  if (kind != cudaMemcpyHostToDevice) touch("copy from the device", from, bytes);
  if (kind == cudaMemcpyHostToDevice && !room(pinned, from))
    uploads.push_back(Upload{s, (const char *)from, std::string((const char *)from, bytes)}),
        contents.push_back(uploads.back().bytes);
  memmove(to, from, bytes);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *to, const void *from, size_t bytes, cudaMemcpyKind kind) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  memmove(to, from, bytes);
  on_its_way = kind == cudaMemcpyHostToDevice && !room(pinned, from);  // (earlier ones end before it begins)
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t bytes) {
  on_its_way = true;
  return memset(p, v, bytes), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t bytes, cudaStream_t) {
  if (!p) return cudaErrorInvalidValue;
  touch("memset", p, bytes);
  return memset(p, v, bytes), cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (!s || s == cudaStreamLegacy) on_its_way = false;
  waited(s);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
std::map<cudaEvent_t, cudaStream_t> recorded;
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  recorded[e] = s;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  return cudaStreamSynchronize(recorded[e]);
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }

// (a captured stream runs its calls at once, a graph launch runs nothing again)
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return handle(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *g, cudaGraph_t, unsigned long long) { return handle(g); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

}  // extern "C"
