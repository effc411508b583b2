// A CUDA runtime without a device, for tests of the host code's launch order:
// the library's host sources are linked with it in place of libcudart and of
// the kernels.  Every stream operation becomes an entry of a log with the set
// of operations that are ordered before it -- by its stream, by the events
// that the stream waited for, and by the host's synchronisations -- which
// fake_before() answers from.  Device memory is host memory (never touched by
// a kernel); an allocation larger than fake_limit() fails.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

#include "engine.h"

namespace {

using Set = std::vector<bool>;

struct Op {
  std::string name;
  long stream;
  Set before;   // operations ordered before this one
  bool whole;   // the plan's buffers were all there
};

std::recursive_mutex mu;
std::vector<Op> ops;
std::map<long, Set> streams;  // what the stream's next operation comes after
std::map<long, Set> events;
std::map<long, int> priority; // streams with one
Set host;                     // what the host has waited for
std::map<char *, size_t> mem;
size_t limit_bytes = (size_t)-1;
std::string failing;
int passes = 0;  // operations of that name that still succeed
long next_handle = 0x1000;

void merge(Set &a, const Set &b) {
  if (a.size() < b.size()) a.resize(b.size());
  for (size_t i = 0; i < b.size(); i++)
    if (b[i]) a[i] = true;
}

cudaError_t op(const char *name, const void *s, bool whole = true) {
  std::lock_guard<std::recursive_mutex> g(mu);
  if (failing == name && passes-- <= 0) return cudaErrorUnknown;
  Set &st = streams[(long)s];
  merge(st, host);
  const size_t i = ops.size();
  ops.push_back(Op{name, (long)s, st, whole});
  if (st.size() <= i) st.resize(i + 1);
  st[i] = true;
  return cudaSuccess;
}

void *allocate(size_t n) {
  if (n > limit_bytes) return nullptr;
  void *p = nullptr;
  if (posix_memalign(&p, 256, n ? n : 16)) return nullptr;
  return p;
}

}  // namespace

extern "C" {

// ------------------------------------------------------ what tests ask --

int fake_ops() { return (int)ops.size(); }
const char *fake_name(int i) { return ops[i].name.c_str(); }
int fake_whole(int i) { return ops[i].whole; }
// Whether operation a is complete when b starts, on every schedule.
int fake_before(int a, int b) { return a < (int)ops[b].before.size() && ops[b].before[a]; }
// Whether the host knows operation a to be complete.
int fake_waited(int a) { return a < (int)host.size() && host[a]; }
void fake_work(void *stream) { op("work", stream); }
int fake_priority(void *stream) { return priority.count((long)stream) ? priority[(long)stream] : 0; }
int fake_op_priority(int i) { return fake_priority((void *)ops[i].stream); }
void fake_limit(size_t bytes) { limit_bytes = bytes; }
void fake_fail_after(const char *name, int count) { failing = name, passes = count; }
void fake_fail(const char *name) { fake_fail_after(name, 0); }

// --------------------------------------------------------- the runtime --

cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { return *a = 0, *b = -5, cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { return *f = *t = (size_t)1 << 38, cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t n) {
  std::lock_guard<std::recursive_mutex> g(mu);
  *p = allocate(n);
  if (!*p) return cudaErrorMemoryAllocation;
  mem[(char *)*p] = n;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  std::lock_guard<std::recursive_mutex> g(mu);
  host.assign(ops.size(), true);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {  // waits for the device
  std::lock_guard<std::recursive_mutex> g(mu);
  if (!p) return cudaSuccess;
  cudaDeviceSynchronize();
  mem.erase((char *)p);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaLaunchHostFunc(cudaStream_t s, cudaHostFn_t f, void *arg) {
  const cudaError_t e = op("host", s);
  if (e == cudaSuccess) f(arg);
  return e;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return (*p = allocate(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  std::lock_guard<std::recursive_mutex> g(mu);
  auto it = mem.upper_bound((char *)p);
  const bool dev = it != mem.begin() && (char *)p < std::prev(it)->first + std::prev(it)->second;
  a->type = dev ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { return n < ((size_t)1 << 28) ? memset(d, v, n) : d, cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  const cudaError_t e = op(k == cudaMemcpyHostToDevice ? "to device" : k == cudaMemcpyDeviceToHost ? "to host" : "copy", st);
  if (e == cudaSuccess) memcpy(d, s, n);
  return e;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  const cudaError_t e = op("memset", st);
  if (e == cudaSuccess) memset(d, v, n);
  return e;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = (cudaStream_t)next_handle++, cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int p) {
  *s = (cudaStream_t)next_handle++;
  priority[(long)*s] = p;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(mu);
  merge(host, streams[(long)s]);
  return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(mu);
  const Set &st = streams[(long)s];
  for (size_t i = 0; i < st.size(); i++)
    if (st[i] && !fake_waited((int)i)) return cudaErrorNotReady;
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
  return *st = cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::recursive_mutex> g(mu);
  merge(streams[(long)s], events[(long)e]);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)next_handle++, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(mu);
  events[(long)e] = streams[(long)s];
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::recursive_mutex> g(mu);
  merge(host, events[(long)e]);
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }

}  // extern "C"

// --------------------------------------------------------- the kernels --

namespace sfft {

int v12_max_fft(int prec) { return prec == PREC_FP64 ? 8192 : 16384; }
int v3_max_smem_fft() { return 8192; }

cudaError_t setup_slots(const int *, int, const void *const *, int, int *, const void **, int *, cudaStream_t s) {
  return op("setup", s);
}
cudaError_t setup_slots_staged(const int *, int, const void *const *, int, int *, const void **, int *, cudaStream_t s) {
  return op("setup", s);
}
cudaError_t v12_run(const V12Dev &d, int nslots, cudaStream_t s, StageEvents *, cudaEvent_t input_read) {
  if (d.counters) memset(d.counters, 0, sizeof(int) * CNT_STRIDE * nslots);  // no results, no errors
  const bool whole = d.xs && d.J && d.sel_bits && d.score && d.hits && d.comb_bits && d.comb_list && d.counters &&
                     d.out_idx && d.out_val && d.rparams && d.inputs && (d.prec != PREC_FP64 || d.xs32) &&
                     (!d.pw || d.xs_tmp) && (!d.comb_pw || d.comb_tmp);
  const cudaError_t e = op("transform", s, whole);
  if (input_read) cudaEventRecord(input_read, s);
  return e;
}
cudaError_t v3_run(const V3Dev &d, int nslots, cudaStream_t s, StageEvents *, cudaEvent_t input_read) {
  if (d.counters) memset(d.counters, 0, sizeof(int) * CNT_STRIDE * nslots);
  const bool whole = d.man && d.man_tmp && d.g1 && d.g2 && d.est_f && d.est_v && d.map_keys && d.map_vals &&
                     d.map_table && d.counters && d.out_idx && d.out_val && d.rparams && d.inputs;
  const cudaError_t e = op("transform", s, whole);
  if (input_read) cudaEventRecord(input_read, s);
  return e;
}
cudaError_t clear_dense(void *const *, int, int, cudaStream_t s) { return op("clear", s); }
cudaError_t copy_ints(const int *src, int *dst, int count, cudaStream_t s) {
  return cudaMemcpyAsync(dst, src, sizeof(int) * count, cudaMemcpyDeviceToDevice, s);
}
cudaError_t scatter_dense(const int *, const void *, int, const int *, int, void *const *, int, cudaStream_t s) {
  return op("scatter", s);
}
cudaError_t global_fft_c128(void *, void *, int, int, long, long, int, const void *, cudaStream_t s) {
  return op("fft", s);
}

}  // namespace sfft
