/* A device made of host memory, for tests of the executor's host logic: the CUDA runtime calls and the
 * kernel launchers it uses, with streams, events and graphs whose work runs when the host waits for it
 * (or at once), and any call made to fail on demand.  "Kernels" only move bytes: a convolution of as
 * many outputs as inputs copies them, get_valid_counts keeps every row, non_max_suppression the last ones.
 */
#include "fake_device.h"

#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>
#include "cvmk_kernels.h"

namespace fake {

bool late = true;
long fail_at = 0, calls = 0, conv_plans = 0;
size_t memory_limit = 0, device_bytes = 0;
int slow_images = 0;

namespace {

struct Event { uint64_t recorded = 0, done = 0; struct Stream* where = nullptr; };
struct Op {
  std::function<void()> run;
  Event* record = nullptr;
  Event* wait = nullptr;
  uint64_t seq = 0;
};
struct Graph { std::vector<Op> ops; };
struct Stream { std::deque<Op> queue; Graph* capture = nullptr; };

std::set<Stream*> streams;
std::set<Event*> events;
std::set<Graph*> graphs;
std::map<char*, std::pair<size_t, cudaMemoryType>> memory;   // start -> bytes, kind

bool fails() { return ++calls == fail_at; }

void step(Stream* s) {   // runs the first operation of a stream, after what it waits for
  Op op = s->queue.front();
  s->queue.pop_front();
  if (op.wait)
    while (op.wait->done < op.seq) step(op.wait->where);
  if (op.run) op.run();
  if (op.record) op.record->done = op.seq;
}
void drain(Stream* s) {
  while (!s->queue.empty()) step(s);
}
void push(Stream* s, Op op) {
  if (s->capture) { s->capture->ops.push_back(std::move(op)); return; }
  s->queue.push_back(std::move(op));
  if (!late) drain(s);
}
void work(void* s, std::function<void()> f) {
  Op op;
  op.run = std::move(f);
  push((Stream*)s, std::move(op));
}
const std::pair<char* const, std::pair<size_t, cudaMemoryType>>* known(const void* p) {
  auto it = memory.upper_bound((char*)p);
  if (it == memory.begin()) return nullptr;
  --it;
  return it->first + it->second.first > (char*)p ? &*it : nullptr;
}
bool leaves_its_range(const void* p, size_t n) {
  auto* m = known(p);
  return m && (char*)p + n > m->first + m->second.first;
}
cudaError_t take(void** p, size_t n, cudaMemoryType kind) {
  if (fails()) return cudaErrorMemoryAllocation;
  if (kind == cudaMemoryTypeDevice) {
    if (memory_limit && device_bytes + n > memory_limit) return cudaErrorMemoryAllocation;
    device_bytes += n;
  }
  char* m = (char*)calloc(1, n ? n : 1);
  memory[m] = {n, kind};
  *p = m;
  return cudaSuccess;
}
cudaError_t give(void* p) {
  auto it = memory.find((char*)p);
  if (it == memory.end()) abort();
  if (it->second.second == cudaMemoryTypeDevice) device_bytes -= it->second.first;
  memory.erase(it);
  free(p);
  return cudaSuccess;
}
cudaError_t ok_or_fail() { return fails() ? cudaErrorUnknown : cudaSuccess; }
int launch(cvmk_stream_t s, std::function<void()> f) {
  if (fails()) return CVMK_ERR_CUDA;
  work(s, std::move(f));
  return CVMK_OK;
}
void images(int64_t n) {
  if (slow_images && n >= slow_images) std::this_thread::sleep_for(std::chrono::milliseconds(2));
}

// virtual memory: a reserved range is ordinary memory from the start, mapping it is bookkeeping
constexpr size_t kGranule = (size_t)64 << 10;
std::map<CUdeviceptr, size_t> reserved;
std::set<CUdeviceptr> mapped;   // granules
size_t chunks = 0;
CUresult granularity(size_t* g, const CUmemAllocationProp*, CUmemAllocationGranularity_flags) { *g = kGranule; return CUDA_SUCCESS; }
CUresult reserve(CUdeviceptr* p, size_t n, size_t, CUdeviceptr, unsigned long long) {
  if (fails()) return CUDA_ERROR_OUT_OF_MEMORY;
  *p = (CUdeviceptr)aligned_alloc(kGranule, n);
  memset((void*)*p, 0, n);
  reserved[*p] = n;
  return CUDA_SUCCESS;
}
CUresult address_free(CUdeviceptr p, size_t n) {
  for (size_t at = 0; at < n; at += kGranule)
    if (mapped.count(p + at)) return CUDA_ERROR_INVALID_VALUE;
  if (reserved[p] != n) abort();
  reserved.erase(p);
  free((void*)p);
  return CUDA_SUCCESS;
}
CUresult create(CUmemGenericAllocationHandle* h, size_t n, const CUmemAllocationProp*, unsigned long long) {
  if (fails() || (memory_limit && device_bytes + n > memory_limit)) return CUDA_ERROR_OUT_OF_MEMORY;
  device_bytes += n;
  *h = ++chunks;
  return CUDA_SUCCESS;
}
CUresult release(CUmemGenericAllocationHandle) {
  --chunks;
  device_bytes -= kGranule;
  return CUDA_SUCCESS;
}
CUresult map(CUdeviceptr p, size_t, size_t, CUmemGenericAllocationHandle, unsigned long long) {
  if (fails()) return CUDA_ERROR_UNKNOWN;
  if (!mapped.insert(p).second) abort();
  return CUDA_SUCCESS;
}
CUresult unmap(CUdeviceptr p, size_t n) {
  for (size_t at = 0; at < n; at += kGranule)
    if (!mapped.erase(p + at)) return CUDA_ERROR_INVALID_VALUE;
  return CUDA_SUCCESS;
}
CUresult set_access(CUdeviceptr, size_t, const CUmemAccessDesc*, size_t) { return fails() ? CUDA_ERROR_UNKNOWN : CUDA_SUCCESS; }

int nothing(cvmk_stream_t s) { return launch(s, [] {}); }

}  // namespace

void reset_calls(long fail) { calls = 0; fail_at = fail; }
size_t pending() {
  size_t n = 0;
  for (Stream* s : streams) n += s->queue.size();
  return n;
}
void host_register(void* p, size_t n) { memory[(char*)p] = {n, cudaMemoryTypeHost}; }
void host_unregister(void* p) { memory.erase((char*)p); }
size_t live_objects() { return streams.size() + events.size() + graphs.size() + memory.size() + reserved.size() + mapped.size() + chunks; }

}  // namespace fake

using namespace fake;

extern "C" {

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaGetDriverEntryPoint(const char* name, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  static const std::map<std::string, void*> known = {
      {"cuMemGetAllocationGranularity", (void*)granularity}, {"cuMemAddressReserve", (void*)reserve},
      {"cuMemAddressFree", (void*)address_free}, {"cuMemCreate", (void*)create}, {"cuMemRelease", (void*)release},
      {"cuMemMap", (void*)map}, {"cuMemUnmap", (void*)unmap}, {"cuMemSetAccess", (void*)set_access}};
  auto it = known.find(name);
  *fn = it == known.end() ? nullptr : it->second;
  *q = *fn ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n, cudaMemoryTypeDevice); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n, cudaMemoryTypeHost); }
cudaError_t cudaFreeHost(void* p) { return give(p); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* at, const void* p) {
  memset(at, 0, sizeof(*at));
  at->type = cudaMemoryTypeUnregistered;
  if (auto* m = known(p)) at->type = m->second.second;
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return ok_or_fail(); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { work(s, [=] { memset(p, v, n); }); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  if (fails()) return cudaErrorUnknown;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  if (fails()) return cudaErrorUnknown;
  if (leaves_its_range(d, n) || leaves_its_range(s, n)) return cudaErrorInvalidValue;
  work(st, [=] { memmove(d, s, n); });
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  if (fails()) return cudaErrorUnknown;
  Stream* t = new Stream;
  streams.insert(t);
  *s = (cudaStream_t)t;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  Stream* t = (Stream*)s;
  drain(t);
  if (t->capture) { graphs.erase(t->capture); delete t->capture; }
  streams.erase(t);
  delete t;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (fails()) return cudaErrorUnknown;
  drain((Stream*)s);
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  for (Stream* s : streams) drain(s);
  return ok_or_fail();
}
cudaError_t cudaStreamQuery(cudaStream_t s) {
  if (fails()) return cudaErrorUnknown;
  Stream* t = (Stream*)s;
  if (!t->queue.empty()) step(t);
  return t->queue.empty() ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  if (fails()) return cudaErrorUnknown;
  Op op;
  op.wait = (Event*)e;
  op.seq = op.wait->recorded;
  push((Stream*)s, op);
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  if (fails()) return cudaErrorUnknown;
  Graph* g = new Graph;
  graphs.insert(g);
  ((Stream*)s)->capture = g;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  Stream* t = (Stream*)s;
  *g = (cudaGraph_t)t->capture;
  t->capture = nullptr;
  return cudaSuccess;
}

cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (fails()) return cudaErrorUnknown;
  Event* v = new Event;
  events.insert(v);
  *e = (cudaEvent_t)v;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { events.erase((Event*)e); delete (Event*)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  if (fails()) return cudaErrorUnknown;
  Event* v = (Event*)e;
  v->where = (Stream*)s;
  Op op;
  op.record = v;
  op.seq = ++v->recorded;
  push(v->where, op);
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  if (fails()) return cudaErrorUnknown;
  Event* v = (Event*)e;
  if (v->done < v->recorded) step(v->where);
  return v->done < v->recorded ? cudaErrorNotReady : cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  if (fails()) return cudaErrorUnknown;
  Event* v = (Event*)e;
  while (v->done < v->recorded) step(v->where);
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }

cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  if (fails()) return cudaErrorUnknown;
  Graph* e = new Graph(*(Graph*)g);
  graphs.insert(e);
  *x = (cudaGraphExec_t)e;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { graphs.erase((Graph*)g); delete (Graph*)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { return cudaGraphDestroy((cudaGraph_t)g); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t g, cudaStream_t s) {
  if (fails()) return cudaErrorUnknown;
  for (const Op& op : ((Graph*)g)->ops) push((Stream*)s, op);
  return cudaSuccess;
}

// ---- kernel launchers ------------------------------------------------------------------------

const char* cvmk_last_error(void) { return "made to fail"; }

int cvmk_elemwise(const void* x, int xd, void* y, int yd, int64_t n, const cvmk_epilogue*, cvmk_stream_t s) {
  return launch(s, [=] {
    for (int64_t i = 0; i < n; ++i) {
      const int32_t v = xd == CVMK_I8 ? ((const int8_t*)x)[i] : ((const int32_t*)x)[i];
      if (yd == CVMK_I8) ((int8_t*)y)[i] = (int8_t)v;
      else ((int32_t*)y)[i] = v;
    }
  });
}
int cvmk_transpose_batched(const void* x, void* y, int32_t dtype, int64_t batch, int32_t rows, int32_t cols, int32_t, int32_t, int32_t,
                           cvmk_stream_t s) {
  return launch(s, [=] {
    memcpy(y, x, (size_t)dtype * batch * rows * cols);
    images(batch);
  });
}
int cvmk_export(const cvmk_export_segment* seg, int32_t n, cvmk_stream_t s) {
  const std::vector<cvmk_export_segment> v(seg, seg + n);
  return launch(s, [v] {
    for (const auto& e : v)
      for (int64_t r = 0; r < e.rows; ++r) memcpy((char*)e.dst + r * e.row_bytes, (const char*)e.src + r * e.src_pitch, e.row_bytes);
  });
}
int cvmk_signal(int32_t* flag, cvmk_stream_t s) { return launch(s, [flag] { *(volatile int32_t*)flag = 1; }); }

int cvmk_conv2d_tc_supported(const cvmk_conv_desc* d) { return d->C % 32 == 0 && d->OC % 8 == 0 && d->groups <= 1; }
int cvmk_conv2d_tc_prepare(const cvmk_conv_desc* d, cvmk_conv_plan* plan) {
  ++conv_plans;
  memset(plan, 0, sizeof(*plan));
  plan->d = *d;
  return fails() ? CVMK_ERR_CUDA : CVMK_OK;
}
int cvmk_conv2d_tc_launch(const cvmk_conv_plan* plan, cvmk_stream_t s) {
  const cvmk_conv_desc d = plan->d;
  const size_t in = (size_t)d.N * d.H * d.W * d.C, out = (size_t)d.N * d.OH * d.OW * d.OC * d.y_dtype;
  return launch(s, [=] {
    if (in == out) memcpy(d.y, d.x, out);
    images(d.N);
  });
}
int cvmk_conv2d_direct(const cvmk_conv_direct_desc*, cvmk_stream_t s) { return nothing(s); }
int cvmk_conv2d_stem_supported(const cvmk_stem_conv_desc*) { return 1; }
int64_t cvmk_conv2d_stem_weight_bytes(const cvmk_stem_conv_desc*) { return 64; }
int cvmk_conv2d_stem_pack_weights(const cvmk_stem_conv_desc*, const int32_t*, int8_t*) { return CVMK_OK; }
int cvmk_conv2d_stem_prepare(const cvmk_stem_conv_desc*, cvmk_stem_conv_plan*) { return CVMK_OK; }
int cvmk_conv2d_stem_launch(const cvmk_stem_conv_plan*, cvmk_stream_t s) { return nothing(s); }
int cvmk_repitch(const void*, void*, int64_t, int32_t, int32_t, cvmk_stream_t s) { return nothing(s); }
int cvmk_stem_pack_supported(const cvmk_stem_pack_desc*) { return 1; }
int cvmk_stem_pack(const cvmk_stem_pack_desc*, cvmk_stream_t s) { return nothing(s); }
int cvmk_im2col_pack(const cvmk_im2col_desc*, cvmk_stream_t s) { return nothing(s); }
int cvmk_max_pool2d(const cvmk_pool_desc*, cvmk_stream_t s) { return nothing(s); }
int cvmk_strided(const cvmk_strided_desc*, cvmk_stream_t s) { return nothing(s); }
int cvmk_strided_batch(const cvmk_strided_desc*, int32_t, cvmk_stream_t s) { return nothing(s); }
int cvmk_reduce(const cvmk_reduce_desc*, cvmk_stream_t s) { return nothing(s); }
int cvmk_take(const cvmk_take_desc*, cvmk_stream_t s) { return nothing(s); }
int cvmk_where(const cvmk_where_desc*, cvmk_stream_t s) { return nothing(s); }

int cvmk_get_valid_counts_clamped(const int32_t* x, int32_t* y, int32_t* count, int32_t B, int32_t N, int32_t K, int32_t, int32_t,
                                  cvmk_stream_t s) {
  return launch(s, [=] {
    memcpy(y, x, (size_t)B * N * K * 4);
    std::fill(count, count + B, N);
  });
}
int64_t cvmk_nms_scratch_bytes(int32_t, int32_t) { return 64; }
int cvmk_non_max_suppression_part(const cvmk_nms_desc* p, int32_t first, int32_t n, cvmk_stream_t s) {
  const cvmk_nms_desc d = *p;
  return launch(s, [=] {
    const size_t rows = std::min(d.N, d.top_k);
    for (int32_t b = first; b < first + n; ++b) {
      const size_t at = (size_t)b * d.N * 6;
      memset(d.y + at, 0xff, (size_t)d.N * 24);
      memcpy(d.y + at, d.x + at + (d.N - rows) * 6, rows * 24);
    }
  });
}
int cvmk_non_max_suppression(const cvmk_nms_desc* d, cvmk_stream_t s) { return cvmk_non_max_suppression_part(d, 0, d->B, s); }

}  // extern "C"
