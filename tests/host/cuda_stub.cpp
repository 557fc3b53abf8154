// The CUDA runtime calls that the library makes, without a device: memory is host
// memory, copies and memsets are done at once, a kernel launch is logged and does
// nothing, streams, events and captured graphs only keep track of order.  The host
// code of the library is linked against this to test what it does around launches:
// allocation failures, the order of frames over streams, what a replay draws.
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "cuda_stub.h"

namespace {

using Clock = std::map<int, long>;   // stream -> operations of it known to be over

void merge(Clock& a, const Clock& b)
{
  for (auto& kv : b) a[kv.first] = std::max(a[kv.first], kv.second);
}

struct Graph { std::vector<std::function<void(int)>> ops; };   // (each run on the stream of its launch)

struct Stream {
  int id;
  Clock clock;
  long seq = 0;
  Graph* capture = nullptr;
  bool gone = false;
};
struct Event { Clock clock; Graph* capture = nullptr; };

std::recursive_mutex mu;
// (kernels register before this file's own objects are constructed)
std::map<const void*, std::string>& names() { static auto* m = new std::map<const void*, std::string>(); return *m; }
std::map<const void*, size_t>& vars() { static auto* m = new std::map<const void*, size_t>(); return *m; }
std::map<int, Stream*> streams;
Clock host_clock;
std::string log_text;
std::map<const void*, std::pair<int, long>> last_use;  // working counters -> last launch on them
std::map<const void*, void*> var_mem;
int fail_skip = -1, fail_count = 0, overflows = 0;
thread_local cudaError_t last_error = cudaSuccess;
thread_local struct { dim3 grid, block; size_t smem; cudaStream_t st; } pushed;
int next_stream = 1;
Stream legacy{0};

void say(const std::string& s) { log_text += s + "\n"; }

Stream& at(cudaStream_t st)
{
  Stream& s = st ? *reinterpret_cast<Stream*>(st) : legacy;
  if (s.gone) say("GONE stream " + std::to_string(s.id));
  return s;
}

cudaError_t fail(cudaError_t e)
{
  last_error = e;
  return e;
}

bool allocation_fails()
{
  if (fail_skip < 0) return false;
  if (fail_skip > 0) { --fail_skip; return false; }
  if (fail_count-- > 0) return true;
  fail_skip = -1;
  return false;
}

// One operation on a stream: recorded while it is captured, else done now.
void enqueue(cudaStream_t st, std::function<void(int)> op)
{
  Stream& s = at(st);
  if (s.capture) { s.capture->ops.push_back(op); return; }
  merge(s.clock, host_clock);
  s.clock[s.id] = ++s.seq;
  op(s.id);
}

void run_launch(const std::string& name, const StubLaunch& l, int stream)
{
  Stream* s = stream ? streams[stream] : &legacy;
  std::string line = "launch " + name + " stream " + std::to_string(stream);
  for (float c : l.cameras()) { char b[32]; snprintf(b, sizeof(b), " %g", c); line += b; }
  say(line);
  if (l.null_argument) say("NULL argument of " + name);
  if (name == "raster_frag8" || name == "raster_bins") l.counts(overflows > 0 && overflows-- > 0);
  if (name == "reyes_pixels") l.counts(false);
  for (const void* o : l.objects) {
    auto& u = last_use[o];
    if (u.second && s->clock[u.first] < u.second) say("RACE " + name + " stream " + std::to_string(stream));
    u = {s->id, s->clock[s->id]};
  }
}

cudaError_t launch(const void* func, void** args, cudaStream_t st)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  const std::string name = names()[func];
  auto l = std::make_shared<StubLaunch>(stub_decode(name.c_str(), args));
  enqueue(st, [=](int s) { run_launch(name, *l, s); });
  return cudaSuccess;
}

cudaError_t allocate(void** p, size_t n)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (allocation_fails()) return fail(cudaErrorMemoryAllocation);
  *p = calloc(1, n ? n : 1);
  return *p ? cudaSuccess : fail(cudaErrorMemoryAllocation);
}

}  // namespace

extern "C" {

// ------------------------------------------------------------------ for the tests
// The count allocations after the next skip ones fail.
void stub_fail_alloc(int skip, int count)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  fail_skip = skip;
  fail_count = count;
}
// The next n raster frames report that their lists overflowed.
void stub_overflow(int n)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  overflows = n;
}
// The next Reyes frame reports so many patches on a frontier, leaves, and that one did not fit.
void stub_patches(unsigned frontier, unsigned leaves)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  stub_frontier = frontier;
  stub_leaves = leaves;
}
int stub_log(char* out, int size)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  snprintf(out, (size_t)size, "%s", log_text.c_str());
  const int n = (int)log_text.size();
  log_text.clear();
  return n;
}
void stub_destroy_stream(void* s) { cudaStreamDestroy(reinterpret_cast<cudaStream_t>(s)); }
// A capture of what the caller enqueues on the stream; stub_end_capture gives a graph to launch.
void stub_begin_capture(void* s) { cudaStreamBeginCapture(reinterpret_cast<cudaStream_t>(s), cudaStreamCaptureModeGlobal); }
void* stub_end_capture(void* s)
{
  cudaGraph_t g;
  cudaStreamEndCapture(reinterpret_cast<cudaStream_t>(s), &g);
  return g;
}
void stub_replay(void* g, void* s)
{
  cudaGraphLaunch(reinterpret_cast<cudaGraphExec_t>(g), reinterpret_cast<cudaStream_t>(s));
}
void* stub_stream()
{
  cudaStream_t s;
  cudaStreamCreateWithFlags(&s, 0);
  return s;
}

// ------------------------------------------------------------------ runtime API
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last_error; last_error = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
  *n = 4;
  return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (!d || !s) return fail(cudaErrorInvalidValue);
  enqueue(st, [=](int) { memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (!d) return fail(cudaErrorInvalidValue);
  enqueue(st, [=](int s) { memset(d, v, n); say("memset stream " + std::to_string(s)); });
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* sym)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (!var_mem[sym]) var_mem[sym] = calloc(1, vars()[sym]);
  *p = var_mem[sym];
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  Stream* n = new Stream{next_stream++};
  streams[n->id] = n;
  *s = reinterpret_cast<cudaStream_t>(n);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t st)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  at(st).gone = true;   // (kept: clocks refer to it; what it was given goes on)
  return cudaSuccess;
}
cudaError_t cudaStreamGetId(cudaStream_t st, unsigned long long* id)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  *id = (unsigned long long)at(st).id;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (at(st).capture) return fail(cudaErrorStreamCaptureUnsupported);
  merge(host_clock, at(st).clock);
  return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t st) { return cudaStreamSynchronize(st); }
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t ev, unsigned)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  Stream& s = at(st);
  Event* e = reinterpret_cast<Event*>(ev);
  if (e->capture) { s.capture = e->capture; return cudaSuccess; }
  if (s.capture) return fail(cudaErrorStreamCaptureIsolation);
  merge(s.clock, e->clock);
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t st, cudaStreamCaptureStatus* o)
{
  *o = at(st).capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t st, cudaStreamCaptureMode)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  at(st).capture = new Graph();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t st, cudaGraph_t* g)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  Graph* c = at(st).capture;
  for (auto& kv : streams)
    if (kv.second->capture == c) kv.second->capture = nullptr;
  *g = reinterpret_cast<cudaGraph_t>(c);
  say("captured");
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long)
{
  *x = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph*>(g)));
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t st)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  for (auto& op : reinterpret_cast<Graph*>(x)->ops) enqueue(st, op);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<Graph*>(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete reinterpret_cast<Graph*>(x); return cudaSuccess; }

cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(new Event()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t st)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  Event* e = reinterpret_cast<Event*>(ev);
  Stream& s = at(st);
  e->capture = s.capture;
  if (!s.capture) { merge(s.clock, host_clock); e->clock = s.clock; }
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t ev)
{
  std::lock_guard<std::recursive_mutex> lk(mu);
  merge(host_clock, reinterpret_cast<Event*>(ev)->clock);
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t st) { return launch(f, args, st); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) { return launch(f, args, c->stream); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t st)
{
  return launch(f, args, st);
}

// ------------------------------------------------------------------ what compiled launches call
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st)
{
  pushed = {grid, block, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st)
{
  *grid = pushed.grid;
  *block = pushed.block;
  *smem = pushed.smem;
  *static_cast<cudaStream_t*>(st) = pushed.st;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 0; }
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, void*, void*, void*, void*, int*)
{
  names()[f] = stub_kernel_name(name);
}
void __cudaRegisterVar(void**, char* var, char*, const char*, int, size_t size, int, int)
{
  vars()[var] = size;
}

}  // extern "C"
