// A CUDA runtime on the CPU for tests of the library's host side: device memory
// is host memory, copies and memsets are done at once, kernels only leave a line
// in a log, graphs replay what was captured.  fake_fail makes one later call fail,
// so that error paths run without a GPU.  The library's objects are linked against
// this file in place of the runtime (test_failed_calls.py).
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace {

using Ops = std::vector<std::function<cudaError_t()>>;
struct Graph {
  Ops ops;
};

std::map<const void *, std::string> kernel_names;
std::map<const void *, size_t> symbol_sizes;
std::map<const void *, void *> symbols;
std::set<const void *> pinned;
Graph *capturing = nullptr;
cudaError_t last_error = cudaSuccess;
std::string log_text;
std::vector<std::pair<std::string, long>> failures;  // armed: part of a log line, calls to go
struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t st;
} config;

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) last_error = e;
  return e;
}

// A call: logged, and failed if fake_fail has armed it.
cudaError_t call(const std::string &what) {
  log_text += what + "\n";
  bool fails = false;
  for (auto &f : failures)
    if (f.second > 0 && what.find(f.first) != std::string::npos && --f.second == 0) fails = true;
  if (!fails) return cudaSuccess;
  log_text += "failed\n";
  return done(what.compare(0, 6, "malloc") == 0 ? cudaErrorMemoryAllocation : cudaErrorInvalidConfiguration);
}

// Work on a stream: done now, or recorded while a stream is captured.
cudaError_t work(const std::string &what, std::function<void()> fn) {
  if (capturing) {
    cudaError_t e = call("capture " + what);
    if (e != cudaSuccess) return e;
    capturing->ops.push_back([=] {
      cudaError_t r = call(what);
      if (r == cudaSuccess) fn();
      return r;
    });
    return cudaSuccess;
  }
  cudaError_t e = call(what);
  if (e == cudaSuccess) fn();
  return e;
}

cudaError_t launch(const void *fn) { return work("launch " + kernel_names[fn], [] {}); }
cudaError_t alloc(void **p, size_t bytes) {
  cudaError_t e = call("malloc " + std::to_string(bytes));
  if (e == cudaSuccess) *p = std::calloc(bytes ? bytes : 1, 1);
  return e;
}
int encode_stub() { return 0; }

}  // namespace

extern "C" {

// The nth call from now on whose log line contains `what` fails.
void fake_fail(const char *what, long nth) { failures.push_back({what, nth}); }
void fake_fail_none() { failures.clear(); }
const char *fake_log() { return log_text.c_str(); }
void fake_log_clear() { log_text.clear(); }

// --- what nvcc's host code calls -------------------------------------------
void **__cudaRegisterFatBinary(void *) {
  static void *handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  kernel_names[host] = name;
}
void __cudaRegisterVar(void **, char *host, char *, const char *, int, size_t size, int, int) { symbol_sizes[host] = size; }
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn) {
  *k = (cudaKernel_t) const_cast<void *>(fn);
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
  config = {grid, block, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *st) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *(cudaStream_t *)st = config.st;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **, size_t, cudaStream_t) { return launch((const void *)k); }

// --- the runtime -------------------------------------------------------------
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *fn, void **) { return launch(fn); }
cudaError_t cudaGetLastError() {
  cudaError_t e = last_error;
  last_error = cudaSuccess;
  return e;
}
cudaError_t cudaGetDeviceCount(int *n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrComputeCapabilityMajor ? 10 : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
  std::memset(a, 0, sizeof *a);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *symbol) {
  if (!symbols[symbol]) symbols[symbol] = std::calloc(symbol_sizes[symbol] + 1, 1);
  *p = symbols[symbol];
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **fn, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *r) {
  *fn = (void *)encode_stub;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t bytes) { return alloc(p, bytes); }
cudaError_t cudaFree(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t bytes) {
  cudaError_t e = alloc(p, bytes);
  if (e == cudaSuccess) pinned.insert(*p);
  return e;
}
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { return cudaMallocHost(p, bytes); }
cudaError_t cudaFreeHost(void *p) {
  pinned.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  std::memset(a, 0, sizeof *a);
  if (pinned.count(p)) {
    a->type = cudaMemoryTypeHost;
    a->devicePointer = a->hostPointer = const_cast<void *>(p);
  }
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
  return work("memset " + std::to_string(n), [=] { std::memset(p, v, n); });
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return work("memcpy " + std::to_string(n), [=] { std::memmove(d, s, n); });
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t) new int;
  return call("stream");
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  delete (int *)s;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return call("synchronize"); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = (cudaEvent_t) new int;
  return call("event");
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete (int *)e;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}

cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
  *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  capturing = new Graph();
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t g, const cudaGraphNode_t *,
                                          const cudaGraphEdgeData *, size_t, cudaStreamCaptureMode) {
  capturing = (Graph *)g;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = (cudaGraph_t)capturing;
  capturing = nullptr;
  return call("end of capture");
}
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus *s, unsigned long long *, cudaGraph_t *,
                                     const cudaGraphNode_t **deps, const cudaGraphEdgeData **, size_t *n) {
  *s = cudaStreamCaptureStatusActive;
  if (deps) *deps = nullptr;
  if (n) *n = 0;
  return cudaSuccess;
}
cudaError_t cudaGraphCreate(cudaGraph_t *g, unsigned) {
  *g = (cudaGraph_t) new Graph();
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete (Graph *)g;
  return cudaSuccess;
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned) {
  *h = 0;
  return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t *node, cudaGraph_t g, const cudaGraphNode_t *, const cudaGraphEdgeData *,
                             size_t, cudaGraphNodeParams *p) {  // a conditional node: its body runs once
  Graph *body = new Graph();
  cudaGraph_t *out = new cudaGraph_t((cudaGraph_t)body);
  p->conditional.phGraph_out = out;
  *node = (cudaGraphNode_t)out;
  ((Graph *)g)->ops.push_back([body] {
    for (auto &op : body->ops)
      if (cudaError_t e = op()) return e;
    return cudaSuccess;
  });
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
  cudaError_t e = call("instantiate");
  if (e == cudaSuccess) *x = (cudaGraphExec_t) new Graph(*(Graph *)g);
  return e;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  delete (Graph *)x;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  cudaError_t e = call("replay");
  for (auto &op : ((Graph *)x)->ops)
    if (e == cudaSuccess) e = op();
  return e;
}

}  // extern "C"
