// A stand-in for the CUDA runtime that records instead of running: linked with
// the library's own objects it shows, without a GPU, what a call puts on
// which stream and in which order.  "Device" memory is host memory, copies and
// clears are done at once, kernels are only logged, except that k_advance's
// step counter moves (closed boxes count their steps there), so that the
// calls see the steps they launched.
//
// The log is one line per operation, "op stream rest":
//   launch S name gx gy gz pdl   kernel launch (pdl 1: programmatic dependent)
//   set S bytes / copy S bytes   asynchronous clear / copy
//   blockcopy 0 bytes in|out     cudaMemcpy (the default stream), to or from the device
//   record S event external      wait S event
//   graph S exec                 sync S (the host waits for stream S)
//   begin S / end S exec         capture (what lies between is in the graph)
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
std::string g_log;
// kernels are registered before this unit's own statics are made
std::map<const void *, std::string> &names() { static std::map<const void *, std::string> m; return m; }
std::map<long, std::vector<int *>> g_counters;     // exec -> step counters its graph advances
std::vector<int *> g_captured;
bool g_capturing = false;
long g_next = 1, g_graph = 0;
struct Call { dim3 grid, block; size_t shm; cudaStream_t st; } g_call;

template <class T>
cudaError_t handle(T *out) { *out = (T)(g_next++); return cudaSuccess; }
void log(const char *op, const void *st, const std::string &rest = "") {
  g_log += std::string(op) + " " + std::to_string((long)st) + (rest.empty() ? "" : " " + rest) + "\n";
}
cudaError_t alloc(void **p, size_t n) { *p = std::calloc(n ? n : 1, 1); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t launched(const void *f, dim3 g, cudaStream_t st, void **args, int pdl) {
  const std::string &name = names()[f];
  log("launch", st, name + " " + std::to_string(g.x) + " " + std::to_string(g.y) + " " + std::to_string(g.z) + " " + std::to_string(pdl));
  if (name.find("k_advance") != std::string::npos) {
    int *it = *(int **)args[0];
    if (g_capturing) g_captured.push_back(it);
    else ++*it;
  }
  // the documented limits of a launch's grid
  return g.y > 65535 || g.z > 65535 ? cudaErrorInvalidConfiguration : cudaSuccess;
}
cudaError_t g_last = cudaSuccess;
cudaError_t keep(cudaError_t e) { if (e != cudaSuccess) g_last = e; return e; }
}  // namespace

extern "C" {

const char *recording_log() { return g_log.c_str(); }
void recording_clear() { g_log.clear(); }

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, void *, void *, void *, void *, int *) { names()[f] = name; }
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t shm, cudaStream_t st) { g_call = { g, b, shm, st }; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *shm, void *st) {
  *g = g_call.grid; *b = g_call.block; *shm = g_call.shm; *(cudaStream_t *)st = g_call.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3, void **args, size_t, cudaStream_t st) { return keep(launched(f, g, st, args, 0)); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
  int pdl = 0;
  for (unsigned n = 0; n < c->numAttrs; n++)
    if (c->attrs[n].id == cudaLaunchAttributeProgrammaticStreamSerialization) pdl = c->attrs[n].val.programmaticStreamSerializationAllowed;
  return keep(launched(f, c->gridDim, c->stream, args, pdl));
}

cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) { return handle(p); }
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = 0; *hi = -1; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "recorded error"; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { static float x; *p = &x; return cudaSuccess; }

cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return alloc(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return alloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  std::memcpy(d, s, n);
  log("blockcopy", nullptr, std::to_string(n) + (k == cudaMemcpyDeviceToHost ? " out" : " in"));
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) { std::memcpy(d, s, n); log("copy", st, std::to_string(n)); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) { std::memset(d, v, n); log("set", st, std::to_string(n)); return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { log("sync", s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { log("wait", s, std::to_string((long)e)); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { log("record", s, std::to_string((long)e) + " 0"); return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned f) {
  log("record", s, std::to_string((long)e) + (f & cudaEventRecordExternal ? " 1" : " 0"));
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { g_capturing = true; g_captured.clear(); log("begin", s); return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
  g_capturing = false;
  handle(g);
  g_graph = (long)*g;
  log("end", s, std::to_string(g_graph));
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) { *x = (cudaGraphExec_t)g; g_counters[(long)g] = g_captured; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  for (int *it : g_counters[(long)x]) ++*it;
  log("graph", s, std::to_string((long)x));
  return cudaSuccess;
}

}  // extern "C"
