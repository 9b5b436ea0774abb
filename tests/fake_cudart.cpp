// fake_cudart.cpp -- a CUDA runtime without a GPU, for tests of the library's
// host code: device memory is host memory, copies and fills are done at once,
// kernels are not run.  What the host code asks for is written to a log, and a
// test can make the n-th call of a function fail.
// Linked with the library's own objects instead of the CUDA runtime.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Op {
  char what[24];
  int64_t a, b;  // stream or event numbers
};
std::vector<Op> ops;
std::map<std::string, int> fail_after;  // function -> successful calls before the one that fails
std::map<void*, size_t> blocks;
int64_t live = 0;
cudaError_t last = cudaSuccess;
int64_t numbers = 0;
std::map<const void*, std::string> names;  // kernels by the address of their host stub
std::string watched;
int watched_arg = 0;
uint64_t watched_value = 0;

cudaError_t step(const char* what, const void* a = nullptr, const void* b = nullptr);
cudaError_t launch(const void* f, void** args, cudaStream_t st) {
  auto n = names.find(f);
  if (!watched.empty() && n != names.end() && n->second.find(watched) != std::string::npos)
    memcpy(&watched_value, args[watched_arg], 8);
  return step("launch", st);
}

int64_t id(const void* p) { return (int64_t)(intptr_t)p; }
void* handle() { return (void*)(intptr_t)++numbers; }
cudaError_t step(const char* what, const void* a, const void* b) {
  auto f = fail_after.find(what);
  if (f != fail_after.end() && f->second-- == 0) {
    fail_after.erase(f);
    return last = cudaErrorMemoryAllocation;
  }
  Op o{{0}, id(a), id(b)};
  strncpy(o.what, what, sizeof(o.what) - 1);
  ops.push_back(o);
  return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- the test's side
void fake_reset() { ops.clear(); fail_after.clear(); last = cudaSuccess; watched.clear(); }
void fake_fail(const char* what, int n) { fail_after[what] = n; }
int fake_failed(const char* what) { return !fail_after.count(what); }
int64_t fake_live_bytes() { return live; }
// the 8 bytes of argument `arg` of the kernel whose name holds `name`, at its last launch
void fake_watch(const char* name, int arg) { watched = name; watched_arg = arg; watched_value = 0; }
uint64_t fake_watched() { return watched_value; }
// bytes from p to the end of the allocation that holds it (0: none does)
int64_t fake_room(uint64_t p) {
  for (auto& b : blocks) {
    const uint64_t lo = (uint64_t)(uintptr_t)b.first;
    if (p >= lo && p < lo + b.second) return (int64_t)(lo + b.second - p);
  }
  return 0;
}
int fake_ops() { return (int)ops.size(); }
const char* fake_op(int k, int64_t* a, int64_t* b) { *a = ops[k].a; *b = ops[k].b; return ops[k].what; }

// ---- registration of the compiled kernels
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static thread_local cudaStream_t pushed;
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t st) { pushed = st; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void* st) { *(cudaStream_t*)st = pushed; return cudaSuccess; }
cudaError_t __cudaGetKernel(void** k, const void* f) { *k = (void*)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(void* k, dim3, dim3, void** args, size_t, cudaStream_t st) { return launch(k, args, st); }

// ---- the runtime
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) { return launch(f, args, c->stream); }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t st) { return launch(f, args, st); }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (cudaError_t e = step("malloc")) return e;
  *p = aligned_alloc(256, (n + 255) / 256 * 256);
  memset(*p, 0, n);
  blocks[*p] = n;
  live += (int64_t)n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (blocks.count(p)) {
    live -= (int64_t)blocks[p];
    blocks.erase(p);
    free(p);
  }
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostRegister(void*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  if (cudaError_t e = step("copy", st)) return e;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  if (cudaError_t e = step("fill", st)) return e;
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 38; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return cudaMalloc(p, 1 << 22); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeHost;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 152;
  p->major = 10;
  p->minor = 3;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { *lo = 0; *hi = -5; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 8;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = 8; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)handle(); return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int priority) {
  *s = (cudaStream_t)handle();
  return step("stream", *s, (void*)(intptr_t)priority);
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) { return step("sync", st); }
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) { return step("wait", st, e); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)handle(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)handle(); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) { return step("record", st, e); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t st, cudaStreamCaptureMode) {
  return step("begin capture", st);
}
cudaError_t cudaStreamEndCapture(cudaStream_t st, cudaGraph_t* g) {
  *g = nullptr;
  if (cudaError_t e = step("end capture", st)) return e;
  *g = (cudaGraph_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  if (cudaError_t e = step("instantiate")) return e;
  *x = (cudaGraphExec_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t st) { return step("graph", st, x); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t*, size_t* n) { *n = 0; return cudaSuccess; }
}
