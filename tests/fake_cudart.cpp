// A CUDA runtime on host memory, preloaded in place of libcudart by test_host_calls.py: it
// records the library's calls in order, copies really, launches nothing, and can refuse
// a launch by kernel name or change what a device-to-host copy brings back.  For
// what the library's host code does before, between and after its launches.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <string>
#include <vector>

static std::string g_log, g_refused;
static std::map<const void*, std::string> g_names;
static size_t g_poke_size = 0;
static std::vector<std::pair<size_t, unsigned long long>> g_pokes;
static long g_handles = 0, g_calls = 0;

static void note(const char* what, const std::string& name, const void* src, cudaStream_t st) {
  char b[96];
  snprintf(b, sizeof(b), " %p %p\n", src, (void*)st);
  g_log += std::string(what) + " " + name + b;
  ++g_calls;
}

extern "C" {
const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }
void fake_refuse(const char* kernel) { g_refused = kernel; }
// from now on a device-to-host copy of `size` bytes brings `value` at `offset`
void fake_poke(size_t size, size_t offset, unsigned long long value) {
  g_poke_size = size;
  g_pokes.push_back({offset, value});
}

void** __cudaRegisterFatBinary(void*) { return (void**)&g_handles; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  g_names[host] = name;
}
static dim3 g_grid, g_block;
static size_t g_smem;
static cudaStream_t g_stream;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
  g_grid = g; g_block = b; g_smem = s; g_stream = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
  *g = g_grid; *b = g_block; *s = g_smem; *(cudaStream_t*)st = g_stream;
  return cudaSuccess;
}
static cudaError_t g_last = cudaSuccess;
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t st) {
  const std::string& n = g_names[f];
  const bool no = !g_refused.empty() && n.find(g_refused) != std::string::npos;
  note(no ? "refused" : "launch", n, nullptr, st);
  if (no) g_last = cudaErrorInvalidValue;
  return no ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_last; }
const char* cudaGetErrorString(cudaError_t) { return "refused"; }

cudaError_t cudaMalloc(void** p, size_t n) { *p = calloc(n ? n : 1, 1); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
static cudaError_t copy(const char* what, void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  note(what, k == cudaMemcpyHostToDevice ? "h2d" : k == cudaMemcpyDeviceToHost ? "d2h" : "d2d", s, st);
  memcpy(d, s, n);
  if (k == cudaMemcpyDeviceToHost && n == g_poke_size)
    for (auto& p : g_pokes) memcpy((char*)d + p.first, &p.second, 8);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return copy("cudaMemcpy", d, s, n, k, 0); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  return copy("cudaMemcpyAsync", d, s, n, k, st);
}
cudaError_t cudaMemset(void* d, int v, size_t n) { note("cudaMemset", "set", d, 0); memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  note("cudaMemsetAsync", "set", d, st);
  memset(d, v, n);
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)++g_handles; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { note("cudaStreamSynchronize", "-", nullptr, s); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { note("cudaDeviceSynchronize", "-", nullptr, 0); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { note("cudaStreamWaitEvent", "-", e, s); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)++g_handles; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
// an event's time is the number of calls before it
static std::map<cudaEvent_t, long> g_time;
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  note("cudaEventRecord", "-", e, s);
  g_time[e] = g_calls;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) { *ms = g_time[b] - g_time[a]; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 232448;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = (void*)s; return cudaSuccess; }
}
