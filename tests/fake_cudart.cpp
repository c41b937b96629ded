// A CUDA runtime that runs nothing: device memory is host memory, copies and
// memsets happen at once, kernels do not.  Every stream-ordered call is
// logged, and a test can make a chosen call fail or choose the words of the
// status that a frame reads back.  Preloaded before the runtime, it lets the
// host code of libvct.so run without a GPU.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
std::string g_log, g_fail;
int g_fail_after = -1;  // matching calls until the one that fails (-1: none)
std::map<const void*, std::string> g_kernels;
std::map<int, unsigned> g_status;  // word -> value of the status copies
size_t g_status_bytes = 0;
size_t g_ids = 0;

void* handle() { return (void*)(0x1000 + 16 * ++g_ids); }

cudaError_t note(const char* what, const std::string& rest, cudaError_t error = cudaErrorUnknown) {
  const std::string line = std::string(what) + " " + rest;
  const bool fails = g_fail_after >= 0 && line.find(g_fail) != std::string::npos && g_fail_after-- == 0;
  g_log += line + (fails ? " FAILED\n" : "\n");
  return fails ? error : cudaSuccess;
}
std::string hex(const void* p) {
  char b[32];
  std::snprintf(b, sizeof(b), "%llx", (unsigned long long)(size_t)p);
  return b;
}
cudaError_t copy(const char* what, void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  const cudaError_t e = note(what, hex(d) + " " + std::to_string(n) + " stream " + hex(st));
  if (e != cudaSuccess) return e;
  std::memcpy(d, s, n);
  if (k == cudaMemcpyDeviceToHost && n == g_status_bytes)
    for (const auto& w : g_status) static_cast<unsigned*>(d)[w.first] = w.second;
  return cudaSuccess;
}
cudaError_t launch(const void* f, void** args, size_t smem, cudaStream_t st) {
  // k_bin's large-triangle records and their capacity
  if (g_kernels[f].find("5k_binILb") != std::string::npos)
    g_log += "records " + hex(*static_cast<void**>(args[7])) + " " + std::to_string(*static_cast<unsigned*>(args[8])) + "\n";
  return note("launch", g_kernels[f] + " smem " + std::to_string(smem) + " stream " + hex(st), cudaErrorLaunchOutOfResources);
}
cudaError_t g_last = cudaSuccess;
dim3 g_grid, g_block;
size_t g_smem;
cudaStream_t g_stream;
CUresult encode_tiled(...) { return CUDA_SUCCESS; }
}  // namespace

extern "C" {
// ---- the test's side ----
const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }
void fake_fail(const char* text, int after) {
  g_fail = text;
  g_fail_after = after;
}
void fake_status(int bytes, int word, unsigned value) {
  g_status_bytes = (size_t)bytes;
  g_status[word] = value;
}

// ---- registration and launches ----
void** __cudaRegisterFatBinary(void*) { return (void**)handle(); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_kernels[host] = name;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
  g_grid = g;
  g_block = b;
  g_smem = smem;
  g_stream = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = g_grid;
  *b = g_block;
  *smem = g_smem;
  *(cudaStream_t*)st = g_stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** args, size_t smem, cudaStream_t st) {
  const cudaError_t e = launch((const void*)k, args, smem, st);
  if (e != cudaSuccess) g_last = e;  // (a plain launch reports by cudaGetLastError)
  return e;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  const cudaError_t e = launch(f, args, c->dynamicSmemBytes, c->stream);
  if (e != cudaSuccess) g_last = e;
  return e;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  return note("attribute", g_kernels[f] + " " + std::to_string((int)a) + " " + std::to_string(v));
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
  *n = 4;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 4;
  return cudaSuccess;
}

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t n) {
  const cudaError_t e = note("malloc", std::to_string(n), cudaErrorMemoryAllocation);
  *p = e == cudaSuccess ? std::calloc(1, n) : nullptr;
  if (*p) g_log += "at " + hex(*p) + "\n";
  return e;
}
cudaError_t cudaFree(void* p) {
  note("free", hex(p));
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  return copy("synchronous-copy", d, s, n, k, nullptr);
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  return copy("copy", d, s, n, k, st);
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
  const cudaError_t e = note("memset", hex(p) + " " + std::to_string(n) + " to " + std::to_string(v) + " stream " + hex(st));
  if (e == cudaSuccess) std::memset(p, v, n);
  return e;
}
cudaError_t cudaMemcpy3D(const cudaMemcpy3DParms*) { return cudaSuccess; }
cudaError_t cudaMemcpy3DAsync(const cudaMemcpy3DParms*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = const_cast<void*>(s);
  return cudaSuccess;
}

// ---- arrays, textures, surfaces: handles ----
cudaError_t cudaMalloc3DArray(cudaArray_t* a, const cudaChannelFormatDesc*, cudaExtent, unsigned) {
  *a = (cudaArray_t)handle();
  return note("malloc3d", "", cudaErrorMemoryAllocation);
}
cudaError_t cudaMallocMipmappedArray(cudaMipmappedArray_t* a, const cudaChannelFormatDesc*, cudaExtent, unsigned,
                                     unsigned) {
  *a = (cudaMipmappedArray_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGetMipmappedArrayLevel(cudaArray_t* a, cudaMipmappedArray_const_t, unsigned) {
  *a = (cudaArray_t)handle();
  return cudaSuccess;
}
cudaError_t cudaFreeArray(cudaArray_t) { return cudaSuccess; }
cudaError_t cudaFreeMipmappedArray(cudaMipmappedArray_t) { return cudaSuccess; }
cudaError_t cudaCreateSurfaceObject(cudaSurfaceObject_t* s, const cudaResourceDesc*) {
  *s = (cudaSurfaceObject_t)(size_t)handle();
  return cudaSuccess;
}
cudaError_t cudaCreateTextureObject(cudaTextureObject_t* t, const cudaResourceDesc*, const cudaTextureDesc*,
                                    const cudaResourceViewDesc*) {
  *t = (cudaTextureObject_t)(size_t)handle();
  return cudaSuccess;
}
cudaError_t cudaDestroySurfaceObject(cudaSurfaceObject_t) { return cudaSuccess; }
cudaError_t cudaDestroyTextureObject(cudaTextureObject_t) { return cudaSuccess; }
cudaChannelFormatDesc cudaCreateChannelDesc(int x, int y, int z, int w, cudaChannelFormatKind f) {
  return {x, y, z, w, f};
}

// ---- streams, events, graphs ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)handle();
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return note("sync", "stream " + hex(s)); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t, unsigned) { return note("wait", "stream " + hex(s)); }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)handle();
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) { return note("record", "stream " + hex(s)); }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t s, unsigned) { return note("record", "stream " + hex(s)); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaErrorNotReady; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { return note("capture", "stream " + hex(s)); }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  *g = (cudaGraph_t)handle();
  return note("captured", "stream " + hex(s));
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return note("graph", "dropped"); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { return note("replay", "stream " + hex(s)); }

// ---- device and errors ----
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) {
  *least = 0;
  *greatest = -1;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** fn, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *fn = (void*)encode_tiled;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "made to fail"; }
}
