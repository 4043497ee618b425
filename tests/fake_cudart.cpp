// A CUDA runtime without a GPU, preloaded over the library's: memory is host
// memory, nothing runs, every stream operation is logged, and one launch,
// asynchronous memset or allocation (or all from one on) can be made to fail.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

static std::map<const void*, std::string>& kernels() {
    static std::map<const void*, std::string> m;
    return m;
}
static std::string g_log;
static long g_next = 1, g_launch = 0, g_fail_launch = -1, g_memset = 0, g_fail_memset = -1;
static long g_malloc = 0, g_fail_malloc_from = -1, g_fail_malloc_to = -1;
static cudaError_t g_last = cudaSuccess;
static struct { dim3 g, b; size_t s; cudaStream_t st; } g_call;

static cudaError_t set(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}
static void log(const char* what, cudaStream_t st, const std::string& arg) {
    g_log += what + std::string(" ") + std::to_string((long)st) + " " + arg + "\n";
}
static cudaError_t launch(const void* f, cudaStream_t st) {
    const bool bad = g_launch++ == g_fail_launch;
    log(bad ? "fail" : "launch", st, kernels()[f]);
    return set(bad ? cudaErrorMemoryAllocation : cudaSuccess);
}

extern "C" {
void fake_reset(long fail_launch, long fail_memset) {
    g_log.clear();
    g_launch = g_memset = 0;
    g_fail_launch = fail_launch;
    g_fail_memset = fail_memset;
}
void fake_fail_mallocs(long from, long to) {  // [from, to) counted from here
    g_malloc = 0;
    g_fail_malloc_from = from;
    g_fail_malloc_to = to;
}
const char* fake_log() { return g_log.c_str(); }

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, void*, void*, void*, void*, int*) {
    kernels()[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
    g_call = {g, b, s, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
    *g = g_call.g;
    *b = g_call.b;
    *s = g_call.s;
    *(cudaStream_t*)st = g_call.st;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t st) { return launch(f, st); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return launch(f, c->stream); }
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaMalloc(void** p, size_t n) {
    const long k = g_malloc++;
    *p = k >= g_fail_malloc_from && k < g_fail_malloc_to ? nullptr : calloc(1, n ? n : 1);
    return set(*p ? cudaSuccess : cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    log("blocking-copy", nullptr, std::to_string(n));
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
    log("default-stream-memset", nullptr, std::to_string(n));
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    log("copy", st, std::to_string(n));
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) {
    return set(cudaErrorNotSupported);
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
    const bool bad = g_memset++ == g_fail_memset;
    log(bad ? "fail" : "memset", st, std::to_string(n));
    if (!bad) memset(p, v, n);
    return set(bad ? cudaErrorUnknown : cudaSuccess);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)g_next++; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) {
    log("wait", st, std::to_string((long)e));
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return set(cudaErrorNotSupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return set(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return set(cudaErrorNotSupported); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return set(cudaErrorNotSupported); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)g_next++; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    log("record", st, std::to_string((long)e));
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 0.f; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return set(cudaErrorNotSupported); }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* r) {
    *f = nullptr;  // no tensor maps: the cp.async staging
    if (r) *r = cudaDriverEntryPointSymbolNotFound;
    return cudaErrorNotSupported;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
}
