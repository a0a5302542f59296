// A CUDA runtime without a device, loaded ahead of the real one, for tests of the library's host side on
// the CPU: device memory is host memory, kernels are logged and do not run, and a chosen call can be made
// to fail.  A launch pass reports path jobs in the first `busy` waves of a phase, so that the host goes on as
// it would behind a device.  Log, one line each:
//   launch <stream> <kernel> [wave npool path_tau ordered max_scatt refill: kernels of a wave] smem <bytes>
//   memset <stream> <bytes>   record <event> <stream>   wait <stream> <event>   malloc <bytes> <ok>
//   capture <stream>   uncapture <stream>   replay <stream> ... end of replay
#include <cuda_runtime_api.h>

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cxxabi.h>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <vector>

// fake_params.cu: the parameters of a wave's kernels as text; `jobs` path jobs from the launch pass of the first `busy` waves
size_t fake_params_size();
void fake_params(const void* params, char* out, size_t n);
void fake_launch_pass(const void* params, int busy, int jobs);

namespace {

struct Graph { std::vector<std::function<void(cudaStream_t)>> ops; };
struct Call { dim3 grid, block; size_t smem; cudaStream_t stream; };

std::recursive_mutex mu;
std::string text;
std::map<const void*, std::string> kernels;
std::map<void*, size_t> allocated;
size_t total = (size_t)8 << 30, used = 0;
int busy = 0, jobs = 0;             // waves of a phase with work, path jobs in each
std::string fail_name;              // launches of kernels whose name holds this ("instantiate": of a graph) ...
int fail_skip = -1;                 // ... fail after this many (-1: none)
cudaError_t last = cudaSuccess;
std::map<cudaStream_t, Graph*> capturing;
intptr_t handles = 0;
thread_local std::vector<Call> calls;

void log(const char* f, ...) {
    char b[1024];
    va_list a;
    va_start(a, f);
    vsnprintf(b, sizeof(b), f, a);
    va_end(a);
    text += b;
    text += '\n';
}
long id(const void* h) { return (long)(intptr_t)h; }

// runs now, or with the graph of a capturing stream
cudaError_t op(cudaStream_t s, std::function<void(cudaStream_t)> f) {
    std::lock_guard<std::recursive_mutex> hold(mu);
    auto c = capturing.find(s);
    if (c != capturing.end()) c->second->ops.push_back(f); else f(s);
    return cudaSuccess;
}

cudaError_t take(void** p, size_t n) {
    std::lock_guard<std::recursive_mutex> hold(mu);
    const bool ok = used + n <= total;
    log("malloc %zu %d", n, (int)ok);
    if (!ok) return last = cudaErrorMemoryAllocation;
    *p = calloc(1, n ? n : 1);
    allocated[*p] = n;
    used += n;
    return cudaSuccess;
}
cudaError_t give(void* p) {
    std::lock_guard<std::recursive_mutex> hold(mu);
    if (!p) return cudaSuccess;
    used -= allocated.at(p);
    allocated.erase(p);
    free(p);
    return cudaSuccess;
}

cudaError_t launch(const void* f, size_t smem, cudaStream_t s, void** args) {
    std::lock_guard<std::recursive_mutex> hold(mu);
    const std::string name = kernels.at(f);
    if (fail_skip >= 0 && name.find(fail_name) != std::string::npos && fail_skip-- == 0)
        return last = cudaErrorLaunchOutOfResources;
    const bool wave = name.find("WaveParams") != std::string::npos;
    if (!wave) return op(s, [=](cudaStream_t q) { log("launch %ld %s smem %zu", id(q), name.c_str(), smem); });
    const std::vector<char> params((const char*)args[0], (const char*)args[0] + fake_params_size());
    return op(s, [=](cudaStream_t q) {
        char fields[256];
        fake_params(params.data(), fields, sizeof(fields));
        log("launch %ld %s %s smem %zu", id(q), name.c_str(), fields, smem);
        if (name.find("launch_kernel") != std::string::npos) fake_launch_pass(params.data(), busy, jobs);
    });
}

}  // namespace

extern "C" {

// ---- the test's side
const char* fake_log() {             // the log so far; the next call starts a new one
    static std::string out;
    std::lock_guard<std::recursive_mutex> hold(mu);
    out.swap(text);
    text.clear();
    return out.c_str();
}
void fake_busy(int waves, int n) { busy = waves; jobs = n; }
void fake_fail(const char* kernel, int after) { fail_name = kernel; fail_skip = after; }
void fake_memory(size_t bytes) { total = bytes; }
size_t fake_used() { return used; }
void fake_fill(size_t bytes) {       // 0, 1, 2, ... in every allocation of this size
    for (auto& a : allocated)
        if (a.second == bytes)
            for (size_t i = 0; i < bytes / sizeof(double); i++) ((double*)a.first)[i] = (double)i;
}

// ---- registration and launches
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* device, int, uint3*, uint3*, dim3*, dim3*, int*) {
    int rc = 0;
    char* d = abi::__cxa_demangle(device, nullptr, nullptr, &rc);
    kernels[host] = rc == 0 && d ? d : device;
    free(d);
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s) { calls.push_back({g, b, smem, s}); return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    const Call c = calls.back();
    calls.pop_back();
    *g = c.grid; *b = c.block; *smem = c.smem; *static_cast<cudaStream_t*>(s) = c.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t smem, cudaStream_t s) { return launch(f, smem, s, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) { return launch(f, c->dynamicSmemBytes, c->stream, args); }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    memset(a, 0, sizeof(*a));
    a->ptxVersion = a->binaryVersion = 100;
    a->maxThreadsPerBlock = 1024;
    a->maxDynamicSharedSizeBytes = 32 << 10;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 4; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 4; return cudaSuccess; }

// ---- device, errors
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1024; return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = (cudaMemPool_t)1; return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) { *static_cast<uint64_t*>(v) = 0; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "a failure of the fake runtime"; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last; }

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = total - used; *t = total; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static char* a = (char*)calloc(1, 32 << 20); *p = a; return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
    return op(s, [=](cudaStream_t q) { memset(p, v, n); log("memset %ld %zu", id(q), n); });
}
cudaError_t cudaMemcpy(void* d, const void* a, size_t n, cudaMemcpyKind) { memcpy(d, a, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* a, size_t n, cudaMemcpyKind, cudaStream_t s) {
    return op(s, [=](cudaStream_t) { memcpy(d, a, n); });
}

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)++handles; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { return op(s, [=](cudaStream_t q) { log("wait %ld %ld", id(q), id(e)); }); }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* c) {
    *c = capturing.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    if (capturing.count(s)) return last = cudaErrorIllegalState;
    capturing[s] = new Graph;
    log("capture %ld", id(s));
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    if (!capturing.count(s)) return last = cudaErrorIllegalState;
    *g = (cudaGraph_t)capturing[s];
    capturing.erase(s);
    log("uncapture %ld", id(s));
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
    if (fail_name == "instantiate" && fail_skip-- == 0) return last = cudaErrorMemoryAllocation;
    *x = (cudaGraphExec_t) new Graph(*(Graph*)g);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph*)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete (Graph*)x; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
    log("replay %ld", id(s));
    for (auto& f : ((Graph*)x)->ops) f(s);
    log("end of replay");
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)++handles; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return op(s, [=](cudaStream_t q) { log("record %ld %ld", id(e), id(q)); }); }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned) { return cudaEventRecord(e, s); }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }

}  // extern "C"
