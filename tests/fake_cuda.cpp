// A stand-in for the CUDA runtime, for tests of the library's host code on a
// machine without a GPU: device memory is host memory, copies are made at
// once, kernels do not run, and every call is written to a log.  A chosen
// call can be made to fail.
#include <cuda_runtime_api.h>
#include <sys/mman.h>
#include <unistd.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {

std::string g_log;
std::map<const void*, std::string> g_kernels;
long g_calls = 0, g_fail_at = 0;
bool g_failed = false;
bool g_pinned = false;  // what host pointers are said to be
int g_int = 0;  // what a 4-byte copy from the device returns, if not 0
dim3 g_grid, g_block;
size_t g_smem = 0;
void* g_stream = nullptr;

// Logs a call; true when it is the one that has to fail.
template <class... A>
bool note(const char* fmt, A... a) {
    char line[512];
    if constexpr (sizeof...(a) == 0) snprintf(line, sizeof(line), "%s", fmt);
    else snprintf(line, sizeof(line), fmt, a...);
    g_log += line;
    ++g_calls;
    const bool f = g_fail_at > 0 && g_calls == g_fail_at;
    if (f) {
        g_log += " FAILS";
        g_failed = true;
    }
    g_log += '\n';
    return f;
}
cudaError_t done(bool failed, cudaError_t e = cudaErrorUnknown) { return failed ? e : cudaSuccess; }

const char* kernel_name(const void* f) {
    auto it = g_kernels.find(f);
    return it == g_kernels.end() ? "?" : it->second.c_str();
}
cudaError_t launch(const void* f, dim3 g, dim3 b, size_t smem) {
    return done(note("launch %s %u %u %u %u %u %zu", kernel_name(f), g.x, g.y, g.z, b.x, b.y, smem));
}

}  // namespace

extern "C" {

const char* fake_log() { return g_log.c_str(); }
void fake_reset(long fail_at) {
    g_log.clear();
    g_calls = 0;
    g_fail_at = fail_at;
    g_failed = false;
}
int fake_failed() { return g_failed; }
void fake_int(int v) { g_int = v; }
void fake_pinned(int v) { g_pinned = v; }

void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
    g_kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st) {
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
    *static_cast<void**>(st) = g_stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) {
    return launch((const void*)k, g, b, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}

cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    return done(note("attribute %s %d %d", kernel_name(f), (int)a, v));
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    memset(a, 0, sizeof(*a));
    a->numRegs = 64;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    memset(p, 0, sizeof(*p));
    snprintf(p->name, sizeof(p->name), "fake");
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrPageableMemoryAccess || a == cudaDevAttrPageableMemoryAccessUsesHostPageTables ? 1
         : a == cudaDevAttrMultiProcessorCount                                                           ? 152
         : a == cudaDevAttrMaxSharedMemoryPerBlockOptin                                                  ? 232448
         : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor                                              ? 233472
                                                                                                         : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) {
    *least = 0;
    *greatest = -5;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult*) {
    return cudaErrorUnknown;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorUnknown; }

cudaError_t cudaMalloc(void** p, size_t n) {
    if (note("malloc %zu", n)) return cudaErrorMemoryAllocation;
    *p = calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    memset(a, 0, sizeof(*a));
    a->type = g_pinned ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
static cudaError_t copy(const char* what, void* d, const void* s, size_t n, cudaMemcpyKind k) {
    if (note("%s %d %zu %p %p", what, (int)k, n, d, s)) return cudaErrorUnknown;
    if (k == cudaMemcpyDeviceToHost) {  // an error where the host may not write, as from the kernel's own copies
        const int fd = memfd_create("copy", 0);
        const bool ok = fd >= 0 && pwrite(fd, s, n, 0) == (ssize_t)n && pread(fd, d, n, 0) == (ssize_t)n;
        close(fd);
        if (!ok) return cudaErrorInvalidValue;
    } else {
        memmove(d, s, n);
    }
    if (n == sizeof(int) && k == cudaMemcpyDeviceToHost && g_int) memcpy(d, &g_int, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    return copy("copy", d, s, n, k);
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return copy("copysync", d, s, n, k); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
    if (note("memset %zu", n)) return cudaErrorUnknown;
    memset(p, v, n);
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    static long id = 0x1000;
    *s = (cudaStream_t)(id += 16);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return done(note("sync stream")); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = (cudaGraph_t)0x10;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = (cudaGraphExec_t)0x20;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiateWithFlags(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long f) {
    return cudaGraphInstantiate(e, g, f);
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return done(note("graph")); }

cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = (cudaEvent_t)0x30;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return done(note("event")); }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return done(note("event")); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return done(note("sync event")); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}

}  // extern "C"
