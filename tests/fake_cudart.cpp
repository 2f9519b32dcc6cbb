// fake_cudart.cpp -- a CUDA runtime for tests of the host engine on machines
// without a GPU: two devices whose memory is the host's, kernels that do
// nothing, and a log of what a real runtime would have been asked to do.  Rules
// of the real one that the tests rest on are kept: a launch with more dynamic
// shared memory than its function's limit on the current device fails, and a
// stream that is being captured, or the legacy one, cannot begin a capture, and no
// graph is launched into a capture.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {

struct Stream { int prio = 0; bool capturing = false; };

std::mutex mu;
std::string text;                                       // the log, a line per call
std::map<const void*, std::string> names;               // kernel entry -> device name
std::map<std::pair<int, const void*>, int> smem_limit;  // per device
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
thread_local struct { dim3 grid, block; size_t smem; void* stream; } config;

void note(const std::string& line)
{
    std::lock_guard<std::mutex> lk(mu);
    text += line + "\n";
}

cudaError_t set(cudaError_t e)
{
    if (e != cudaSuccess) last = e;
    return e;
}

Stream* of(cudaStream_t s) { return (uintptr_t)s > 2 ? reinterpret_cast<Stream*>(s) : nullptr; }

void* get(size_t bytes) { return std::calloc(1, bytes ? bytes : 1); }

cudaError_t launch(const void* f, size_t smem, cudaStream_t s)
{
    std::string name;
    {
        std::lock_guard<std::mutex> lk(mu);
        const auto it = smem_limit.find({device, f});
        if ((long)smem > (it == smem_limit.end() ? 48 * 1024 : it->second)) return set(cudaErrorInvalidValue);
        name = names[f];
    }
    note("launch device " + std::to_string(device) + " priority " + std::to_string(of(s) ? of(s)->prio : 0) + " " + name);
    return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- what the tests call
const char* fake_log() { return text.c_str(); }
void fake_clear() { text.clear(); }
void fake_capturing(cudaStream_t s, int on) { of(s)->capturing = on != 0; }

// ---- what compiled kernels and their launches call
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*)
{
    names[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s)
{
    config = {g, b, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s)
{
    *g = config.grid;
    *b = config.block;
    *smem = config.smem;
    *(void**)s = config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t smem, cudaStream_t s) { return launch((const void*)k, smem, s); }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t s) { return launch(f, smem, s); }

// ---- the runtime
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int)
{
    std::memset(p, 0, sizeof(*p));
    std::snprintf(p->name, sizeof(p->name), "fake");
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v)
{
    std::lock_guard<std::mutex> lk(mu);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_limit[{device, f}] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int threads, size_t)
{
    *n = threads < 512 ? 512 / threads : 1;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return set(cudaErrorInvalidSymbol); }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             enum cudaDriverEntryPointQueryResult*)
{
    *f = nullptr;
    return set(cudaErrorNotSupported);
}
cudaError_t cudaMemGetInfo(size_t* fr, size_t* total) { *fr = *total = (size_t)64 << 30; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = get(n); return *p ? cudaSuccess : set(cudaErrorMemoryAllocation); }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }

cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int prio)
{
    Stream* n = new Stream;
    n->prio = prio;
    *s = reinterpret_cast<cudaStream_t>(n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { return cudaStreamCreateWithPriority(s, f, 0); }
cudaError_t cudaStreamGetPriority(cudaStream_t s, int* prio) { *prio = of(s) ? of(s)->prio : 0; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete of(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st)
{
    *st = of(s) && of(s)->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode)
{
    if (!of(s) || of(s)->capturing) return set(cudaErrorStreamCaptureUnsupported);
    of(s)->capturing = true;
    note("capture");
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g)
{
    of(s)->capturing = false;
    *g = reinterpret_cast<cudaGraph_t>(get(1));
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long)
{
    *e = reinterpret_cast<cudaGraphExec_t>(get(1));
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { std::free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s)
{
    if (of(s) && of(s)->capturing) return set(cudaErrorStreamCaptureUnsupported);
    note("replay");
    return cudaSuccess;
}

cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(get(1)); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }

}  // extern "C"
