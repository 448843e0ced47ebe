// A stand-in for the CUDA runtime, linked with the engine's objects in place of it, so that
// host code runs where there is no GPU: memory is counted against a settable total, kernels
// do nothing, and launches are recorded.  Copies and fills do nothing either (memory is zero
// when it is allocated).
#include <sys/mman.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

#include <cuda.h>
#include <cuda_runtime_api.h>

namespace {
std::mutex m;
std::map<void*, size_t> blocks;
size_t total = (size_t)288 << 30, used = 0;
bool capturing = false;
// launches: plain, cooperative, cooperative inside a capture, graph; captures begun
long long counts[5];
char last[256];  // the first bytes of the last cooperative launch's first argument
char handles[4096];
unsigned next_handle = 0;

template <typename T>
cudaError_t make(T* out)
{
    *out = reinterpret_cast<T>(handles + 1 + next_handle++ % 4000);
    return cudaSuccess;
}
CUresult encode(CUtensorMap*, ...) { return CUDA_SUCCESS; }
}  // namespace

extern "C" {

void fake_set_total(unsigned long long bytes) { total = bytes; }
unsigned long long fake_used() { return used; }
void fake_counts(long long* out, int clear)
{
    memcpy(out, counts, sizeof counts);
    if (clear) memset(counts, 0, sizeof counts);
}

cudaError_t cudaMalloc(void** p, size_t n)
{
    std::lock_guard<std::mutex> lock(m);
    *p = nullptr;
    if (n > total || used > total - n) return cudaErrorMemoryAllocation;
    void* q = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE,
                   MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (q == MAP_FAILED) return cudaErrorMemoryAllocation;
    blocks[q] = n;
    used += n;
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    std::lock_guard<std::mutex> lock(m);
    auto it = blocks.find(p);
    if (it == blocks.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    used -= it->second;
    munmap(p, it->second ? it->second : 1);
    blocks.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t)
{
    std::lock_guard<std::mutex> lock(m);
    *f = total > used ? total - used : 0;
    *t = total;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    return (*p = calloc(n, 1)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }

cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind)
{
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind,
                              cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return make(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return make(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return make(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }

cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s)
{
    *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    capturing = true;
    ++counts[4];
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g)
{
    capturing = false;
    return make(g);
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long)
{
    return make(e);
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*)
{
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { ++counts[3]; return cudaSuccess; }

void fake_last_cooperative(void* out, int n) { memcpy(out, last, n); }

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void** args)
{
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeCooperative && c->attrs[i].val.cooperative) {
            ++counts[capturing ? 2 : 1];
            memcpy(last, args[0], sizeof last);
            return cudaSuccess;
        }
    ++counts[0];
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t)
{
    ++counts[0];
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void*) { return make(k); }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st)
{
    *g = *b = dim3(1);
    *s = 0;
    *static_cast<cudaStream_t*>(st) = nullptr;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*,
                            dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int,
                                                                   size_t, unsigned)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetPCIBusId(char* b, int n, int)
{
    strncpy(b, "fake", n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeDevice;
    a->devicePointer = const_cast<void*>(p);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*)
{
    static char area[1 << 16];
    *p = area;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** fn, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q)
{
    *fn = reinterpret_cast<void*>(encode);
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }

}  // extern "C"
