// A CUDA runtime without a GPU, for tests of the library's host code: device
// memory is host memory, kernels are not run, copies take their time. It
// counts what a GPU could not stand: a launch on another device than the one
// its memory is on, or with freed memory.
#include <cuda_runtime_api.h>

#include <chrono>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>

namespace {
struct Block {
    size_t bytes;
    int device;
};
std::mutex mu;
std::map<char*, Block> live;
std::map<const void*, std::string> kernels;
thread_local int current = 0;
int delay_us = 0, launches = 0, on_other_device = 0, with_freed_memory = 0;

void pause_us()
{
    if (delay_us)
        std::this_thread::sleep_for(std::chrono::microseconds(delay_us));
}

// the live block that holds [p, p + bytes), or NULL; under mu
const Block* block_of(const void* p, size_t bytes)
{
    auto it = live.upper_bound((char*)p);
    if (it == live.begin())
        return nullptr;
    --it;
    return (char*)p + bytes <= it->first + it->second.bytes ? &it->second : nullptr;
}
}  // namespace

extern "C" {

void fake_delay_us(int us) { delay_us = us; }
int fake_launches() { return launches; }
int fake_on_other_device() { return on_other_device; }
int fake_with_freed_memory() { return with_freed_memory; }

void** __cudaRegisterFatBinary(void*)
{
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*)
{
    std::lock_guard<std::mutex> lock(mu);
    kernels[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }

cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t)
{
    std::lock_guard<std::mutex> lock(mu);
    if (kernels[f].find("k_task_rows") == std::string::npos)
        return cudaSuccess;
    ++launches;
    // (state, outputs, ids, first, n, rows, ...)
    const int n = *(int*)args[4];
    const Block* rows = block_of(*(void**)args[5], (size_t)n * 25 * sizeof(double));
    const void* ids = *(void**)args[2];
    const Block* list = ids ? block_of(ids, n * sizeof(int)) : nullptr;
    with_freed_memory += !rows || (ids && !list);
    on_other_device += rows && rows->device != current;
    return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t bytes)
{
    std::lock_guard<std::mutex> lock(mu);
    *p = std::calloc(1, bytes);
    live[(char*)*p] = Block{bytes, current};
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    // kept, so that a read of it is a count here and no fault
    std::lock_guard<std::mutex> lock(mu);
    live.erase((char*)p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) { return (*p = std::calloc(1, bytes)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) { return cudaMallocHost(p, bytes); }
cudaError_t cudaFreeHost(void* p)
{
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    std::memcpy(d, s, n);
    pause_us();
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n)
{
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaGetDevice(int* d)
{
    *d = current;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d)
{
    current = d;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n)
{
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int)
{
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    pause_us();
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorNotSupported; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }

}  // extern "C"
