// A CUDA runtime without a device, preloaded over the real one by
// test_host_driver.py: two devices whose memory is the host's, kernels that do
// nothing (the root partition counts its roots), and the launches and events of
// the host driver noted.  A launch is refused, as by the real one, when its
// dynamic shared memory was not allowed for that kernel on the current device.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {
constexpr int DEVICES = 2;
std::mutex mu;
std::map<const void*, std::string> name_of;
std::map<std::pair<int, const void*>, size_t> allowed;
std::string launches, dump;
int device = 0, events = 0;
cudaError_t last = cudaSuccess;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
thread_local Config config;

cudaError_t launch(const void* fn, dim3 block, void** args, size_t smem)
{
    std::lock_guard<std::mutex> lk(mu);
    const auto limit = allowed.find({device, fn});
    if (smem > (limit == allowed.end() ? 48u * 1024 : limit->second)) return last = cudaErrorInvalidValue;
    const std::string& name = name_of[fn];
    std::string line = name + " " + std::to_string(block.x);
    if (name.find("k_partition_roots") != std::string::npos) {  // (boards, depths, n, level, counters, ...)
        const unsigned char* depths = *(const unsigned char**)args[1];
        const unsigned n = *(unsigned*)args[2];
        unsigned* counters = *(unsigned**)args[4];
        line += " counters " + std::to_string(counters[0]) + " " + std::to_string(counters[1]);
        counters[0] += n;
        for (unsigned i = 0; i < n; i++) {
            if (depths[i] < counters[2]) counters[2] = depths[i];
            if (depths[i] > counters[3]) counters[3] = depths[i];
        }
    }
    launches += line + "\n";
    return cudaSuccess;
}
void* memory(size_t n) { return calloc(n + 256, 1); }
}  // namespace

extern "C" {

// the launches since the last question ("name block" a line) and the waits for a
// stream ("wait"), the events recorded; host_error leaves an error for the next check
const char* host_launches()
{
    std::lock_guard<std::mutex> lk(mu);
    dump.swap(launches);
    launches.clear();
    return dump.c_str();
}
void host_error() { last = cudaErrorInvalidValue; }
int host_events()
{
    const int n = events;
    events = 0;
    return n;
}

void** __cudaRegisterFatBinary(void*) { return (void**)memory(8); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* fn, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*)
{
    name_of[fn] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, CUstream_st* stream)
{
    config = Config{grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream)
{
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *(cudaStream_t*)stream = config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* kernel, const void* fn)
{
    *kernel = (cudaKernel_t)fn;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3, dim3 block, void** args, size_t smem, cudaStream_t)
{
    return launch((const void*)kernel, block, args, smem);
}
cudaError_t cudaLaunchCooperativeKernel(const void* fn, dim3, dim3 block, void** args, size_t smem, cudaStream_t)
{
    return launch(fn, block, args, smem);
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute, int value)
{
    allowed[{device, fn}] = (size_t)value;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* fn, int threads, size_t smem)
{
    return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, fn, threads, smem, 0);
}
cudaError_t cudaGetDeviceCount(int* n) { *n = DEVICES; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int)
{
    memset(p, 0, sizeof(*p));
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* free, size_t* total) { *free = *total = 8ull << 30; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = memory(n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = memory(n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)memory(8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free((void*)s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    std::lock_guard<std::mutex> lk(mu);
    launches += "wait\n";
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)memory(8); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free((void*)e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { events++; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)memory(8); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { *x = (cudaGraphExec_t)memory(8); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free((void*)g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { free((void*)x); return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "refused by the host runtime"; }
}
