// A CUDA runtime that launches nothing: it records what the library's host code enqueues, and from which thread, and can refuse one of
// the launches.  Linked with the library's own object files by test_launch_sequence.py.
#include <cuda_runtime_api.h>
#include <unistd.h>

#include <atomic>
#include <map>
#include <mutex>
#include <string>

namespace {
std::mutex g_mutex;
std::map<const void*, std::string>* g_names;      // host stub -> device function
std::string g_log;                                // one "thread:kernel" line per piece of work
int g_refuse = -1, g_count = 0, g_pause_us = 0;
std::atomic<int> g_attributes{0};                 // kernel attributes set
std::atomic<int> g_threads{0};
thread_local int t_id = -1;
thread_local cudaError_t t_last = cudaSuccess;
thread_local struct { dim3 grid, block; size_t smem; cudaStream_t stream; } t_config;

cudaError_t enqueue(const std::string& name) {
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        if (t_id < 0) t_id = g_threads++;
        const bool refuse = g_count++ == g_refuse;
        g_log += std::to_string(t_id) + ":" + name + (refuse ? ":refused\n" : "\n");
        if (refuse) return t_last = cudaErrorInvalidConfiguration;
    }
    if (g_pause_us) usleep(g_pause_us);           // room for another thread to come in between
    return cudaSuccess;
}
cudaError_t launch(const void* stub) {
    std::string name;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        name = g_names && g_names->count(stub) ? (*g_names)[stub] : "?";
    }
    return enqueue(name);
}
extern "C" int fake_encode() { return 0; }
}  // namespace

extern "C" {
void fake_start(int refuse, int pause_us) {
    std::lock_guard<std::mutex> lock(g_mutex);
    g_log.clear();
    g_refuse = refuse;
    g_pause_us = pause_us;
    g_count = 0;
    g_attributes = 0;
}
const char* fake_log() { return g_log.c_str(); }
const char* fake_kernels() {                      // every kernel of the library, one per line
    static std::string names;
    names.clear();
    if (g_names) for (const auto& k : *g_names) names += k.second + "\n";
    return names.c_str();
}
int fake_last_error() { return t_last; }
int fake_attributes() { return g_attributes; }

void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, void*, void*, void*, void*, int*) {
    if (!g_names) g_names = new std::map<const void*, std::string>();
    (*g_names)[stub] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) {
    t_config = {g, b, m, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
    *g = t_config.grid; *b = t_config.block; *m = t_config.smem; *static_cast<cudaStream_t*>(s) = t_config.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t) { return launch(f); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void**) { return launch(f); }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return enqueue("memset"); }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return enqueue("memcpy"); }
cudaError_t cudaGetLastError() { const cudaError_t e = t_last; t_last = cudaSuccess; return e; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrComputeCapabilityMajor ? 10 : 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { ++g_attributes; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* r) {
    *f = reinterpret_cast<void*>(fake_encode);
    if (r) *r = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = nullptr; return cudaErrorNotSupported; }
cudaError_t cudaMalloc(void**, size_t) { return cudaErrorNotSupported; }
cudaError_t cudaFree(void*) { return cudaErrorNotSupported; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t*, void*) { return cudaErrorNotSupported; }
cudaError_t cudaIpcOpenMemHandle(void**, cudaIpcMemHandle_t, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaErrorNotSupported; }
}
