// A stand-in for the CUDA runtime on the host, for tests of the host side's error paths without a GPU:
// device memory is host memory, copies happen at once, kernels do nothing but get recorded, and any call
// can be made to fail. Linked with the library's sources in place of the real runtime (-cudart none).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Launch {
    std::string name;
    std::vector<uint8_t> arg;          // the bytes of the argument asked for (fake_capture)
};
std::map<void const*, std::string>& kernels() {       // (the library registers them before main's statics are up)
    static std::map<void const*, std::string> k;
    return k;
}
std::vector<Launch> g_launches;
std::vector<std::string> g_calls;
std::string g_fail_call;               // the call that fails, and how many of it succeed first
int g_fail_after = -1;
std::string g_capture_kernel;
int g_capture_arg = -1;
size_t g_capture_bytes = 0;
std::vector<std::pair<void*, size_t>> g_blocks;      // live device memory, oldest first
cudaError_t g_last = cudaSuccess;
struct { dim3 grid, block; size_t smem; cudaStream_t stream; } g_config;

cudaError_t call(char const* name) {
    g_calls.push_back(name);
    if (g_fail_after < 0 || g_fail_call != name || g_fail_after-- > 0) return cudaSuccess;
    return g_last = cudaErrorMemoryAllocation;
}
cudaError_t launched(void const* fn, void** args, char const* api) {
    if (cudaError_t e = call(api)) return e;
    Launch l{kernels()[fn], {}};
    if (g_capture_arg >= 0 && l.name.find(g_capture_kernel) != std::string::npos) {
        auto const* p = static_cast<uint8_t const*>(args[g_capture_arg]);
        l.arg.assign(p, p + g_capture_bytes);
    }
    g_launches.push_back(std::move(l));
    return cudaSuccess;
}
} // namespace

extern "C" {

// ---- what a test sets and reads
void fake_reset(void) {
    g_launches.clear();
    g_calls.clear();
    g_fail_after = g_capture_arg = -1;
    g_last = cudaSuccess;
}
void fake_fail(char const* name, int after) {
    g_fail_call = name;
    g_fail_after = after;
}
void fake_capture(char const* kernel, int arg, size_t bytes) {
    g_capture_kernel = kernel;
    g_capture_arg = arg;
    g_capture_bytes = bytes;
}
int fake_count(char const* name) {                  // calls, or launches of kernels with `name` in their symbol
    int n = 0;
    for (auto const& c : g_calls) n += c == name;
    for (auto const& l : g_launches) n += l.name.find(name) != std::string::npos;
    return n;
}
size_t fake_arg(int nth, void* out) {               // the argument's bytes in the nth launch captured
    for (auto const& l : g_launches)
        if (!l.arg.empty() && nth-- == 0) {
            std::memcpy(out, l.arg.data(), l.arg.size());
            return l.arg.size();
        }
    return 0;
}
size_t fake_log(char* out, size_t size) {           // the calls since the reset, one a line
    std::string s;
    for (auto const& c : g_calls) s += c + "\n";
    if (s.size() < size) std::memcpy(out, s.c_str(), s.size() + 1);
    return s.size();
}
void* fake_block(size_t bytes) {                    // the live device block of that size (the newest)
    void* found = nullptr;
    for (auto const& b : g_blocks)
        if (b.second == bytes) found = b.first;
    return found;
}

// ---- the runtime
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, char const* fn, char*, char const* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels()[fn] = name;
}
void __cudaRegisterVar(void**, char*, char*, char const*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    g_config = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = g_config.grid;
    *block = g_config.block;
    *smem = g_config.smem;
    *static_cast<cudaStream_t*>(stream) = g_config.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(void const* fn, dim3, dim3, void** args, size_t, cudaStream_t) {
    return launched(fn, args, "cudaLaunchKernel");
}
cudaError_t cudaLaunchKernelExC(cudaLaunchConfig_t const*, void const* fn, void** args) {
    return launched(fn, args, "cudaLaunchKernelExC");
}
cudaError_t cudaGetLastError(void) {
    cudaError_t const e = g_last;
    g_last = cudaSuccess;
    return e;
}
char const* cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaSetDevice(int) { return call("cudaSetDevice"); }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    return call("cudaGetDeviceProperties");
}
cudaError_t cudaFuncSetAttribute(void const*, cudaFuncAttribute, int) { return call("cudaFuncSetAttribute"); }
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return call("cudaGetDevice");
}
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return call("cudaGetDeviceCount");
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472
         : a == cudaDevAttrReservedSharedMemoryPerBlock   ? 1024
         : a == cudaDevAttrMultiProcessorCount            ? 148
                                                          : 0;
    return call("cudaDeviceGetAttribute");
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, void const*) {
    std::memset(a, 0, sizeof *a);
    return call("cudaFuncGetAttributes");
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, void const*, int, size_t, unsigned) {
    *n = 1;
    return call("cudaOccupancyMaxActiveBlocksPerMultiprocessor");
}
cudaError_t cudaGetSymbolAddress(void** p, void const*) {
    static unsigned char word[4096];
    *p = word;
    return call("cudaGetSymbolAddress");
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = nullptr;
    return call("cudaStreamCreateWithFlags");
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return call("cudaStreamDestroy"); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return call("cudaStreamSynchronize"); }
cudaError_t cudaDeviceSynchronize(void) { return call("cudaDeviceSynchronize"); }
cudaError_t cudaMalloc(void** p, size_t bytes) {
    if (cudaError_t e = call("cudaMalloc")) return e;
    *p = std::calloc(bytes, 1);
    g_blocks.emplace_back(*p, bytes);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::erase_if(g_blocks, [&](auto const& b) { return b.first == p; });
    std::free(p);
    return call("cudaFree");
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
    if (cudaError_t e = call("cudaHostAlloc")) return e;
    *p = std::calloc(bytes, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return call("cudaFreeHost");
}
cudaError_t cudaMemcpy(void* dst, void const* src, size_t bytes, cudaMemcpyKind) {
    if (cudaError_t e = call("cudaMemcpy")) return e;
    if (bytes && (!dst || !src)) return g_last = cudaErrorInvalidValue;
    std::memcpy(dst, src, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, void const* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
    if (cudaError_t e = call("cudaMemcpyAsync")) return e;
    if (bytes && (!dst || !src)) return g_last = cudaErrorInvalidValue;
    std::memcpy(dst, src, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t bytes) {
    if (cudaError_t e = call("cudaMemset")) return e;
    std::memset(p, v, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t bytes, cudaStream_t) {
    if (cudaError_t e = call("cudaMemsetAsync")) return e;
    std::memset(p, v, bytes);
    return cudaSuccess;
}

} // extern "C"
