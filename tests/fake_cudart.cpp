// Stand-ins for the CUDA runtime functions that the library calls, linked with its object files in place of the runtime: launches
// are written down instead of made, and any call can be told to fail.  For tests that run without a GPU.
#include <cuda_runtime_api.h>

#include <cstring>
#include <map>
#include <string>
#include <vector>

#define HIDDEN __attribute__((visibility("hidden")))

namespace {
struct Launch {
    std::string kernel;
    unsigned grid, block;      // CTAs, threads
    int beside;                // launched as a programmatic dependent
};
std::map<const void *, std::string> &names()
{
    static std::map<const void *, std::string> m;
    return m;
}
std::vector<Launch> launches;
std::map<std::string, int> calls, fail_at;
cudaError_t last = cudaSuccess;
struct { dim3 grid, block; size_t shared; cudaStream_t stream; } pushed;

cudaError_t enter(const char *function)
{
    const int n = ++calls[function];
    const auto it = fail_at.find(function);
    if (it == fail_at.end() || it->second != n) return cudaSuccess;
    return last = cudaErrorLaunchOutOfResources;
}
void record(const void *f, dim3 g, dim3 b, int beside)
{
    const auto it = names().find(f);
    launches.push_back({it == names().end() ? "?" : it->second, g.x * g.y * g.z, b.x * b.y * b.z, beside});
}
}  // namespace

extern "C" {
// what a test uses
int fake_launches() { return int(launches.size()); }
const char *fake_launch(int i, unsigned *grid, unsigned *block, int *beside)
{
    *grid = launches[i].grid;
    *block = launches[i].block;
    *beside = launches[i].beside;
    return launches[i].kernel.c_str();
}
void fake_reset() { launches.clear(); calls.clear(); fail_at.clear(); last = cudaSuccess; }
int fake_last_error() { return last; }
void fake_fail(const char *function, int nth) { fail_at[function] = nth; }

// what the library uses
HIDDEN void **__cudaRegisterFatBinary(void *) { static void *handle; return &handle; }
HIDDEN void __cudaRegisterFatBinaryEnd(void **) {}
HIDDEN void __cudaUnregisterFatBinary(void **) {}
HIDDEN void __cudaRegisterFunction(void **, const char *host, char *, const char *device, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) { names()[host] = device; }
HIDDEN void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
HIDDEN unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t shared, cudaStream_t s) { pushed = {g, b, shared, s}; return 0; }
HIDDEN cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *shared, void *s)
{
    *g = pushed.grid;
    *b = pushed.block;
    *shared = pushed.shared;
    *static_cast<cudaStream_t *>(s) = pushed.stream;
    return cudaSuccess;
}
HIDDEN cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t, cudaStream_t)
{
    if (const cudaError_t e = enter("cudaLaunchKernel")) return e;
    record(f, g, b, 0);
    return cudaSuccess;
}
HIDDEN cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **)
{
    if (const cudaError_t e = enter("cudaLaunchKernelExC")) return e;
    record(f, c->gridDim, c->blockDim, 1);
    return cudaSuccess;
}
HIDDEN cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
HIDDEN cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return enter("cudaFuncSetAttribute"); }
HIDDEN cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *, const void *) { return enter("cudaFuncGetAttributes"); }
HIDDEN cudaError_t cudaGetDevice(int *d) { *d = 0; return enter("cudaGetDevice"); }
HIDDEN const char *cudaGetErrorString(cudaError_t) { return "fake"; }
HIDDEN cudaError_t cudaGetSymbolAddress(void **p, const void *) { *p = reinterpret_cast<void *>(256); return cudaSuccess; }
HIDDEN cudaError_t cudaMemcpyFromSymbol(void *p, const void *, size_t n, size_t, cudaMemcpyKind) { std::memset(p, 0, n); return cudaSuccess; }
HIDDEN cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
HIDDEN cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}
