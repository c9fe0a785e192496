// fake_cuda.cpp -- a CUDA runtime without a GPU for tests of the host side: linked with
// the library's objects in place of the static runtime (fakecuda.py). Device memory is
// addresses only, copies and memsets move nothing, launches are written to a log by
// kernel name, and a test can make allocations fail.
#include <cuda_runtime.h>
#include <cxxabi.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {

std::map<const void *, std::string> &names()
{
    static std::map<const void *, std::string> m;
    return m;
}

std::string g_log;
long g_fail = 0;  // cudaMalloc calls that fail from now on
uintptr_t g_next = uintptr_t(1) << 40;
struct Config { dim3 grid, block; size_t smem; cudaStream_t st; } g_config;

void log_launch(const void *f, unsigned grid, bool chained)
{
    int rc = 0;
    char *d = abi::__cxa_demangle(names()[f].c_str(), nullptr, nullptr, &rc);
    g_log += std::string(chained ? "1 " : "0 ") + std::to_string(grid) + " " + (d ? d : names()[f]) + "\n";
    std::free(d);
}

}  // namespace

extern "C" {

// The log since the last call: a line "chained grid kernel" per launch.
const char *fake_take_log()
{
    static std::string out;
    out.swap(g_log);
    g_log.clear();
    return out.c_str();
}
void fake_fail_malloc(long calls) { g_fail = calls; }

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, void *, void *, void *, void *, int *)
{
    names()[f] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void *st)
{
    g_config = {g, b, s, static_cast<cudaStream_t>(st)};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st)
{
    *g = g_config.grid;
    *b = g_config.block;
    *s = g_config.smem;
    *static_cast<cudaStream_t *>(st) = g_config.st;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3, void **, size_t, cudaStream_t)
{
    log_launch(f, g.x, false);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **)
{
    bool chained = false;
    for (unsigned i = 0; i < c->numAttrs; i++)
        chained |= c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization &&
                   c->attrs[i].val.programmaticStreamSerializationAllowed;
    log_launch(f, c->gridDim.x, chained);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n)
{
    *p = nullptr;
    if (g_fail > 0 && g_fail--) return cudaErrorMemoryAllocation;
    *p = reinterpret_cast<void *>(g_next);
    g_next += (n + 511) & ~size_t(511);
    return cudaSuccess;
}
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { return (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int)
{
    std::memset(p, 0, sizeof(*p));
    std::strcpy(p->name, "fake");
    p->multiProcessorCount = 148;
    p->major = 10;
    p->totalGlobalMem = size_t(180) << 30;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = nullptr; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { *p = const_cast<void *>(s); return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }

}  // extern "C"
