// A stand-in for the CUDA runtime, for tests of the library's host code
// without a GPU: device memory is host memory, copies are made, kernels are
// written to a log and do nothing.  Allocations and launches can be made to
// fail, and a launch can set a word that one of its arguments points to, as
// a kernel that reports an error does.  Freed memory is kept aside, so that
// an argument of a cooperative launch that points into it is seen.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
std::map<const void *, std::string> g_kernels;
std::map<char *, size_t> g_live, g_freed;
long long g_limit = -1, g_used = 0, g_refused_size = -1;
int g_stale = 0, g_coop_error = 0;
bool g_capture = false;
std::string g_log;
struct Rule {
    std::string kernel;
    int error, arg, offset, value;
};
std::vector<Rule> g_rules;
cudaError_t g_last = cudaSuccess;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
std::vector<Config> g_config;

cudaError_t result(cudaError_t e)
{
    if (e != cudaSuccess) g_last = e;
    return e;
}

cudaError_t launch(const void *fn, dim3 grid, void **args, bool cooperative)
{
    const std::string &name = g_kernels[fn];
    if (cooperative && g_coop_error) return result((cudaError_t)g_coop_error);
    for (const Rule &r : g_rules)
        if (r.error && name.find(r.kernel) != std::string::npos) return result((cudaError_t)r.error);
    if (cooperative)   // one argument, a struct of more than 160 bytes
        for (int i = 0; i < 20; ++i) {
            char *q;
            memcpy(&q, (char *)args[0] + 8 * i, 8);
            auto it = g_freed.upper_bound(q);
            if (it != g_freed.begin() && q < std::prev(it)->first + std::prev(it)->second) ++g_stale;
        }
    for (const Rule &r : g_rules)
        if (!r.error && name.find(r.kernel) != std::string::npos) memcpy(*(char **)args[r.arg] + r.offset, &r.value, sizeof(int));
    g_log += (g_capture ? "captured " : "") + name + " " + std::to_string(grid.x) + "\n";
    return cudaSuccess;
}

cudaError_t allocate(void **p, size_t bytes)
{
    *p = nullptr;
    if ((g_limit >= 0 && g_used + (long long)bytes > g_limit) || (long long)bytes == g_refused_size) return result(cudaErrorMemoryAllocation);
    char *q = (char *)calloc(bytes ? bytes : 1, 1);
    g_live[q] = bytes;
    g_used += (long long)bytes;
    *p = q;
    return cudaSuccess;
}

cudaError_t release(void *p)
{
    auto it = g_live.find((char *)p);
    if (it == g_live.end()) return p ? result(cudaErrorInvalidValue) : cudaSuccess;
    g_used -= (long long)it->second;
    g_freed[it->first] = it->second;
    g_live.erase(it);
    return cudaSuccess;
}

int encode(void *, ...) { return 0; }
}  // namespace

extern "C" {
// the tests' controls
void fake_reset()
{
    g_limit = g_refused_size = -1;
    g_stale = g_coop_error = 0;
    g_rules.clear();
    g_log.clear();
    for (auto &f : g_freed) free(f.first);
    g_freed.clear();
    g_last = cudaSuccess;
}
void fake_clear_log() { g_log.clear(); }
const char *fake_log() { return g_log.c_str(); }
long long fake_used() { return g_used; }
void fake_limit(long long bytes) { g_limit = bytes; }
void fake_refuse_size(long long bytes) { g_refused_size = bytes; }
int fake_stale() { return g_stale; }
void fake_coop_error(int e) { g_coop_error = e; }
void fake_fail(const char *kernel, int e) { g_rules.push_back({kernel, e, 0, 0, 0}); }
void fake_poke(const char *kernel, int arg, int offset, int value) { g_rules.push_back({kernel, 0, arg, offset, value}); }
void fake_clear_rules() { g_rules.clear(); }

// the runtime
void **__cudaRegisterFatBinary(void *)
{
    static void *h = nullptr;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *fn, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *)
{
    g_kernels[fn] = name;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn)
{
    *k = (cudaKernel_t)fn;
    return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, CUstream_st *stream)
{
    g_config.push_back({grid, block, smem, stream});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream)
{
    const Config c = g_config.back();
    g_config.pop_back();
    *grid = c.grid;
    *block = c.block;
    *smem = c.smem;
    *(cudaStream_t *)stream = c.stream;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3, void **args, size_t, cudaStream_t)
{
    return launch((const void *)k, grid, args, false);
}
cudaError_t cudaLaunchKernel(const void *fn, dim3 grid, dim3, void **args, size_t, cudaStream_t)
{
    return launch(fn, grid, args, false);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fn, void **args)
{
    return launch(fn, c->gridDim, args, false);
}
cudaError_t cudaLaunchCooperativeKernel(const void *fn, dim3 grid, dim3, void **args, size_t, cudaStream_t)
{
    return launch(fn, grid, args, true);
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **p, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *q)
{
    *p = (void *)encode;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
    memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeDevice;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *)
{
    *p = nullptr;
    return result(cudaErrorInvalidSymbol);
}
cudaError_t cudaGetDeviceCount(int *n)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError()
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return g_last; }
const char *cudaGetErrorString(cudaError_t) { return "an error of the stand-in runtime"; }
cudaError_t cudaMalloc(void **p, size_t bytes) { return allocate(p, bytes); }
cudaError_t cudaMallocAsync(void **p, size_t bytes, cudaStream_t) { return allocate(p, bytes); }
cudaError_t cudaFree(void *p) { return release(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return release(p); }
cudaError_t cudaMallocHost(void **p, size_t bytes)
{
    *p = calloc(bytes, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind)
{
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n)
{
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t)
{
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    *s = (cudaStream_t)calloc(1, 1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    g_capture = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g)
{
    g_capture = false;
    *g = (cudaGraph_t)calloc(1, 1);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long)
{
    *e = (cudaGraphExec_t)calloc(1, 1);
    return cudaSuccess;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo *) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t)
{
    g_log += "graph\n";
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g)
{
    free(g);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e)
{
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e)
{
    *e = (cudaEvent_t)calloc(1, 1);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 1.0f;
    return cudaSuccess;
}
}
