// host_runtime.cpp -- a CUDA runtime of two make-believe devices on the host, for tests of the
// library's host logic (linked with the library's own object files in place of cudart).  Kernels do
// not run: a launch is recorded with its kernel, device, grid, shared memory and, where the first
// parameter is a DpLaunch, its group size.  Device memory is host memory; allocations are counted and
// may be limited.  A launch with more dynamic shared memory than its kernel may use on the current
// device is refused, as the runtime refuses it.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

extern "C" int dp_launch_group(const void *launch);      // DpLaunch::G (the test compiles it with nvcc)

namespace {
struct Config { dim3 grid, block; size_t smem; void *stream; };
std::mutex mu;
std::map<const void *, std::string> names;
std::map<std::pair<int, const void *>, int> smem_limit;      // per device, as the attribute is
std::map<void *, size_t> allocations;
std::vector<Config> pending;
std::string events;
size_t in_use = 0, most = 0, limit = ~(size_t)0;
int device = 0, capturing = 0;
cudaError_t last = cudaSuccess;

void note(const std::string &s) { events += s + "\n"; }
cudaError_t set(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
std::string name_of(const void *f) { auto it = names.find(f); return it == names.end() ? "?" : it->second; }

cudaError_t record(const void *f, dim3 grid, void **args, size_t smem)
{
    std::lock_guard<std::mutex> lock(mu);
    const std::string n = name_of(f);
    auto it = smem_limit.find({device, f});
    if (smem > (size_t)(it == smem_limit.end() ? 48 << 10 : it->second)) {
        note("refused " + n + " device " + std::to_string(device));
        return set(cudaErrorInvalidValue);
    }
    std::string s = "launch " + n + " device " + std::to_string(device) + " grid " + std::to_string(grid.x);
    if (n.find("8DpLaunch") != std::string::npos) s += " G " + std::to_string(dp_launch_group(args[0]));
    note(s);
    return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- for the tests ----
const char *host_runtime_events() { return events.c_str(); }
void host_runtime_reset() { events.clear(); most = in_use; }
size_t host_runtime_most() { return most; }
void host_runtime_limit(size_t bytes) { limit = bytes; }

// ---- what the compiler's launch code calls ----
void **__cudaRegisterFatBinary(void *) { static void *h[1]; return h; }
void __cudaRegisterFatBinaryEnd(void **) {}
char __cudaInitModule(void **) { return 1; }
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *)
{
    names[f] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st)
{
    pending.push_back({g, b, smem, st});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st)
{
    *g = pending.back().grid; *b = pending.back().block; *smem = pending.back().smem;
    *(void **)st = pending.back().stream;
    pending.pop_back();
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void **args, size_t smem, cudaStream_t)
{
    return record((const void *)k, g, args, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args)
{
    return record(f, c->gridDim, args, c->dynamicSmemBytes);
}

// ---- the runtime ----
cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { if (d < 0 || d > 1) return set(cudaErrorInvalidDevice); device = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrComputeCapabilityMajor ? 10
       : a == cudaDevAttrComputeCapabilityMinor ? 3 : 227 << 10;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { if (lo) *lo = 0; if (hi) *hi = -5; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "host runtime error"; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v)
{
    std::lock_guard<std::mutex> lock(mu);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_limit[{device, f}] = v;
    return cudaSuccess;
}
static cudaError_t occupancy(int *v, const void *f)
{
    std::lock_guard<std::mutex> lock(mu);
    if (capturing) note("occupancy in a capture " + name_of(f));
    *v = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *v, const void *f, int, size_t) { return occupancy(v, f); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *v, const void *f, int, size_t, unsigned) { return occupancy(v, f); }
cudaError_t cudaOccupancyMaxActiveClusters(int *v, const void *, const cudaLaunchConfig_t *) { *v = 64; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { static char x[1 << 16]; *p = x; return cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t n)
{
    std::lock_guard<std::mutex> lock(mu);
    *p = nullptr;
    if (in_use + n > limit) return set(cudaErrorMemoryAllocation);
    void *q = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (q == MAP_FAILED) return set(cudaErrorMemoryAllocation);
    allocations[q] = n;
    in_use += n;
    most = in_use > most ? in_use : most;
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    std::lock_guard<std::mutex> lock(mu);
    auto it = allocations.find(p);
    if (it == allocations.end()) return p ? set(cudaErrorInvalidValue) : cudaSuccess;
    in_use -= it->second;
    munmap(p, it->second);
    allocations.erase(it);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }     // memory starts as zeros

static cudaError_t handle(void **h) { *h = malloc(1); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle((void **)s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return handle((void **)s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle((void **)e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle((void **)e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s)
{
    *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = 1; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { capturing = 0; return handle((void **)g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { return handle((void **)e); }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { free(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
}
