// A stand-in for the CUDA runtime on a machine without a GPU: device memory is host
// memory, copies and fills happen at once, kernels do nothing.  It records
//  - launches, copies and fills on another stream while work of the legacy stream (allocations, copies,
//    fills, kernels) may still be under way: no host wait and no event orders them
//    (a copy to the device from pageable memory may return before it has arrived);
//  - kernels in launch order, and fails the launches whose name holds FAKE_CUDA_FAIL.
// fake_report() returns one line per event: "unordered NAME", "launch NAME", "grid X Y
// NAME" or "capture begin".
// FAKE_CUDA_SMS: the device's SM count (148).
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<const void *, std::string> names;
std::string report;
long legacy = 0, waited = 0;                  // legacy-stream work issued / waited for by the host
std::map<void *, long> stream_waited, event_at;
cudaError_t last = cudaSuccess;
dim3 cfg_grid, cfg_block;
size_t cfg_smem;
cudaStream_t cfg_stream;
long handles = 0x1000;
bool capturing = false;

void *handle() { return reinterpret_cast<void *>(handles += 16); }
cudaError_t set(cudaError_t e)
{
    if (e != cudaSuccess) last = e;
    return e;
}
void touch(cudaStream_t s) { legacy += s == nullptr; }
void join(cudaStream_t s) { if (!s) waited = legacy; }
void check(cudaStream_t s, const std::string &what)
{
    if (s && !capturing && std::max(waited, stream_waited[s]) < legacy) report += "unordered " + what + "\n";
}
cudaError_t launch(const void *f, dim3 grid, cudaStream_t s)
{
    const std::string &n = names[f];
    check(s, n);
    report += "launch " + n + "\ngrid " + std::to_string(grid.x) + " " + std::to_string(grid.y) + " " + n + "\n";
    touch(s);
    const char *fail = std::getenv("FAKE_CUDA_FAIL");
    return set(fail && *fail && n.find(fail) != std::string::npos ? cudaErrorInvalidConfiguration : cudaSuccess);
}
}  // namespace

extern "C" {
const char *fake_report() { return report.c_str(); }
void fake_reset() { report.clear(); }

void **__cudaRegisterFatBinary(void *) { static void *h = nullptr; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *,
                            dim3 *, int *) { names[f] = name; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s)
{
    cfg_grid = g; cfg_block = b; cfg_smem = m; cfg_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s)
{
    *g = cfg_grid; *b = cfg_block; *m = cfg_smem; *static_cast<cudaStream_t *>(s) = cfg_stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3, void **, size_t, cudaStream_t s) { return launch(f, g, s); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) { return launch(f, c->gridDim, c->stream); }

cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }

cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    const char *sms = std::getenv("FAKE_CUDA_SMS");
    *v = a == cudaDevAttrMultiProcessorCount ? (sms ? std::atoi(sms) : 148) : a == cudaDevAttrComputeCapabilityMajor ? 10
         : a == cudaDevAttrComputeCapabilityMinor ? 0 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { waited = legacy; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) { std::memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) { *n = 8; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { static void *m = std::calloc(1, 64u << 20); *p = m; return cudaSuccess; }

cudaError_t cudaMallocHost(void **p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t s)
{
    *p = std::calloc(1, n);
    touch(s);
    return *p ? cudaSuccess : set(cudaErrorMemoryAllocation);
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { *p = static_cast<cudaMemPool_t>(handle()); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k)
{
    std::memcpy(d, s, n);
    touch(nullptr);
    if (k == cudaMemcpyDeviceToHost) join(nullptr);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    check(st, "copy");
    std::memcpy(d, s, n);
    touch(st);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t s)
{
    check(s, "fill");
    std::memset(d, v, n);
    touch(s);
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = static_cast<cudaStream_t>(handle()); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { join(s); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = static_cast<cudaEvent_t>(handle()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    event_at[e] = s ? std::max(waited, stream_waited[s]) : legacy;
    return cudaSuccess;
}
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned) { return cudaEventRecord(e, s); }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { waited = std::max(waited, event_at[e]); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { *t = 1.f; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    stream_waited[s] = std::max(stream_waited[s], event_at[e]);
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    capturing = true;
    report += "capture begin\n";
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { capturing = false; *g = static_cast<cudaGraph_t>(handle()); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { *e = static_cast<cudaGraphExec_t>(handle()); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t *, size_t *n) { *n = 0; return cudaSuccess; }
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType *) { return cudaSuccess; }
}
