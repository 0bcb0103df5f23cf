// A CUDA runtime for tests of the engine's host code without a GPU: the
// engine's own objects are linked against this file instead of the toolkit's
// runtime.  Device memory is zeroed host memory, kernels are not run, every
// call succeeds unless a test says otherwise, and the calls whose order or
// count matters are written to a log, one "name|stream|detail" a line.
#include <cuda_runtime_api.h>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {

struct Fail {
    int skip, count;
    cudaError_t err;
    std::string until;
};
std::mutex mu;
std::string text;
std::map<std::string, Fail> fails;
std::map<const void *, std::string> &kernels = *new std::map<const void *, std::string>();
std::map<void *, size_t> live;
size_t live_bytes = 0, peak_bytes = 0;
std::vector<size_t> free_list; // answers of cudaMemGetInfo in turn; the last one stays
std::string gate; // calls of this name wait for each other ...
int gate_left = 0; // ... until this many have come
std::condition_variable gate_cv;
size_t next_handle = 0x1000;
cudaError_t last = cudaSuccess;
thread_local struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} config;

cudaError_t call(const char *name, cudaStream_t s, const std::string &detail = "")
{
    text += std::string(name) + "|" + std::to_string((size_t)s) + "|" + detail + "\n";
    for (auto it = fails.begin(); it != fails.end();)
        it = it->second.until == name ? fails.erase(it) : std::next(it);
    auto it = fails.find(name);
    if (it == fails.end()) return cudaSuccess;
    if (it->second.skip > 0) {
        it->second.skip--;
        return cudaSuccess;
    }
    const cudaError_t e = it->second.err;
    if (it->second.count > 0 && --it->second.count == 0) fails.erase(it);
    return last = e;
}
cudaError_t simple(const char *name, cudaStream_t s = nullptr, const std::string &detail = "")
{
    std::unique_lock<std::mutex> lk(mu);
    if (gate_left > 0 && gate == name) {
        if (--gate_left == 0) gate_cv.notify_all();
        else gate_cv.wait_for(lk, std::chrono::seconds(10), [] { return gate_left <= 0; });
    }
    return call(name, s, detail);
}
template <class T> cudaError_t handle(const char *name, T *out)
{
    std::lock_guard<std::mutex> lk(mu);
    const cudaError_t e = call(name, nullptr);
    if (e == cudaSuccess) *out = reinterpret_cast<T>(next_handle++);
    return e;
}
cudaError_t take(const char *name, void **p, size_t bytes, cudaStream_t s)
{
    std::lock_guard<std::mutex> lk(mu);
    const cudaError_t e = call(name, s, std::to_string(bytes));
    if (e != cudaSuccess) return e;
    *p = calloc(bytes ? bytes : 1, 1);
    live[*p] = bytes;
    live_bytes += bytes;
    if (live_bytes > peak_bytes) peak_bytes = live_bytes;
    return cudaSuccess;
}
cudaError_t give(const char *name, void *p, cudaStream_t s)
{
    std::lock_guard<std::mutex> lk(mu);
    if (!p) return cudaSuccess;
    auto it = live.find(p);
    const cudaError_t e = call(name, s, it == live.end() ? "unknown" : std::to_string(it->second));
    if (e != cudaSuccess || it == live.end()) return e;
    live_bytes -= it->second;
    live.erase(it);
    free(p);
    return cudaSuccess;
}
const char *kind_name(cudaMemcpyKind k)
{
    return k == cudaMemcpyHostToDevice ? "H2D " : k == cudaMemcpyDeviceToHost ? "D2H " : "D2D ";
}

} // namespace

extern "C" {

// ---- what the tests call
void fake_reset()
{
    std::lock_guard<std::mutex> lk(mu);
    text.clear();
    fails.clear();
    last = cudaSuccess;
    free_list.clear();
    peak_bytes = live_bytes;
}
size_t fake_log(char *out, size_t cap)
{
    std::lock_guard<std::mutex> lk(mu);
    if (out && cap) snprintf(out, cap, "%s", text.c_str());
    return text.size();
}
// After `skip` more calls of `name`, `count` of them fail (all, if negative),
// or all until a call of `until`.
void fake_fail(const char *name, int skip, int count, int err, const char *until)
{
    std::lock_guard<std::mutex> lk(mu);
    fails[name] = Fail{skip, count, (cudaError_t)err, until ? until : ""};
}
void fake_free_bytes(const size_t *v, int n)
{
    std::lock_guard<std::mutex> lk(mu);
    free_list.assign(v, v + n);
}
// The next `count` calls of `name` return only once all of them have come.
void fake_gather(const char *name, int count)
{
    std::lock_guard<std::mutex> lk(mu);
    gate = name;
    gate_left = count;
}
size_t fake_live_bytes() { return live_bytes; }
size_t fake_peak_bytes() { return peak_bytes; }

// ---- registration and launches (as nvcc's host code calls them)
void **__cudaRegisterFatBinary(void *) { return (void **)calloc(1, sizeof(void *)); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *)
{
    kernels[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream)
{
    config = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream)
{
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *(cudaStream_t *)stream = config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *entry)
{
    *k = (cudaKernel_t)entry;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **, size_t, cudaStream_t s)
{
    return simple("launch", s, kernels[(const void *)k]);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **)
{
    return simple("launch", c->stream, kernels[f]);
}

// ---- the runtime
cudaError_t cudaGetLastError()
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }
cudaError_t cudaGetDeviceCount(int *n)
{
    *n = 1;
    return simple("cudaGetDeviceCount");
}
cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int)
{
    *v = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return simple("cudaDeviceSynchronize"); }
cudaError_t cudaMemGetInfo(size_t *fr, size_t *tot)
{
    std::lock_guard<std::mutex> lk(mu);
    const cudaError_t e = call("cudaMemGetInfo", nullptr);
    *tot = (size_t)1 << 40;
    *fr = free_list.empty() ? *tot : free_list.front();
    if (free_list.size() > 1) free_list.erase(free_list.begin());
    return e;
}
cudaError_t cudaMalloc(void **p, size_t n) { return take("cudaMalloc", p, n, nullptr); }
cudaError_t cudaFree(void *p) { return give("cudaFree", p, nullptr); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return take("cudaHostAlloc", p, n, nullptr); }
cudaError_t cudaMallocHost(void **p, size_t n) { return take("cudaHostAlloc", p, n, nullptr); }
cudaError_t cudaFreeHost(void *p) { return give("cudaFreeHost", p, nullptr); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { return handle("cudaMemPoolCreate", p); }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return simple("cudaMemPoolTrimTo"); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t s)
{
    return take("cudaMallocFromPoolAsync", p, n, s);
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) { return give("cudaFreeAsync", p, s); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k)
{
    const cudaError_t e = simple("cudaMemcpy", nullptr, kind_name(k) + std::to_string(n));
    if (e == cudaSuccess) memcpy(d, s, n);
    return e;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st)
{
    const cudaError_t e = simple("cudaMemcpyAsync", st, kind_name(k) + std::to_string(n));
    if (e == cudaSuccess) memcpy(d, s, n);
    return e;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind k,
                              cudaStream_t st)
{
    const cudaError_t e = simple("cudaMemcpyAsync", st, kind_name(k) + std::to_string(w * h));
    for (size_t i = 0; e == cudaSuccess && i < h; i++) memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
    return e;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s)
{
    const cudaError_t e = simple("cudaMemsetAsync", s, std::to_string(n));
    if (e == cudaSuccess) memset(p, v, n);
    return e;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle("cudaStreamCreate", s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return simple("cudaStreamSynchronize", s); }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c)
{
    *c = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { return handle("cudaStreamEndCapture", g); }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m)
{
    static thread_local cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
    const cudaStreamCaptureMode was = mode;
    mode = *m;
    *m = was;
    return simple("cudaThreadExchangeStreamCaptureMode", nullptr,
                  mode == cudaStreamCaptureModeRelaxed ? "relaxed" : "other");
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *g, cudaGraph_t, unsigned long long)
{
    return handle("cudaGraphInstantiate", g);
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { return simple("cudaGraphLaunch", s); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle("cudaEventCreate", e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle("cudaEventCreate", e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return simple("cudaEventDestroy"); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) { return simple("cudaEventRecord", s); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return simple("cudaEventSynchronize"); }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 0.5f;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *)
{
    static char area[2 << 20];
    *p = area;
    return cudaSuccess;
}

} // extern "C"
