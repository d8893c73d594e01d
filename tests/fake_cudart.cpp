// A CUDA runtime on host memory, for tests of the host paths that a GPU shows only when a device call fails: the library
// links libcudart dynamically, so a process that finds this one first runs all of its host code without a device. Device
// memory is host memory, copies and memsets are done at once, kernels are not run: each launch is shown to a callback.
// Built with the soname of the real runtime; the test side drives it through the fake_* functions.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

namespace {
std::recursive_mutex mu;
using Lock = std::lock_guard<std::recursive_mutex>;
std::map<void *, size_t> dev_mem;                        // live device allocations
size_t dev_bytes = 0, dev_peak = 0;
std::map<const void *, std::string> kernel_names;
// work issued to a stream and how much of it the host has waited for; what an event or a stream stands behind, by stream
struct Stream { long long issued = 0, done = 0; };
std::map<cudaStream_t, Stream> streams;
typedef std::map<cudaStream_t, long long> Behind;
std::map<cudaStream_t, Behind> stream_behind;
std::map<cudaEvent_t, Behind> event_behind;
void merge(Behind &a, const Behind &b) { for (auto &e : b) if (a[e.first] < e.second) a[e.first] = e.second; }
void wait_all() { for (auto &s : streams) s.second.done = s.second.issued; }
void wait_stream(cudaStream_t s) {
    streams[s].done = streams[s].issued;
    for (auto &e : stream_behind[s]) if (streams[e.first].done < e.second) streams[e.first].done = e.second;
}
std::map<cudaStream_t, std::vector<std::function<void()>>> capturing;
std::map<std::string, long long> calls;
std::string fail_name;                                   // the fail_at-th call of this function from now on fails
long long fail_at = 0;
long long slow_at = 0;                                   // the slow_at-th wait of the host from now on takes slow_ms
int slow_ms = 0;
void take_time() {                                       // (outside the lock: the thread waits, the others go on)
    int ms = 0;
    {
        Lock l(mu);
        if (slow_at && --slow_at == 0) ms = slow_ms;
    }
    if (ms) usleep(1000 * ms);
}
typedef void (*launch_cb)(const char *kernel, void **args, int recorded);   // kernel "": a graph is launched
typedef void (*hook_cb)();
launch_cb on_launch = nullptr;
hook_cb on_capture = nullptr;
thread_local cudaError_t last_error = cudaSuccess;
thread_local cudaStreamCaptureMode capture_mode = cudaStreamCaptureModeGlobal;
bool foreign_capture = false;                            // another library of the process records in global mode
long long broken_captures = 0;
// calls that end such a recording unless their thread has asked for the relaxed mode
void unsafe_call() { if (foreign_capture && capture_mode != cudaStreamCaptureModeRelaxed) broken_captures++; }
thread_local dim3 cfg_grid, cfg_block;
thread_local size_t cfg_smem;
thread_local cudaStream_t cfg_stream;
uintptr_t next_handle = 0x1000;

bool fails(const char *name) {
    calls[name]++;
    if (fail_name != name || --fail_at != 0) return false;
    fail_name.clear();
    last_error = cudaErrorUnknown;
    return true;
}
template <typename T> T handle() { next_handle += 16; return reinterpret_cast<T>(next_handle); }
// device work: done now, or recorded when the stream is being captured
template <typename F> cudaError_t work(cudaStream_t st, F f) {
    auto c = capturing.find(st);
    if (c != capturing.end()) { c->second.push_back(f); return cudaSuccess; }
    streams[st].issued++;
    f();
    return cudaSuccess;
}
// kernel arguments live on the caller's stack: a recorded launch is shown when it is recorded
cudaError_t launch(const void *func, void **args, cudaStream_t st) {
    hook_cb hook = nullptr;
    {
        Lock l(mu);
        if (fails("cudaLaunchKernel")) return cudaErrorLaunchFailure;
        const bool recorded = capturing.count(st) != 0;
        if (recorded) capturing[st].push_back([] {});
        else streams[st].issued++;
        if (on_launch) on_launch(kernel_names[func].c_str(), args, recorded);
        if (recorded) { hook = on_capture; on_capture = nullptr; }
    }
    if (hook) hook();                                    // once, in the middle of a capture, outside the lock
    return cudaSuccess;
}
std::map<cudaGraph_t, std::vector<std::function<void()>>> graphs;
std::map<cudaGraphExec_t, std::vector<std::function<void()>>> execs;
int encode_tiled(...) { return 0; }
}  // namespace

extern "C" {
// ---- driven by the test
void fake_reset() { Lock l(mu); calls.clear(); fail_name.clear(); fail_at = 0; dev_peak = dev_bytes; }
void fake_fail(const char *name, long long nth) { Lock l(mu); fail_name = name; fail_at = nth; }
void fake_slow(long long nth, int ms) { Lock l(mu); slow_at = nth; slow_ms = ms; }
int fake_failed() { Lock l(mu); return fail_name.empty(); }
long long fake_calls(const char *name) { Lock l(mu); return calls[name]; }
int fake_pending() {                                     // streams with work nobody has waited for
    Lock l(mu);
    int n = 0;
    for (auto &s : streams) n += s.second.done < s.second.issued;
    return n;
}
size_t fake_device_bytes() { Lock l(mu); return dev_bytes; }
size_t fake_device_peak() { Lock l(mu); return dev_peak; }
size_t fake_room(const void *p) {                        // bytes from p to the end of its allocation, 0 outside of all
    Lock l(mu);
    for (auto &m : dev_mem) if (p >= m.first && p < (char *)m.first + m.second) return (size_t)((char *)m.first + m.second - (char *)p);
    return 0;
}
void fake_on_launch(launch_cb cb) { Lock l(mu); on_launch = cb; }
void fake_on_capture(hook_cb cb) { Lock l(mu); on_capture = cb; }

void fake_foreign_capture(int on) { Lock l(mu); foreign_capture = on; broken_captures = 0; }
long long fake_broken_captures() { Lock l(mu); return broken_captures; }

// ---- registration
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *) { kernel_names[host] = name; }
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) { cfg_grid = g; cfg_block = b; cfg_smem = s; cfg_stream = st; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) { *g = cfg_grid; *b = cfg_block; *s = cfg_smem; *(cudaStream_t *)st = cfg_stream; return cudaSuccess; }

// ---- device
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrCooperativeLaunch ? 1 : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { Lock l(mu); wait_all(); return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last_error; last_error = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "an error of the fake runtime"; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { *p = nullptr; return cudaErrorInvalidSymbol; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **p, unsigned long long, cudaDriverEntryPointQueryResult *q) {
    *p = (void *)encode_tiled;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

// ---- memory
cudaError_t cudaMalloc(void **p, size_t n) {
    Lock l(mu);
    unsafe_call();
    if (fails("cudaMalloc")) return cudaErrorMemoryAllocation;
    *p = calloc(1, n);
    dev_mem[*p] = n;
    dev_bytes += n;
    if (dev_bytes > dev_peak) dev_peak = dev_bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {                          // waits for the device, as the real one does
    Lock l(mu);
    calls["cudaFree"]++;
    unsafe_call();
    if (!p) return cudaSuccess;
    if (!dev_mem.count(p)) return cudaErrorInvalidValue;
    wait_all();
    dev_bytes -= dev_mem[p];
    dev_mem.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMallocHost(void **p, size_t n) { Lock l(mu); if (fails("cudaMallocHost")) return cudaErrorMemoryAllocation; *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { Lock l(mu); if (fails("cudaHostAlloc")) return cudaErrorMemoryAllocation; *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { memset(a, 0, sizeof(*a)); a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    Lock l(mu);
    if (fails("cudaMemcpyAsync")) return cudaErrorInvalidValue;
    return work(st, [=] { memcpy(d, s, n); });
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t st) {
    Lock l(mu);
    return work(st, [=] { for (size_t i = 0; i < h; i++) memcpy((char *)d + i * dp, (const char *)s + i * sp, w); });
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t st) {
    Lock l(mu);
    if (fails("cudaMemsetAsync")) return cudaErrorInvalidValue;
    return work(st, [=] { memset(p, v, n); });
}

// ---- streams and events
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { Lock l(mu); if (fails("cudaStreamCreate")) return cudaErrorMemoryAllocation; *s = handle<cudaStream_t>(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { Lock l(mu); streams.erase(s); stream_behind.erase(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { take_time(); Lock l(mu); calls["cudaStreamSynchronize"]++; wait_stream(s); return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t s) { Lock l(mu); unsafe_call(); return streams[s].done < streams[s].issued ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { Lock l(mu); calls["cudaStreamWaitEvent"]++; merge(stream_behind[s], event_behind[e]); return work(s, [] {}); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { Lock l(mu); if (fails("cudaEventCreate")) return cudaErrorMemoryAllocation; *e = handle<cudaEvent_t>(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    Lock l(mu);
    if (fails("cudaEventRecord")) return cudaErrorInvalidValue;
    event_behind[e] = stream_behind[s];
    event_behind[e][s] = streams[s].issued;
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
    Lock l(mu);
    unsafe_call();
    for (auto &b : event_behind[e]) if (streams.count(b.first) && streams[b.first].done < b.second) return cudaErrorNotReady;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    take_time();
    Lock l(mu);
    for (auto &b : event_behind[e]) if (streams.count(b.first) && streams[b.first].done < b.second) streams[b.first].done = b.second;
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

// ---- launches and graphs
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t, cudaStream_t st) { return launch(f, args, st); }
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3, dim3, void **args, size_t, cudaStream_t st) { return launch(f, args, st); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) { return launch(f, args, c->stream); }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) { std::swap(*m, capture_mode); return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { Lock l(mu); capturing[s]; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
    Lock l(mu);
    *g = handle<cudaGraph_t>();
    graphs[*g] = capturing[s];
    capturing.erase(s);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) { Lock l(mu); *x = handle<cudaGraphExec_t>(); execs[*x] = graphs[g]; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { Lock l(mu); graphs.erase(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { Lock l(mu); calls["cudaGraphExecDestroy"]++; execs.erase(x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
    Lock l(mu);
    if (fails("cudaGraphLaunch")) return cudaErrorInvalidValue;
    streams[s].issued++;
    if (on_launch) on_launch("", nullptr, 0);
    for (auto &f : execs[x]) f();
    return cudaSuccess;
}
}  // extern "C"
