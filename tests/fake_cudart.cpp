// A stand-in for the CUDA runtime, preloaded over the real one, that runs the
// library's host code without a GPU: allocations are host memory, kernels do
// nothing, and the failures a test asks for (an allocation that does not fit,
// a copy that is refused, a launch above its kernel's shared-memory limit)
// come back as error codes.  Every call is logged for the test to read.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {

std::recursive_mutex mu;
std::string log_text;
std::map<void *, size_t> live;
size_t live_bytes = 0, max_single = ~(size_t)0, max_total = ~(size_t)0;
int fill = 0;            // byte of fresh allocations
int refuse_d2h = 0;      // the n-th copy to the host from now on fails
bool deferred = false;   // asynchronous copies happen when their stream is waited for (pinned memory)
bool capturing = false;
long next_handle = 16;
cudaError_t last = cudaSuccess;
std::map<const void *, std::string> names;
std::map<const void *, int> limits;
std::map<const void *, std::vector<char>> symbols;
std::map<void *, std::deque<std::function<void()>>> pending;
struct Config { dim3 grid, block; size_t smem; void *stream; };
std::vector<Config> configs;

void note(const std::string &s) { log_text += s + "\n"; }
cudaError_t fail(cudaError_t e) { return last = e; }
std::string id(void *p) { return std::to_string((long)p); }
void drain(void *s) {
    auto &q = pending[s];
    while (!q.empty()) {
        auto f = q.front();
        q.pop_front();
        f();
    }
}
cudaError_t copy(void *dst, const void *src, size_t n, int kind, void *stream, bool async) {
    std::lock_guard<std::recursive_mutex> g(mu);
    const char *k = kind == cudaMemcpyHostToDevice ? "h2d" : kind == cudaMemcpyDeviceToHost ? "d2h" : "d2d";
    note(std::string(k) + " " + std::to_string(n) + " stream " + id(stream));
    if (kind == cudaMemcpyDeviceToHost && refuse_d2h && --refuse_d2h == 0) return fail(cudaErrorUnknown);
    if (async && deferred) pending[stream].push_back([=] { std::memcpy(dst, src, n); });
    else std::memcpy(dst, src, n);
    return cudaSuccess;
}
cudaError_t launch(const void *f, size_t smem, void *stream) {
    std::lock_guard<std::recursive_mutex> g(mu);
    const int lim = limits.count(f) ? limits[f] : 48 * 1024;
    if (smem > (size_t)lim) {
        note("refused " + names[f] + " smem " + std::to_string(smem) + " limit " + std::to_string(lim));
        return fail(cudaErrorInvalidValue);
    }
    note((capturing ? "capture " : "launch ") + names[f] + " smem " + std::to_string(smem) + " stream " + id(stream));
    return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- the test's side ----
void fake_memory(size_t single, size_t total) { max_single = single; max_total = total; }
void fake_fill(int byte) { fill = byte; }
void fake_refuse_d2h(int n) { refuse_d2h = n; }
void fake_deferred(int on) { deferred = on; }
size_t fake_live_bytes() { return live_bytes; }
void fake_log_clear() { log_text.clear(); }
size_t fake_log(char *out, size_t cap) {
    std::lock_guard<std::recursive_mutex> g(mu);
    if (out && cap) {
        const size_t n = std::min(cap - 1, log_text.size());
        std::memcpy(out, log_text.data(), n);
        out[n] = 0;
    }
    return log_text.size();
}

// ---- registration ----
void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    names[host] = name;
}
void __cudaRegisterVar(void **, char *host, char *, const char *, int, size_t size, int, int) {
    symbols[host].assign(size, 0);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> g(mu);
    configs.push_back({grid, block, smem, s});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s) {
    std::lock_guard<std::recursive_mutex> g(mu);
    const Config c = configs.back();
    configs.pop_back();
    *grid = c.grid;
    *block = c.block;
    *smem = c.smem;
    *(void **)s = c.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **, size_t smem, cudaStream_t s) {
    return launch((const void *)k, smem, s);
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t smem, cudaStream_t s) {
    return launch(f, smem, s);
}

// ---- device ----
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    std::memset(p, 0, sizeof *p);
    std::strcpy(p->name, "stand-in");
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "an error"; }

// ---- memory ----
cudaError_t cudaMalloc(void **p, size_t n) {
    std::lock_guard<std::recursive_mutex> g(mu);
    note("malloc " + std::to_string(n));
    if (n > max_single || live_bytes + n > max_total) return fail(cudaErrorMemoryAllocation);
    *p = std::calloc(n, 1);
    if (fill) std::memset(*p, fill, n);
    live[*p] = n;
    live_bytes += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::recursive_mutex> g(mu);
    for (auto &q : pending) drain(q.first);
    if (!p) return cudaSuccess;
    note("free " + std::to_string(live[p]));
    live_bytes -= live[p];
    live.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) { return copy(d, s, n, k, nullptr, false); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
    return copy(d, s, n, k, st, true);
}
cudaError_t cudaMemcpyToSymbolAsync(const void *sym, const void *s, size_t n, size_t o, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(symbols[sym].data() + o, s, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) {
    *p = symbols[sym].data();
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> g(mu);
    note("memset " + std::to_string(n));
    if (capturing) return cudaSuccess;
    if (deferred) pending[s].push_back([=] { std::memset(p, v, n); });
    else std::memset(p, v, n);
    return cudaSuccess;
}

// ---- kernels ----
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
    std::lock_guard<std::recursive_mutex> g(mu);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (v > 232448) return fail(cudaErrorInvalidValue);
        limits[f] = v;
        note("limit " + names[f] + " " + std::to_string(v));
    }
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int threads, size_t smem) {
    *n = (int)std::min<size_t>(512 / threads, 232448 / (smem + 1024));   // 128 registers a thread
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int threads, size_t smem,
                                                                   unsigned) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, threads, smem);
}

// ---- streams, events, graphs ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = (cudaStream_t)(next_handle++);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> g(mu);
    drain(s);
    note("sync stream " + id(s));
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    capturing = false;
    *g = (cudaGraph_t)(next_handle++);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    *e = (cudaGraphExec_t)(next_handle++);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { note("graph stream " + id(s)); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)(next_handle++); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

}  // extern "C"
