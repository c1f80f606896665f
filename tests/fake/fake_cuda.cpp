// A CUDA runtime for tests of libmdg's host side without a GPU: linked with mdg_api.o
// in place of the real one (fake_kernels.cu: the kernels).  Device memory is host
// memory, work runs when it is issued, or when the graph it was captured into is
// launched, and any call can be made to return an error (fake_fail).
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

namespace {

using Op = std::function<void()>;
struct Stream {
    unsigned flags = 0;
};
std::vector<Op> *capture = nullptr;  // the graph being captured, if any
cudaStream_t capturing = nullptr;    // and the stream that began it
std::map<std::string, int> calls, fail_at;

// counts the call; true if it is the one that fake_fail picked
bool fails(const char *name) {
    const int n = ++calls[name];
    auto it = fail_at.find(name);
    if (it == fail_at.end() || n != it->second) return false;
    fail_at.erase(it);
    return true;
}

}  // namespace

cudaError_t issue(const char *name, std::function<void()> op) {
    if (fails(name)) return cudaErrorMemoryAllocation;
    if (capture) capture->push_back(std::move(op));
    else op();
    return cudaSuccess;
}

#define FAKE_API extern "C" __attribute__((visibility("default")))

FAKE_API void fake_reset() {
    calls.clear();
    fail_at.clear();
}
// the nth call from now on of `name` fails
FAKE_API void fake_fail(const char *name, int nth) { fail_at[name] = calls[name] + nth; }
FAKE_API int fake_calls(const char *name) { return calls[name]; }

// ---- the runtime -----------------------------------------------------------------
extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
    *v = 4;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) {
    *lo = *hi = 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "an error of the fake runtime"; }
cudaError_t cudaMalloc(void **p, size_t n) {
    if (fails("cudaMalloc")) return cudaErrorMemoryAllocation;
    *p = calloc(n, 1);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
    if (fails("cudaMallocHost")) return cudaErrorMemoryAllocation;
    *p = calloc(n, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return issue("cudaMemcpyAsync", [=] { memcpy(d, s, n); });
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
    return issue("cudaMemsetAsync", [=] { memset(d, v, n); });
}
cudaError_t cudaMemset2DAsync(void *d, size_t pitch, int v, size_t w, size_t h, cudaStream_t) {
    return issue("cudaMemset2DAsync", [=] {
        for (size_t r = 0; r < h; ++r) memset((char *)d + r * pitch, v, w);
    });
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned flags) {
    *s = (cudaStream_t) new Stream{flags};
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned flags, int) {
    return cudaStreamCreateWithFlags(s, flags);
}
cudaError_t cudaStreamGetFlags(cudaStream_t s, unsigned *flags) {
    *flags = ((Stream *)s)->flags;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    delete (Stream *)s;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    return capture && s == capturing ? cudaErrorStreamCaptureUnsupported : cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = (cudaEvent_t) new Stream();
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete (Stream *)e;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *st) {
    if (s == cudaStreamLegacy) return cudaErrorStreamCaptureImplicit;
    *st = capture && s == capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    if (fails("cudaStreamBeginCapture")) return cudaErrorMemoryAllocation;
    if (s == cudaStreamLegacy) return cudaErrorStreamCaptureUnsupported;
    if (capture) return cudaErrorIllegalState;
    capture = new std::vector<Op>();
    capturing = s;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
    if (!capture || s != capturing) return cudaErrorIllegalState;
    *g = (cudaGraph_t)capture;
    capture = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long) {
    if (fails("cudaGraphInstantiate")) return cudaErrorMemoryAllocation;
    *e = (cudaGraphExec_t) new std::vector<Op>(*(std::vector<Op> *)g);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    if (fails("cudaGraphLaunch")) return cudaErrorMemoryAllocation;
    if (capture) return cudaErrorStreamCaptureUnsupported;
    for (Op &op : *(std::vector<Op> *)e) op();
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    delete (std::vector<Op> *)g;
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
    delete (std::vector<Op> *)e;
    return cudaSuccess;
}
}

// a caller's own stream, and its capture
FAKE_API void *fake_stream(unsigned flags) { return new Stream{flags}; }
FAKE_API int fake_begin_capture(void *s) {
    return cudaStreamBeginCapture((cudaStream_t)s, cudaStreamCaptureModeRelaxed);
}
FAKE_API int fake_end_capture_and_run(void *s) {
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture((cudaStream_t)s, &g);
    if (e != cudaSuccess) return e;
    for (Op &op : *(std::vector<Op> *)g) op();
    return cudaGraphDestroy(g);
}

