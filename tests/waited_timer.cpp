// WaitedTimer on a runtime that is made up: what it leaves behind when a call fails, and in which capture mode it calls.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../let-it-slide_b200/csrc/waited_timer.cuh"

static int g_calls, g_fail_at, g_host, g_device, g_streams;
static cudaStreamCaptureMode g_mode = cudaStreamCaptureModeGlobal;
#define CHECK(x) ((x) ? (void)0 : (std::printf("line %d: %s\n", __LINE__, #x), std::exit(1)))
static cudaError_t step() {      // of a call that another thread's capture forbids
    CHECK(g_mode == cudaStreamCaptureModeRelaxed);
    return ++g_calls == g_fail_at ? cudaErrorMemoryAllocation : cudaSuccess;
}
static cudaError_t allocate(void **p, size_t size, int &count) {
    const cudaError_t e = step();
    if (e == cudaSuccess) *p = std::malloc(size), ++count;
    return e;
}
extern "C" {
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *mode) {
    const cudaStreamCaptureMode before = g_mode;
    g_mode = *mode, *mode = before;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t size, unsigned int) { return allocate(p, size, g_host); }
cudaError_t cudaMalloc(void **p, size_t size) { return allocate(p, size, g_device); }
cudaError_t cudaFreeHost(void *p) {
    CHECK(g_mode == cudaStreamCaptureModeRelaxed);
    std::free(p), --g_host;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    CHECK(g_mode == cudaStreamCaptureModeRelaxed);
    std::free(p), --g_device;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned int flags) {
    CHECK(flags == cudaStreamNonBlocking);
    const cudaError_t e = step();
    if (e == cudaSuccess) *s = reinterpret_cast<cudaStream_t>(&g_streams), ++g_streams;
    return e;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return --g_streams, cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t size, cudaMemcpyKind, cudaStream_t s) {
    CHECK(s);                    // not the legacy stream
    const cudaError_t e = step();
    if (e == cudaSuccess) std::memcpy(to, from, size);
    return e;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return step(); }
}

int main() {
    for (int fail_at = 1; fail_at <= 5; ++fail_at) {
        rptc::WaitedTimer t;
        t.ticket = 41;
        g_calls = 0, g_fail_at = fail_at;
        CHECK(t.ready() != cudaSuccess);
        CHECK(!t.device && !t.host && g_host == 0 && g_device == 0 && g_streams == 0 && g_mode == cudaStreamCaptureModeGlobal);
        g_fail_at = 0;
        CHECK(t.ready() == cudaSuccess);
        CHECK(t.device && t.device->begin == ~0ull && t.device->ended == 0 && t.host->ticket == 41 && g_host == 1 && g_device == 1 && g_streams == 0);
        CHECK(g_mode == cudaStreamCaptureModeGlobal);
        g_calls = 0;
        CHECK(t.ready() == cudaSuccess && g_calls == 0);
        t.release();
        CHECK(g_host == 0 && g_device == 0 && g_mode == cudaStreamCaptureModeGlobal);
        CHECK(t.ready() == cudaSuccess);
    }
    CHECK(g_host == 0 && g_device == 0);
    return 0;
}
