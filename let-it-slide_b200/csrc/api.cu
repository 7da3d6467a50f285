// Host-side plumbing of the C ABI: status strings, device checks, the device status word.
#include "common.cuh"
#include "matmul.cuh"

namespace rptc {

thread_local int g_last_cuda_error = 0;
static thread_local bool g_pdl = false;      // per calling thread: two threads that launch with different settings do not race

int cuda_fail(cudaError_t e) {
    g_last_cuda_error = (int)e;
    (void)cudaGetLastError();   // clear the sticky-free error so that later launches are not blamed for it
    return RPTC_ERR_CUDA;
}

bool pdl_enabled() { return g_pdl; }

static int g_sms[kMaxDevices];
static int g_cc[kMaxDevices];

int current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
    return dev;
}

int num_sms() {
    const int dev = current_device();
    if (dev < 0) return kNumSMsFallback;
    if (g_sms[dev] == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = kNumSMsFallback;
        g_sms[dev] = v;
    }
    return g_sms[dev];
}

// One status word per device (each device that loads this module has its own copy of the symbol).
__device__ unsigned int g_status_word;
static unsigned int *g_status_ptr[kMaxDevices];

unsigned int *device_status_word() {
    const int dev = current_device();
    if (dev < 0) return nullptr;
    if (!g_status_ptr[dev]) {
        void *ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_status_word);
        if (e != cudaSuccess) {
            cuda_fail(e);
            return nullptr;
        }
        g_status_ptr[dev] = static_cast<unsigned int *>(ptr);
    }
    return g_status_ptr[dev];
}

int check_format(const rptc_format *f) {
    if (!f) return RPTC_ERR_ARG;
    if (f->code < RPTC_CODE_LUT || f->code > RPTC_CODE_LITE) return RPTC_ERR_ARG;
    if (f->layout < RPTC_LAYOUT_ROWMAJOR || f->layout > RPTC_LAYOUT_TILED) return RPTC_ERR_ARG;
    if (f->quirk < RPTC_QUIRK_NONE || f->quirk > RPTC_QUIRK_K2_LANE0_CARRY) return RPTC_ERR_ARG;
    if (f->K < 2 || f->K > 4) return RPTC_ERR_ARG;
    if (f->L < 1 || f->L > 16) return RPTC_ERR_ARG;
    if (f->quirk != RPTC_QUIRK_NONE && f->K != 2) return RPTC_ERR_UNSUPPORTED;
    switch (f->code) {
        case RPTC_CODE_LUT:
            if (f->L < 3) return RPTC_ERR_ARG;
            break;
        case RPTC_CODE_HASH:
            if (f->K != 2) return RPTC_ERR_UNSUPPORTED;
            if (f->S < 1 || f->S > 8) return RPTC_ERR_ARG;
            break;
        case RPTC_CODE_LITE:
            if (f->K == 3) return RPTC_ERR_UNSUPPORTED;
            if (f->S < 1 || f->S > 10 || f->S > f->L) return RPTC_ERR_ARG;
            break;
    }
    return RPTC_OK;
}

}  // namespace rptc

using namespace rptc;

extern "C" const char *rptc_strerror(int status) {
    switch (status) {
        case RPTC_OK: return "ok";
        case RPTC_ERR_ARG: return "invalid argument (null pointer or bad enum value)";
        case RPTC_ERR_SHAPE: return "shape violates a divisibility or leading-dimension rule";
        case RPTC_ERR_ALIGN: return "pointer or leading dimension not aligned as required";
        case RPTC_ERR_UNSUPPORTED: return "combination of code, K and layout is not implemented";
        case RPTC_ERR_CUDA: return "a CUDA runtime call failed (see rptc_last_cuda_error)";
        case RPTC_ERR_TIMEOUT: return "a bounded device-side wait ran out";
        case RPTC_ERR_TOO_LARGE: return "size beyond a documented maximum";
        case RPTC_ERR_DEVICE: return "current device is not a compute-capability 10.x GPU";
        case RPTC_ERR_INTERNAL: return "a kernel found its shared-memory plan violated and did nothing";
        case RPTC_ERR_RANGE: return "a sequence position lay outside the KV cache; the access was skipped";
    }
    return "unknown status";
}

extern "C" int rptc_version(void) { return 100; }

extern "C" int rptc_last_cuda_error(void) { return g_last_cuda_error; }

extern "C" void rptc_set_pdl(int enable) { g_pdl = enable != 0; }
extern "C" int rptc_pdl(void) { return g_pdl; }

extern "C" int rptc_check_device(void) {
    const int dev = current_device();
    if (dev < 0) return cuda_fail(cudaErrorNoDevice);
    if (g_cc[dev] == 0) {
        int major = 0;
        RPTC_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
        g_cc[dev] = major;
    }
    return g_cc[dev] == 10 ? RPTC_OK : RPTC_ERR_DEVICE;
}

extern "C" int rptc_device_status(void) {
    unsigned int *w = device_status_word();
    if (!w) return RPTC_ERR_CUDA;
    RPTC_CUDA(cudaDeviceSynchronize());
    unsigned int v = 0;
    RPTC_CUDA(cudaMemcpy(&v, w, sizeof(v), cudaMemcpyDeviceToHost));
    if (v) {
        const unsigned int zero = 0;
        RPTC_CUDA(cudaMemcpy(w, &zero, sizeof(zero), cudaMemcpyHostToDevice));
        if (v == kStatusSmemPlan) return RPTC_ERR_INTERNAL;
        if (v == kStatusPosition) return RPTC_ERR_RANGE;
        return RPTC_ERR_TIMEOUT;
    }
    return RPTC_OK;
}

// ---- device time of a piece of work ------------------------------------------------------------------
namespace rptc {
struct TimerEvents {
    cudaEvent_t begin = nullptr, end = nullptr;
    ~TimerEvents() {      // the thread ends (a runtime that has been shut down before refuses, and holds them no more)
        if (begin) cudaEventDestroy(begin);
        if (end) cudaEventDestroy(end);
    }
};
static thread_local TimerEvents g_timers[kMaxDevices];      // kept: creating a pair costs as much as a launch
static int timer_events(TimerEvents *&t) {
    const int dev = current_device();
    if (dev < 0) return cuda_fail(cudaErrorNoDevice);
    t = &g_timers[dev];
    if (!t->begin) RPTC_CUDA(cudaEventCreate(&t->begin));
    if (!t->end) RPTC_CUDA(cudaEventCreate(&t->end));
    return RPTC_OK;
}
}  // namespace rptc

extern "C" int rptc_timer_begin(rptc_stream_t stream) {
    TimerEvents *t;
    if (int e = rptc_check_device()) return e;
    if (int e = timer_events(t)) return e;
    RPTC_CUDA(cudaEventRecord(t->begin, static_cast<cudaStream_t>(stream)));
    return RPTC_OK;
}

extern "C" int rptc_timer_end(float *ms, rptc_stream_t stream) {
    if (!ms) return RPTC_ERR_ARG;
    TimerEvents *t;
    if (int e = rptc_check_device()) return e;
    if (int e = timer_events(t)) return e;
    RPTC_CUDA(cudaEventRecord(t->end, static_cast<cudaStream_t>(stream)));
    BesideCaptures mode;
    RPTC_CUDA(cudaEventSynchronize(t->end));
    RPTC_CUDA(cudaEventElapsedTime(ms, t->begin, t->end));
    return RPTC_OK;
}

// ---- a matvec whose caller waits for it ----
namespace rptc {
static thread_local WaitedTimer g_waited[kMaxDevices];
// Until the kernel with `ticket` has left its time.  The stream is asked now and then: work that failed leaves none.
static int wait_for(WaitedTimer &t, cudaStream_t stream, float *ms) {
    // Asked behind the launch, under the kernel's time: in front of it the question is 0.2 us of a call.  A capture now holds a kernel that writes to
    // this thread's timer, and must not become a graph: asking for the stream's state ends it.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    RPTC_CUDA(cudaStreamIsCapturing(stream, &capture));
    if (capture != cudaStreamCaptureStatusNone) {
        cudaStreamQuery(stream);
        return cuda_fail(cudaErrorStreamCaptureUnsupported);      // nothing to wait for
    }
    volatile HostTime *h = t.host;
    for (unsigned int spin = 1;; ++spin) {
        if (h->ticket == t.ticket) break;
        if (spin % 4096) continue;
        BesideCaptures mode;
        const cudaError_t e = cudaStreamQuery(stream);
        if (e == cudaErrorNotReady) continue;
        if (e == cudaSuccess && h->ticket == t.ticket) break;
        t.release();
        return e == cudaSuccess ? RPTC_ERR_TIMEOUT : cuda_fail(e);      // the kernel gave up, or the stream failed
    }
    __atomic_thread_fence(__ATOMIC_ACQUIRE);
    *ms = (float)((double)h->ns * 1e-6);
    return RPTC_OK;
}
static bool overlap(const void *a, int64_t a_bytes, const void *b, int64_t b_bytes) {
    const uintptr_t p = reinterpret_cast<uintptr_t>(a), q = reinterpret_cast<uintptr_t>(b);
    return p < q + (uintptr_t)b_bytes && q < p + (uintptr_t)a_bytes;
}
// Whether y may be written while the product is under way: a CTA of gemv_whole stores its rows when others still read (x == y with m == n is
// a call that the product with a kernel behind it answers).
static bool written_apart(const void *y, const void *codes, const void *lut, const void *x, int64_t m, int64_t n, const rptc_format &f) {
    const int64_t lut_bytes = f.code == RPTC_CODE_LUT ? int64_t(2) << f.L : int64_t(4) << f.S;
    return !overlap(y, 2 * m, x, 2 * n) && !overlap(y, 2 * m, lut, lut_bytes) && !overlap(y, 2 * m, codes, m * n / 8 * f.K);
}
}  // namespace rptc

extern "C" int rptc_gemv_timed(const void *codes, const void *lut, const void *x, float *acc, void *y, int64_t m, int64_t n, int x_order,
                               int accumulate, const rptc_format *fmt, float *ms, rptc_stream_t stream) {
    if (!y || !ms) return RPTC_ERR_ARG;
    if (int e = validate_gemv_args(codes, lut, x, n, acc, m, m, n, 1, x_order, fmt)) return e;
    if (int e = rptc_check_device()) return e;
    const int dev = current_device();
    if (dev < 0) return cuda_fail(cudaErrorNoDevice);
    if (gemv_whole_takes(n, x_order, *fmt) && written_apart(y, codes, lut, x, m, n, *fmt)) {
        WaitedTimer &t = g_waited[dev];
        RPTC_CUDA(t.ready());
        const int e = gemv_whole(codes, lut, x, y, m, n, x_order, accumulate, *fmt, {t.device, t.host, ++t.ticket}, static_cast<cudaStream_t>(stream));
        return e == RPTC_OK ? wait_for(t, static_cast<cudaStream_t>(stream), ms) : e;
    }
    if (int e = rptc_timer_begin(stream)) return e;
    if (int e = rptc_gemv(codes, lut, nullptr, x, n, acc, m, m, n, 1, x_order, fmt, stream)) return e;
    {
        // the finish behind the product may start early: it waits for the product's sums itself
        const bool before = pdl_enabled();
        rptc_set_pdl(1);
        const int e = rptc_gemv_finish(acc, m, y, m, m, 1, 1.f, accumulate, 1, stream);
        rptc_set_pdl(before ? 1 : 0);
        if (e) return e;
    }
    return rptc_timer_end(ms, stream);
}
