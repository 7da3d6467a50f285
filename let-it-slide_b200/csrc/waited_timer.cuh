// How a thread waits for a kernel and learns its device time without events: the memory that kernel and thread share.  Plain C++ but for
// the kernel's side, so that the host's can be compiled and run without a GPU.
#pragma once
#include <cuda_runtime_api.h>

namespace rptc {

// The device time of a kernel, left in host memory by the last of its CTAs together with `ticket`, which tells the waiting thread that
// the kernel's results are there.
struct DeviceTime {
    unsigned long long begin;            // earliest start; all ones between kernels
    unsigned int ended;                  // CTAs that have; 0 between kernels
};
struct HostTime {
    unsigned long long ns;
    unsigned int ticket;
    DeviceTime idle;                     // what DeviceTime is set up from
};
struct DeviceTimer {
    DeviceTime *device;
    HostTime *host;                      // pinned, as the device sees it
    unsigned int ticket;
#ifdef __CUDACC__
    static __device__ __forceinline__ unsigned long long now() {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)::"memory");
        return t;
    }
    __device__ __forceinline__ void begin() const { atomicMin(&device->begin, now()); }
    // by one thread of each of `ctas` CTAs, behind a barrier behind its last result
    __device__ __forceinline__ void end(unsigned int ctas) const {
        __threadfence();
        if (atomicAdd(&device->ended, 1u) + 1u != ctas) return;
        __threadfence();
        const unsigned long long from = atomicExch(&device->begin, ~0ull);
        device->ended = 0u;
        const unsigned long long to = now();      // another SM's reading than `from`
        *reinterpret_cast<volatile unsigned long long *>(&host->ns) = to > from ? to - from : 0ull;
        __threadfence_system();
        *reinterpret_cast<volatile unsigned int *>(&host->ticket) = ticket;
    }
#endif
};

// While a thread captures a graph in the default mode, calls that allocate or wait are refused to every thread, and spoil the capture
// (cudaMalloc, cudaEventSynchronize and cudaStreamQuery do).  Those here touch no captured stream, which this tells the runtime.
class BesideCaptures {
public:
    BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    ~BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    BesideCaptures(const BesideCaptures &) = delete;

private:
    cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;      // the thread's own meanwhile
};

// A thread's timer on a device; kept, and given back when the thread ends.
struct WaitedTimer {
    HostTime *host = nullptr;
    DeviceTime *device = nullptr;
    unsigned int ticket = 0;
    ~WaitedTimer() { release(); }
    void release() {
        if (!device) return;
        BesideCaptures mode;
        cudaFree(device);                  // waits for a kernel that may still write
        cudaFreeHost(host);
        device = nullptr, host = nullptr;
    }
    // All of it or nothing: a timer that could not be set up is set up by the next call.
    cudaError_t ready() {
        if (device) return cudaSuccess;
        BesideCaptures mode;
        HostTime *h = nullptr;
        DeviceTime *d = nullptr;
        cudaStream_t s = nullptr;
        cudaError_t e = cudaHostAlloc(reinterpret_cast<void **>(&h), sizeof(HostTime), cudaHostAllocMapped);
        if (e == cudaSuccess) {
            *h = {0, ticket, {~0ull, 0u}};
            e = cudaMalloc(reinterpret_cast<void **>(&d), sizeof(DeviceTime));
        }
        // on a stream of its own: the legacy one waits for others
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaMemcpyAsync(d, &h->idle, sizeof(DeviceTime), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (s) cudaStreamDestroy(s);
        if (e == cudaSuccess) {
            host = h, device = d;
            return e;
        }
        if (d) cudaFree(d);
        if (h) cudaFreeHost(h);
        return e;
    }
};

}  // namespace rptc
