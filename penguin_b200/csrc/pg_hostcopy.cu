// Device planes to pageable host arrays (the state readers of every kind of disk).
//
// cudaMemcpyAsync to pageable memory goes through the driver's own staging on the calling
// thread, which also takes the page faults of a fresh array.  Large reads are cut into chunks
// that COPY_THREADS threads take in turn, each through two pinned slots of its own: while one
// slot fills from the device the other is copied out.  100 FP32 steps of 1024x3072 and the
// read of its state: 50.5 ms through the driver, 36.8 so.  Slots of 1 MB read 4 % faster and
// cost the first read 4 ms.
#include <cstring>
#include <system_error>
#include <thread>

#include "pg_internal.h"

namespace pg {

constexpr size_t COPY_CHUNK = HostCopy::SLOT;     // doubles: 256 KB
constexpr size_t COPY_DIRECT = (size_t)1 << 20;   // doubles: smaller reads take the driver's path

namespace {

// the chunks w, w + COPY_THREADS, ... of the read
cudaError_t copy_share(HostCopy& h, int w, int device, const double* src, double* const* dst, int planes, size_t count,
                       cudaStream_t s) {
    cudaError_t e = cudaSetDevice(device);
    const size_t per = (count + COPY_CHUNK - 1) / COPY_CHUNK, total = per * planes;
    double* out[2] = {nullptr, nullptr};
    size_t len[2] = {0, 0};
    int slot = 0;
    for (size_t k = w; e == cudaSuccess; k += COPY_THREADS, slot ^= 1) {
        const bool more = k < total;
        if (more) {
            const size_t at = (k % per) * COPY_CHUNK;
            len[slot] = count - at < COPY_CHUNK ? count - at : COPY_CHUNK;
            out[slot] = dst[k / per] + at;
            e = cudaMemcpyAsync(h.slot(w, slot), src + (k / per) * count + at, len[slot] * sizeof(double),
                                cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaEventRecord(h.ev[w][slot], s);
        }
        const int prev = slot ^ 1;
        if (out[prev]) {
            const cudaError_t r = cudaEventSynchronize(h.ev[w][prev]);
            if (r != cudaSuccess) return r;
            std::memcpy(out[prev], h.slot(w, prev), len[prev] * sizeof(double));
            out[prev] = nullptr;
        }
        if (!more) break;
    }
    return e;
}

}  // namespace

HostCopy::~HostCopy() {
    for (auto& t : ev)
        for (auto& x : t)
            if (x) cudaEventDestroy(x);
    if (pinned) cudaFreeHost(pinned);
}

cudaError_t copy_planes_out(HostCopy& h, int device, const double* src, double* const* dst, int planes, size_t count,
                            cudaStream_t s) {
    // a per-thread stream is another one in every thread; arrays that overlap are written in the planes' order
    bool staged = count * planes >= COPY_DIRECT && s != cudaStreamPerThread;
    for (int f = 0; f < planes; ++f)
        for (int g = 0; g < f; ++g) staged = staged && !(dst[f] < dst[g] + count && dst[g] < dst[f] + count);
    for (int f = 0; f < planes && staged; ++f) {  // page-locked and managed arrays are copied to directly
        cudaPointerAttributes at{};
        staged = cudaPointerGetAttributes(&at, dst[f]) == cudaSuccess && at.type == cudaMemoryTypeUnregistered;
    }
    if (staged && !h.pinned) {
        void* p = nullptr;
        if (cudaMallocHost(&p, 2 * COPY_THREADS * COPY_CHUNK * sizeof(double)) == cudaSuccess) {
            bool ok = true;
            for (auto& t : h.ev)
                for (auto& x : t)
                    if (!x) ok = ok && cudaEventCreateWithFlags(&x, cudaEventDisableTiming) == cudaSuccess;
            if (ok) h.pinned = (double*)p;
            else cudaFreeHost(p);
        }
        if (!h.pinned) cudaGetLastError();  // no room to pin: the driver's path
    }
    if (!staged || !h.pinned) {
        for (int f = 0; f < planes; ++f) {
            const cudaError_t e =
                cudaMemcpyAsync(dst[f], src + f * count, count * sizeof(double), cudaMemcpyDeviceToHost, s);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    cudaError_t err[COPY_THREADS];
    std::thread th[COPY_THREADS];
    for (int w = 1; w < COPY_THREADS; ++w) {
        try {
            th[w] = std::thread([&, w] { err[w] = copy_share(h, w, device, src, dst, planes, count, s); });
        } catch (const std::system_error&) {  // no thread to be had: this one does the share below
        }
    }
    err[0] = copy_share(h, 0, device, src, dst, planes, count, s);
    for (int w = 1; w < COPY_THREADS; ++w) {
        if (th[w].joinable()) th[w].join();
        else err[w] = copy_share(h, w, device, src, dst, planes, count, s);
    }
    for (const cudaError_t e : err)
        if (e != cudaSuccess) return e;
    return cudaSuccess;
}

}  // namespace pg
