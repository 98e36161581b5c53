// Host vectors to and from the device through two pinned buffers per handle.
//
// Callers pass ordinary (pageable) arrays, FP64 where the device works in FP32.  A copy from pageable memory runs
// through the CUDA driver's single-threaded staging, and converting on the device moves eight bytes per value over
// the bus and needs a device buffer.  Here host threads convert or copy chunk after chunk into (out of) one
// pinned buffer while the other one is on the bus, so the bus carries the device's own type and nothing is
// allocated per call.  An operator application on a 132 MB angular vector took 82 ms with pageable copies.
// Transfers up to 4 MB use a pair of 95 KB buffers that come with the handle; larger ones a pair of 512 KB that is allocated
// when first needed, and one of 4 MB once the handle has moved 128 MB through it.  Pinning costs 0.5 ms per MB, paid by the
// call that needs it, and so has to be small against that call: the first sweep of a handle on a vector of 31 MB (7.7 MB)
// took 11.4 (3.9) ms with pageable copies, 23 (10) with a pair of 8 MB, 6.2 (3.1) with 1 MB and 3.4 (1.6) with 512 KB.
// Later ones take 65.8 MB there and back in 7.0 ms with 512 KB and 5.2 with 4 MB (24.6 MB of results in 1.94 and 1.6).  The 4.4 ms
// that these cost come when the first 128 MB have saved as much against pageable copies (3.0 ms for the 24.6 MB).
// All go with the handle.  Only chunks of 256 KB up use several threads: waking them costs a small one more than it
// saves, and they are half the host's (at most 8), so that threads still spinning after a transfer leave the
// caller its core.
#include "lb_internal.h"
#include <algorithm>
#include <cstring>
#include <new>
#include <omp.h>

namespace lb {

namespace {

constexpr size_t kPipeLarge = (size_t)1 << 19;    // bytes of a large buffer at first
constexpr size_t kPipeMax = (size_t)4 << 20;      // and after kGrowAfter bytes
constexpr size_t kGrowAfter = (size_t)1 << 27;
constexpr size_t kLarge = (size_t)4 << 20;        // transfers above take the large buffers (and smaller ones once they exist)
constexpr size_t kHoldMax = (size_t)256 << 20;     // bytes of a vector on its way that a handle keeps the place of
constexpr size_t kThreaded = (size_t)1 << 18;     // bytes of a chunk from which several threads do the work

int threads_for(size_t bytes) { return bytes >= kThreaded ? std::max(1, std::min(8, omp_get_max_threads() / 2)) : 1; }

// The buffer pair for a transfer of `bytes` bytes; null after an error.
Handle::Pipe* pipe_for(Handle* h, size_t bytes) {
    const bool large = bytes > kLarge || (h->pipe_large.bytes && bytes > 2 * kPipeSmall);
    Handle::Pipe& p = large ? h->pipe_large : h->pipe_small;
    const size_t want = !large ? kPipeSmall : p.moved < kGrowAfter ? kPipeLarge : kPipeMax;
    p.moved += bytes;
    if (p.bytes >= want) return &p;
    void* buf[2] = {nullptr, nullptr};
    cudaError_t e = cudaSuccess;
    for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
        if (large) e = cudaMallocHost(&buf[b], want);
        else buf[b] = reinterpret_cast<char*>(h->h_red + kRedHost) + b * kPipeSmall;
    }
    if (e != cudaSuccess) {
        // no pinned memory: the pair there is, or the handle's own small one, in more chunks
        if (buf[0]) cudaFreeHost(buf[0]);
        cudaGetLastError();
        p.moved = 0;
        return p.bytes ? &p : pipe_for(h, 0);
    }
    for (int b = 0; b < 2 && e == cudaSuccess; ++b)
        e = p.ev[b] ? cudaEventSynchronize(p.ev[b]) : cudaEventCreateWithFlags(&p.ev[b], cudaEventDisableTiming);
    for (int b = 0; b < 2; ++b) {
        if (p.buf[b]) cudaFreeHost(p.buf[b]);   // (of a pair that grows: its last copies are done)
        p.buf[b] = buf[b];
    }
    p.bytes = want;
    if (e != cudaSuccess) {
        pipe_free(h);
        cuda_fail(h, e, "transfer buffers");
        return nullptr;
    }
    return &p;
}

void copy_bytes(void* dst, const void* src, size_t bytes) {
    const int nt = threads_for(bytes);
    const size_t part = nt > 1 ? (size_t)1 << 17 : bytes;
    const long long parts = (long long)((bytes + part - 1) / part);
#pragma omp parallel for schedule(static) num_threads(nt) if (nt > 1)
    for (long long p = 0; p < parts; ++p) {
        const size_t o = (size_t)p * part;
        std::memcpy((char*)dst + o, (const char*)src + o, std::min(part, bytes - o));
    }
}

void to_f32(float* dst, const double* src, size_t n) {
    const int nt = threads_for(n * sizeof(float));
#pragma omp parallel for schedule(static) num_threads(nt) if (nt > 1)
    for (size_t q = 0; q < n; ++q) dst[q] = (float)src[q];
}

void to_f64(double* dst, const float* src, size_t n, bool subtract) {
    const int nt = threads_for(n * sizeof(float));
    if (subtract) {
#pragma omp parallel for schedule(static) num_threads(nt) if (nt > 1)
        for (size_t q = 0; q < n; ++q) dst[q] = dst[q] - (double)src[q];
    } else {
#pragma omp parallel for schedule(static) num_threads(nt) if (nt > 1)
        for (size_t q = 0; q < n; ++q) dst[q] = (double)src[q];
    }
}

// fill(buffer, first, count): count elements of `elem` bytes from element `first` into the buffer
template <class F>
int up(Handle* h, void* dst, size_t n, size_t elem, const char* what, F&& fill) {
    if (n == 0) return LB_OK;
    Handle::Pipe* p = pipe_for(h, n * elem);
    if (!p) return LB_ERR_OOM;
    const size_t chunk = p->bytes / elem;
    for (size_t o = 0; o < n; o += chunk) {
        const size_t c = std::min(chunk, n - o);
        const int b = p->next;
        p->next ^= 1;
        cudaError_t e = cudaEventSynchronize(p->ev[b]);   // its last copy has read it
        if (e == cudaSuccess) {
            fill(p->buf[b], o, c);
            e = cudaMemcpyAsync((char*)dst + o * elem, p->buf[b], c * elem, cudaMemcpyHostToDevice, h->stream);
        }
        if (e == cudaSuccess) e = cudaEventRecord(p->ev[b], h->stream);
        if (e != cudaSuccess) return cuda_fail(h, e, what);
    }
    return LB_OK;
}

// drain(buffer, first, count): takes the elements out of the buffer; all are taken on return
template <class F>
int down(Handle* h, const void* src, size_t n, size_t elem, const char* what, F&& drain) {
    if (n == 0) return LB_OK;
    Handle::Pipe* p = pipe_for(h, n * elem);
    if (!p) return LB_ERR_OOM;
    const size_t chunk = p->bytes / elem;
    auto fetch = [&](size_t o, int b) {
        cudaError_t e = cudaMemcpyAsync(p->buf[b], (const char*)src + o * elem, std::min(chunk, n - o) * elem,
                                        cudaMemcpyDeviceToHost, h->stream);
        return e == cudaSuccess ? cudaEventRecord(p->ev[b], h->stream) : e;
    };
    // a buffer still being read by an upload is safe to fill: the copies are ordered by the stream
    cudaError_t e = fetch(0, 0);
    for (size_t o = 0, i = 0; o < n; o += chunk, ++i) {
        const int b = (int)(i & 1);
        if (e == cudaSuccess && o + chunk < n) e = fetch(o + chunk, b ^ 1);
        if (e == cudaSuccess) e = cudaEventSynchronize(p->ev[b]);
        if (e != cudaSuccess) return cuda_fail(h, e, what);
        drain(p->buf[b], o, std::min(chunk, n - o));
    }
    return LB_OK;
}

}  // namespace

void pipe_free(Handle* h) {
    for (int b = 0; b < 2; ++b) {
        if (h->pipe_large.buf[b]) cudaFreeHost(h->pipe_large.buf[b]);
        for (Handle::Pipe* p : {&h->pipe_small, &h->pipe_large})
            if (p->ev[b]) cudaEventDestroy(p->ev[b]);
    }
    h->pipe_small = Handle::Pipe{};
    h->pipe_large = Handle::Pipe{};
}

int pipe_up_f32(Handle* h, float* dst, const double* src, size_t n, const char* what) {
    return up(h, dst, n, sizeof(float), what, [&](void* b, size_t o, size_t c) { to_f32((float*)b, src + o, c); });
}

int pipe_down_f32(Handle* h, double* dst, const float* src, size_t n, bool subtract, const char* what) {
    auto drain = [&](const void* b, size_t o, size_t c) { to_f64(dst + o, (const float*)b, c, subtract); };
    if (!subtract || n * sizeof(float) <= kPipeSmall) return down(h, src, n, sizeof(float), what, drain);
    // what dst holds is an operand: it changes only when all of src is here, or a copy that fails half way would leave it
    // half changed.  (A vector that fits one buffer is drained when all of it has come.)  The handle keeps the place
    // up to 256 MB: page faults on a fresh one cost as much as the rest (65.8 MB: an operator application takes 11.4 ms
    // with a fresh place, 7.5 with a kept one, 6.0 if every chunk were subtracted as it comes).
    if (h->hold_cap < n) {
        h->hold_cap = 0;
        h->hold.reset(new (std::nothrow) float[n]);
        if (!h->hold) return fail(h, LB_ERR_OOM, std::string(what) + ": no host memory");
        h->hold_cap = n;
    }
    const int rc = pipe_down(h, h->hold.get(), src, n * sizeof(float), what);
    if (!rc) drain(h->hold.get(), 0, n);
    if (h->hold_cap * sizeof(float) > kHoldMax) {
        h->hold.reset();
        h->hold_cap = 0;
    }
    return rc;
}

int pipe_up(Handle* h, void* dst, const void* src, size_t bytes, const char* what) {
    return up(h, dst, bytes, 1, what, [&](void* b, size_t o, size_t c) { copy_bytes(b, (const char*)src + o, c); });
}

int pipe_down(Handle* h, void* dst, const void* src, size_t bytes, const char* what) {
    return down(h, src, bytes, 1, what, [&](const void* b, size_t o, size_t c) { copy_bytes((char*)dst + o, b, c); });
}

int pipe_up_rows(Handle* h, void* dst, size_t rows, size_t row_bytes, const std::function<void(void*, size_t)>& row,
                 const char* what) {
    return up(h, dst, rows, row_bytes, what, [&](void* b, size_t o, size_t c) {
        const int nt = threads_for(c * row_bytes);
#pragma omp parallel for schedule(static) num_threads(nt) if (nt > 1)
        for (size_t q = 0; q < c; ++q) row((char*)b + q * row_bytes, o + q);
    });
}

}  // namespace lb
