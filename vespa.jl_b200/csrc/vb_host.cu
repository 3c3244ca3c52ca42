// vb_host.cu -- large pageable host arrays.
//
// A copy from or to pageable memory is staged by the driver on one core, 10 to
// 15 GB/s, and a fresh array's page faults fall on that core too.  Here a few
// threads ("lanes"), each with its own stream, move pieces of about a megabyte
// through pinned buffers of their own, so that the host copies of different
// pieces run on different cores and overlap the transfers (and, for face
// batches, the kernels).  200 k faces (17 MB in, 8 MB out): 1.59 -> 1.17 ms with
// arrays new to every call, 0.9 ms with the same ones again; the PCIe link alone
// takes 0.35 ms.  Smaller copies, where the threads would cost more than
// they give, and copies of pinned arrays stay plain.
//
// The lanes belong to their context, which one host thread uses at a time, are
// made once its large copies and face batches add up to LANES_FROM (16 MB pinned,
// 16 MB device) and freed with it.
#include <cstdint>
#include <cstring>
#include <new>
#include <thread>

#include "vb_internal.h"

using vb::detail::fail;

namespace {

constexpr int LANES = 8;
constexpr int64_t FACES = 8192;             // faces of a piece: 84 B each in, 40 B out
constexpr size_t FACES_IN = (size_t)FACES * 84;
constexpr size_t FACE_BYTES = 124;
constexpr size_t PIECE = (size_t)FACES * FACE_BYTES;
constexpr size_t COPY_MIN = 4u << 20;
// the lanes are made once this much has gone plainly: making them (16 MB to
// page-lock, 8 streams) takes 12 ms, which short runs never earn back.  Face
// batches gain about 1 ms per 25 MB, so they do after some 300 MB.
constexpr size_t LANES_FROM = 256u << 20;

struct Lane {
    char *pin = nullptr, *dev = nullptr;  // pinned: two pieces; device: a piece of faces
    cudaStream_t s = nullptr;
    cudaEvent_t done[2] = {};
};

}  // namespace

struct vb_host_lanes {
    Lane lane[LANES];
    cudaEvent_t start = nullptr;
};

void vb::detail::host_lanes_free(vb_host_lanes *hl)
{
    if (!hl) return;
    for (Lane &l : hl->lane) {
        if (l.s) cudaStreamSynchronize(l.s);
        cudaFreeHost(l.pin);
        cudaFree(l.dev);
        for (cudaEvent_t e : l.done)
            if (e) cudaEventDestroy(e);
        if (l.s) cudaStreamDestroy(l.s);
    }
    if (hl->start) cudaEventDestroy(hl->start);
    delete hl;
}

namespace {

// Whether `bytes` more of large arrays find the lanes there, made now if they
// add up to enough.  When they cannot be (no
// page-locked or device memory left) the caller's arrays go plainly, and the
// next try comes when they add up anew.
bool make_lanes(vb_ctx *ctx, size_t bytes)
{
    if (ctx->lanes) return true;
    ctx->copied += bytes;
    if (ctx->copied < LANES_FROM) return false;
    vb_host_lanes *hl = new (std::nothrow) vb_host_lanes;
    if (!hl) return false;
    cudaError_t e = cudaEventCreateWithFlags(&hl->start, cudaEventDisableTiming);
    for (Lane &l : hl->lane) {
        if (e == cudaSuccess) e = cudaMallocHost(&l.pin, 2 * PIECE);
        if (e == cudaSuccess) e = cudaMalloc(&l.dev, 2 * PIECE);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&l.s, cudaStreamNonBlocking);
        for (cudaEvent_t &ev : l.done)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    }
    if (e != cudaSuccess) {
        vb::detail::host_lanes_free(hl);
        cudaGetLastError();
        ctx->copied = 0;
        return false;
    }
    ctx->lanes = hl;
    return true;
}

// work(lane, index, count) on min(lanes, pieces) threads, this one among them,
// each lane's stream ordered after the context's; the first error
template <typename F>
int run_lanes(vb_ctx *ctx, int64_t pieces, F &&work, const char *what)
{
    vb_host_lanes *hl = ctx->lanes;
    int n = (int)std::thread::hardware_concurrency() / 2;
    n = n < 1 ? 1 : n > LANES ? LANES : n;
    if (n > pieces) n = (int)pieces;
    VB_CUDA(cudaEventRecord(hl->start, ctx->stream));
    for (int i = 0; i < n; ++i) VB_CUDA(cudaStreamWaitEvent(hl->lane[i].s, hl->start, 0));
    cudaError_t err[LANES] = {};
    std::thread th[LANES];
    auto lane = [&](int i) {
        cudaError_t e = cudaSetDevice(ctx->device);
        if (e == cudaSuccess) e = work(hl->lane[i], i, n);
        if (e != cudaSuccess) cudaStreamSynchronize(hl->lane[i].s);
        err[i] = e;
    };
    int started = 1;
    try {
        for (; started < n; ++started) th[started] = std::thread(lane, started);
    } catch (...) {  // no more threads: this one takes the lanes left
    }
    lane(0);
    for (int i = started; i < n; ++i) lane(i);
    for (int i = 1; i < started; ++i) th[i].join();
    for (int i = 0; i < n; ++i)
        if (err[i] != cudaSuccess)
            return fail(VB_ECUDA, std::string(what) + ": " + cudaGetErrorString(err[i]));
    return VB_OK;
}

// plain pageable memory: not page-locked, managed or on a device
bool pageable(const void *p)
{
    cudaPointerAttributes at{};
    const bool known = cudaPointerGetAttributes(&at, p) == cudaSuccess;
    cudaGetLastError();
    return known && at.type == cudaMemoryTypeUnregistered;
}

}  // namespace

int vb::detail::host_copy(vb_ctx *ctx, void *dst, const void *src, size_t bytes, bool to_device)
{
    if (bytes < COPY_MIN || !pageable(to_device ? src : dst) || !make_lanes(ctx, bytes)) {
        VB_CUDA(cudaMemcpyAsync(dst, src, bytes, to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost,
                                ctx->stream));
        VB_CUDA(cudaStreamSynchronize(ctx->stream));
        return VB_OK;
    }
    const int64_t pieces = (int64_t)((bytes + PIECE - 1) / PIECE);
    auto work = [&](Lane &l, int i, int n) {
        cudaError_t e = cudaSuccess;
        int64_t held[2] = {-1, -1};  // the piece in flight in each half
        auto size = [&](int64_t p) { return bytes - (size_t)p * PIECE < PIECE ? bytes - (size_t)p * PIECE : PIECE; };
        auto finish = [&](int h) {
            if (held[h] < 0) return;
            const cudaError_t r = cudaEventSynchronize(l.done[h]);
            if (e == cudaSuccess) e = r;
            if (e == cudaSuccess && !to_device)
                std::memcpy((char *)dst + (size_t)held[h] * PIECE, l.pin + h * PIECE, size(held[h]));
            held[h] = -1;
        };
        int h = 0;
        for (int64_t p = i; p < pieces && e == cudaSuccess; p += n, h ^= 1) {
            finish(h);
            if (e != cudaSuccess) break;
            char *pin = l.pin + h * PIECE;
            const size_t at_ = (size_t)p * PIECE, w = size(p);
            if (to_device) std::memcpy(pin, (const char *)src + at_, w);
            e = to_device ? cudaMemcpyAsync((char *)dst + at_, pin, w, cudaMemcpyHostToDevice, l.s)
                          : cudaMemcpyAsync(pin, (const char *)src + at_, w, cudaMemcpyDeviceToHost, l.s);
            if (e == cudaSuccess) e = cudaEventRecord(l.done[h], l.s);
            if (e == cudaSuccess) held[h] = p;
        }
        finish(h);
        finish(h ^ 1);
        return e;
    };
    return run_lanes(ctx, pieces, work, "host copy");
}

// Pinned arrays go as whole copies (200 k faces: 0.63 ms against 0.93 through
// the lanes, 40 k: 0.17 against 0.37), and so do batches whose fluxes overlap
// their states: a piece's fluxes land while later pieces' states are still read.
bool vb::detail::host_faces_staged(vb_ctx *ctx, int64_t nf, const double *WL, const double *WR,
                                   const double *F)
{
    auto apart = [&](const double *W) {
        const uintptr_t w = (uintptr_t)W, f = (uintptr_t)F, n = 5 * sizeof(double) * (uintptr_t)nf;
        return w + n <= f || f + n <= w;
    };
    return nf >= HOST_FACES && apart(WL) && apart(WR) && pageable(WL) && pageable(WR) && pageable(F) &&
           make_lanes(ctx, FACE_BYTES * (size_t)nf);
}

int vb::detail::host_faces(vb_ctx *ctx, int64_t nf, const double *WL, const double *WR,
                           const int32_t *axis, double gamma, double *F)
{
    const int64_t pieces = (nf + FACES - 1) / FACES;
    auto work = [&](Lane &l, int i, int n) {
        cudaError_t e = cudaSuccess;
        int64_t held[2] = {-1, -1};
        auto size = [&](int64_t p) { return nf - p * FACES < FACES ? nf - p * FACES : FACES; };
        auto finish = [&](int h) {
            if (held[h] < 0) return;
            const cudaError_t r = cudaEventSynchronize(l.done[h]);
            if (e == cudaSuccess) e = r;
            if (e == cudaSuccess)
                std::memcpy(F + 5 * held[h] * FACES, l.pin + h * PIECE + FACES_IN, 40 * (size_t)size(held[h]));
            held[h] = -1;
        };
        int h = 0;
        for (int64_t p = i; p < pieces && e == cudaSuccess; p += n, h ^= 1) {
            finish(h);
            if (e != cudaSuccess) break;
            char *pin = l.pin + h * PIECE, *dev = l.dev + h * PIECE;
            const int64_t f0 = p * FACES, m = size(p);
            const size_t w = 40 * (size_t)m;
            std::memcpy(pin, WL + 5 * f0, w);
            std::memcpy(pin + w, WR + 5 * f0, w);
            std::memcpy(pin + 2 * w, axis + f0, 4 * (size_t)m);
            e = cudaMemcpyAsync(dev, pin, 84 * (size_t)m, cudaMemcpyHostToDevice, l.s);
            if (e != cudaSuccess) break;
            vb::launch_hllc_faces(m, (const double *)dev, (const double *)(dev + w),
                                  (const int32_t *)(dev + 2 * w), gamma, (double *)(dev + FACES_IN), l.s);
            e = cudaGetLastError();
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(pin + FACES_IN, dev + FACES_IN, w, cudaMemcpyDeviceToHost, l.s);
            if (e == cudaSuccess) e = cudaEventRecord(l.done[h], l.s);
            if (e == cudaSuccess) held[h] = p;
        }
        finish(h);
        finish(h ^ 1);
        return e;
    };
    const int rc = run_lanes(ctx, pieces, work, "face batch");
    ctx->launches += pieces;
    return rc;
}
