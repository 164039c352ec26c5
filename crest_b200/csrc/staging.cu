// Large copies between pageable host memory and the device.
//
// The runtime copies pageable memory through its own staging buffer with one
// host thread: 4 GB/s into freshly allocated arrays (every page is faulted in
// on the way), about 10 GB/s out of warm ones, against 55 GB/s for the link.
// Here a few threads of the call move pieces through two pinned buffers each,
// a piece's transfer overlapping the memory copies of the next one and of the
// other threads, so the page faults and the copying spread over cores (98 MB of
// a chunk's entries: 3.4 ms instead of 9.5; 40 MB of scores into a new array:
// 2.6 to 4 ms instead of 8.8).  Threads live for the call only (nothing to hand
// over a fork).  The first large copy on a device takes 12 MB of pinned buffers
// and the process keeps them, like the per-chunk workspaces: pinning them takes
// 10 to 15 ms and giving them back 1.5, which a program that opens, reduces and
// frees one matrix after another would otherwise pay for each.  A call that
// finds the buffers in use by another thread, or cannot have them, copies as
// before.
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <unistd.h>

#include <atomic>
#include <mutex>
#include <thread>
#include <vector>

#include "host.cuh"

namespace crest {
namespace {

constexpr size_t kPiece = 1u << 20;     // 256 kB: the driver calls cost as much as the copies; 2 MB: no gain
// Sizes from which the threads save more than they cost.  They find cold cores,
// so a copy of a few MB takes 0.15 to 0.5 ms (both sides warm), where the plain
// one takes 0.07 ms per MB (less when the caller has just written the data, as
// zeroed accumulators are); out into pages that are not there yet the plain one
// takes 0.45 ms per MB.  Plain against staged, in a Python process: two arrays
// in of 8 / 12 / 16 / 24 MB 1.17 / 1.59 / 2.05 / 3.13 ms (whole call) against
// 1.04 / 1.28 / 1.56 / 2.06, one of them zeroed just before 5 / 8 / 12 / 16 / 24
// MB 1.01 / 1.43 / 1.96 / 2.51 / 4.64 against 1.35 / 1.83 / 2.38 / 2.55 / 3.53;
// QC's two sums out into warm arrays of 2.3 / 4.6 / 9.2 MB 0.94 / 1.65 / 3.2 ms
// against 1.4 / 2.4 / 3.2, into new ones 3.5 / 6.8 / 13.6 against 2.6 / 4.3 /
// 6.5.  Sums added to the caller's (AddOut) go through the threads whatever the
// pages: group sums of three warm arrays of 3.2 / 5.4 / 6.4 / 10.7 MB 4.4 / 4.3 /
// 8.5 / 7.5 ms against 2.4 / 2.6 / 2.7 / 3.0.  An array that a call copies in and
// out again goes the same way both times (the threads leave its lines in other
// cores' caches, which a plain copy then fetches one by one): a chunk's Gram of 5.1
// / 8 / 13.5 MB that the caller keeps 1.0 / 1.38 / 2.13 ms (300 cells) and 2.17 /
// 2.55 / 3.31 (8,000) plain, 0.76 to 1.10 / 0.95 / 1.25 and 2.18 to 2.44 / 2.43
// to 2.61 / 2.84 to 3.01 staged; with one way by the threads alone slower than
// either.
constexpr size_t kStageIn = 16u << 20, kStageOutNew = 2u << 20, kStageOutWarm = 12u << 20,
                 kStageAdd = 2u << 20, kStageUpdated = 6u << 20;
constexpr int kStageThreads = 6;        // 4 to 12 within 5 %
constexpr int kSlots = 2 * kStageThreads;

struct Ring {
    std::mutex mu;
    unsigned char *buf = nullptr;
    cudaEvent_t ev[kSlots] = {};
    bool ready = false;
    bool ensure() {
        if (ready) return true;
        bool ok = cudaHostAlloc((void **)&buf, kSlots * kPiece, cudaHostAllocDefault) == cudaSuccess;
        for (int t = 0; ok && t < kSlots; ++t)
            ok = cudaEventCreateWithFlags(&ev[t], cudaEventDisableTiming) == cudaSuccess;
        if (!ok) {
            cudaGetLastError();
            release();
            return false;
        }
        return ready = true;
    }
    void release() {
        for (auto &e : ev) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        if (buf) cudaFreeHost(buf);
        buf = nullptr;
        ready = false;
    }
};

Ring g_ring[64];

bool pageable(const void *p) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

// Whether most pages of a host array of less than kStageOutWarm bytes exist
// (false when the system does not say).
bool mostly_there(const void *p, size_t bytes) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), a = (size_t)p / page * page;
    const size_t n = ((size_t)p + bytes - a + page - 1) / page;
    unsigned char there[kStageOutWarm / 4096 + 2];
    if (n > sizeof there || mincore(reinterpret_cast<void *>(a), n * page, there) != 0) return false;
    size_t have = 0;
    for (size_t i = 0; i < n; ++i) have += there[i] & 1;
    return 2 * have > n;
}

// body(t) for t < n on n threads, as many as can be had.
template <class F>
void on_threads(int n, F &&body) {
    std::vector<std::thread> th;
    int started = 1;
    try {
        th.reserve(n);
        for (; started < n; ++started) th.emplace_back(body, started);
    } catch (...) {  // no more threads: this one takes the rest
    }
    body(0);
    for (int t = started; t < n; ++t) body(t);
    for (auto &x : th) x.join();
}

// A thread's share of a copy: pieces first, first + step, ... of `bytes`, its
// two buffers and their events.
struct Share {
    size_t first, step, bytes;
    unsigned char *buf[2];
    cudaEvent_t ev[2];
    size_t count() const {
        const size_t pieces = (bytes + kPiece - 1) / kPiece;
        return first < pieces ? (pieces - first + step - 1) / step : 0;
    }
    size_t at(size_t i) const { return (first + i * step) * kPiece; }
    size_t size(size_t i) const { return std::min(kPiece, bytes - at(i)); }
};

// Runs work(share) on a few threads that cover `bytes`; false when the copy
// has to go the plain way.
template <class F>
bool in_pieces(const void *host, size_t bytes, cudaError_t &err, F &&work) {
    if (!pageable(host)) return false;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return false;
    }
    Ring &r = g_ring[dev];
    std::unique_lock<std::mutex> lock(r.mu, std::try_to_lock);
    if (!lock.owns_lock() || !r.ensure()) return false;
    const int cores = (int)std::max(2u, std::thread::hardware_concurrency());
    const int n = (int)std::min<size_t>((bytes + 2 * kPiece - 1) / (2 * kPiece), std::min(kStageThreads, cores / 2));
    std::atomic<int> bad{(int)cudaSuccess};
    on_threads(n, [&](int t) {
        const Share sh{(size_t)t, (size_t)n, bytes, {r.buf + 2 * t * kPiece, r.buf + (2 * t + 1) * kPiece},
                       {r.ev[2 * t], r.ev[2 * t + 1]}};
        cudaError_t e = cudaSetDevice(dev);
        if (e == cudaSuccess) e = work(sh);
        for (cudaEvent_t ev : sh.ev) {  // the buffers are free for the next call once their last transfers are over
            const cudaError_t w = cudaEventSynchronize(ev);
            if (e == cudaSuccess) e = w;
        }
        if (e != cudaSuccess) bad = (int)e;
    });
    err = (cudaError_t)bad.load();
    return true;
}

}  // namespace

int copy_in(void *dev, const void *host, size_t bytes, cudaStream_t st, bool updated) {
    cudaError_t err = cudaSuccess;
    const bool done = bytes >= (updated ? kStageUpdated : kStageIn) && in_pieces(host, bytes, err, [&](const Share &sh) {
        cudaError_t e = cudaSuccess;
        for (size_t i = 0; i < sh.count() && e == cudaSuccess; ++i) {
            e = cudaEventSynchronize(sh.ev[i & 1]);  // the buffer's transfer before
            if (e != cudaSuccess) break;
            memcpy(sh.buf[i & 1], static_cast<const unsigned char *>(host) + sh.at(i), sh.size(i));
            e = cudaMemcpyAsync(static_cast<unsigned char *>(dev) + sh.at(i), sh.buf[i & 1], sh.size(i),
                                cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(sh.ev[i & 1], st);
        }
        return e;
    });
    if (!done) err = cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
    CREST_CUDA_TRY(err);
    return CREST_OK;
}

namespace {
bool stage_out(const void *host, size_t bytes) {
    return bytes >= kStageOutNew && (bytes >= kStageOutWarm || !mostly_there(host, bytes));
}

// Device data through the buffers into sink(pointer, offset, bytes); false: not taken.
template <class F>
bool drain(const void *host, const void *dev, size_t bytes, cudaStream_t st, cudaError_t &err, F &&sink) {
    return in_pieces(host, bytes, err, [&](const Share &sh) {
        auto fetch = [&](size_t i) {
            cudaError_t e = cudaMemcpyAsync(sh.buf[i & 1], static_cast<const unsigned char *>(dev) + sh.at(i), sh.size(i),
                                            cudaMemcpyDeviceToHost, st);
            return e == cudaSuccess ? cudaEventRecord(sh.ev[i & 1], st) : e;
        };
        const size_t n = sh.count();
        cudaError_t e = n ? fetch(0) : cudaSuccess;
        for (size_t i = 0; i < n && e == cudaSuccess; ++i) {
            if (i + 1 < n) e = fetch(i + 1);
            if (e == cudaSuccess) e = cudaEventSynchronize(sh.ev[i & 1]);
            if (e == cudaSuccess) sink(sh.buf[i & 1], sh.at(i), sh.size(i));
        }
        return e;
    });
}
}  // namespace

int copy_out(void *host, const void *dev, size_t bytes, cudaStream_t st, bool updated) {
    cudaError_t err = cudaSuccess;
    const bool staged = (updated ? bytes >= kStageUpdated : stage_out(host, bytes)) &&
                        drain(host, dev, bytes, st, err, [&](const unsigned char *p, size_t at, size_t n) {
                            memcpy(static_cast<unsigned char *>(host) + at, p, n);
                        });
    if (!staged)
        err = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
    CREST_CUDA_TRY(err);
    return CREST_OK;
}

AddOut::AddOut(double *host, const void *dev, int64_t n, bool narrow)
    : host_(host), dev_(dev), n_(host && n > 0 ? n : 0), narrow_(narrow),
      stage_((narrow ? sizeof(uint32_t) : sizeof(double)) * (size_t)n_ >= kStageAdd) {
    if (!stage_) buf_.resize((narrow ? sizeof(uint32_t) : sizeof(double)) * (size_t)n_);
}

template <class T>
int AddOut::add_as(cudaStream_t st) {
    const size_t bytes = sizeof(T) * (size_t)n_;
    cudaError_t err = cudaSuccess;
    auto sum = [this](const T *v, size_t first, size_t n) {
        double *o = host_ + first;
        for (size_t i = 0; i < n; ++i) o[i] += (double)v[i];
    };
    if (stage_ && drain(host_, dev_, bytes, st, err, [&](const unsigned char *p, size_t at, size_t n) {
            sum(reinterpret_cast<const T *>(p), at / sizeof(T), n / sizeof(T));
        })) {
        CREST_CUDA_TRY(err);
        return CREST_OK;
    }
    buf_.resize(bytes);  // when the pinned buffers were not to be had
    CREST_CUDA_TRY(cudaMemcpyAsync(buf_.data(), dev_, bytes, cudaMemcpyDeviceToHost, st));
    CREST_CUDA_TRY(cudaStreamSynchronize(st));
    sum(reinterpret_cast<const T *>(buf_.data()), 0, (size_t)n_);
    return CREST_OK;
}

int AddOut::add(cudaStream_t st) {
    if (n_ == 0) return CREST_OK;
    return narrow_ ? add_as<uint32_t>(st) : add_as<double>(st);
}

}  // namespace crest
