// Staged copies between pageable host memory and device memory (host_copy.h).
//
// The ring holds kSlots chunks of kChunk bytes of pinned memory.  Chunk j of
// a copy uses slot j % kSlots.  A read-back (device to host): the calling
// thread queues the DMA of chunk j into its slot once every worker has
// emptied the slot's previous chunk, records the slot's event and posts j;
// each worker waits for the post and the event, then copies its stripe of
// the chunk to the destination.  An upload (host to device) runs the other
// way round: the workers fill a slot once the DMA of its previous chunk has
// completed (its event), and the calling thread queues the chunk's DMA when
// every worker has filled its stripe.  A failed CUDA call on any thread
// stops all of them; the error is raised on the calling thread after the
// workers have joined.
#include "host_copy.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "common.h"

namespace orr {
namespace {

constexpr std::size_t kChunk = std::size_t(4) << 20;
constexpr int kSlots = 8;
constexpr int kMaxWorkers = 16;
constexpr std::size_t kAloneBytes = std::size_t(2) << 20;
constexpr std::size_t kThreadBytes = std::size_t(512) << 10;

// One staged copy at a time in the process: the ring is shared.  It is
// allocated on first use (portable, so every device's DMA can use it) and
// kept for the life of the process.
std::mutex g_ring_lock;
unsigned char* g_ring = nullptr;

unsigned char* ring() {
    if (g_ring == nullptr) {
        void* p = nullptr;
        check(cudaHostAlloc(&p, kChunk * kSlots, cudaHostAllocPortable), "pinned staging buffer");
        g_ring = static_cast<unsigned char*>(p);
    }
    return g_ring;
}

// A read-back writes the caller's arrays, usually fresh ones whose pages
// fault in on first touch: it takes a thread per core.  An upload reads
// pages that exist already; half the cores keep up with the bus.
int worker_count(bool upload) {
    const unsigned n = std::thread::hardware_concurrency();
    return static_cast<int>(std::clamp<unsigned>(upload ? n / 2 : n, 1, kMaxWorkers));
}

struct Events {
    cudaEvent_t e[kSlots] = {};
    Events() {
        for (auto& x : e) {
            check(cudaEventCreateWithFlags(&x, cudaEventDisableTiming), "staging event");
        }
    }
    ~Events() {
        for (auto x : e) {
            if (x) cudaEventDestroy(x);
        }
    }
};

// Progress shared by the calling thread and the workers.
struct Progress {
    std::mutex m;
    std::condition_variable cv;
    std::size_t posted = 0;      // chunks whose DMA is queued and event recorded
    std::vector<int> filled;     // per chunk: workers done with their stripe
    bool stop = false;
    cudaError_t error = cudaSuccess;
    const char* what = nullptr;

    void fail(cudaError_t e, const char* text) {
        std::lock_guard<std::mutex> g(m);
        if (error == cudaSuccess) {
            error = e;
            what = text;
        }
        stop = true;
        cv.notify_all();
    }
    // Waits until `ready()` holds or the copy stopped; true when ready.
    template <class F> bool wait(F&& ready) {
        std::unique_lock<std::mutex> g(m);
        cv.wait(g, [&] { return stop || ready(); });
        return !stop;
    }
    void mark_filled(std::size_t j) {
        std::lock_guard<std::mutex> g(m);
        ++filled[j];
        cv.notify_all();
    }
    void post(std::size_t j) {
        std::lock_guard<std::mutex> g(m);
        posted = j + 1;
        cv.notify_all();
    }
};

// Stripe [a, b) of a chunk of `len` bytes for worker t of n (64-byte aligned
// boundaries, so workers never share a cache line).
void stripe(std::size_t len, int t, int n, std::size_t& a, std::size_t& b) {
    const std::size_t part = ((len + n - 1) / n + 63) & ~std::size_t(63);
    a = std::min(len, part * t);
    b = std::min(len, a + part);
}

// Chunk j of a copy: `len` bytes at `device` and at `host` (2 * len there
// for a widening chunk).
struct Chunk {
    unsigned char* host;
    unsigned char* device;
    std::size_t len;
    bool widen = false;
    double add = 0.0;
};

// Binary32 values [a, b) (byte offsets) of a staged chunk to the host as
// binary64 plus `add`.
void widen_stripe(const Chunk& c, const unsigned char* from, std::size_t a, std::size_t b) {
    const auto* src = reinterpret_cast<const float*>(from + a);
    auto* dst = reinterpret_cast<double*>(c.host + 2 * a);
    const std::size_t n = (b - a) / sizeof(float);
    for (std::size_t k = 0; k < n; ++k) {
        dst[k] = static_cast<double>(src[k]) + c.add;
    }
}

// A read-back's threads start while the stream's earlier work runs; the ring is
// taken once that work is done, so that a solver in the middle of a long run
// does not keep it from the others'.
void staged(bool upload, const std::vector<Chunk>& chunks, cudaStream_t stream, int device) {
    std::unique_lock<std::mutex> hold(g_ring_lock, std::defer_lock);
    unsigned char* slots = nullptr;
    const auto take_ring = [&] {
        check(cudaStreamSynchronize(stream), "staged copy");
        hold.lock();
        slots = ring();
    };
    if (upload) {
        take_ring();   // the threads fill it from their start
    }
    Events ev;
    const std::size_t n = chunks.size();
    // One thread moves the fields at 10 GB/s in some processes and at 4 in others (the
    // cause is not known), and threads take 100 us and more to start after a run: this
    // thread up to kAloneBytes of host memory, then one for each kThreadBytes, up to
    // worker_count (so only widening read-backs below 8 MiB take fewer).  us per
    // read-back of the fields after 200 steps with one thread (the two kinds of
    // process), one per 0.5 MiB, and sixteen: 48 x 24 x 24 (0.8 MiB) 95 to 240, 180, 485;
    // 64 x 32 x 32 (2 MiB) 190 to 515, 350, 495; 72 x 36 x 36 250 to 710, 380 to 410, 540;
    // 80 x 40 x 40 (3.9 MiB) 315 to 960, 420 to 515, 595.
    std::size_t host_bytes = 0;
    for (const Chunk& c : chunks) {
        host_bytes += c.widen ? 2 * c.len : c.len;
    }
    const std::size_t wanted = host_bytes <= kAloneBytes ? 1 : (host_bytes + kThreadBytes - 1) / kThreadBytes;
    const int nworkers = static_cast<int>(std::min<std::size_t>(wanted, worker_count(upload)));
    Progress pr;
    pr.filled.assign(n, 0);
    const auto slot = [&](std::size_t j) { return slots + (j % kSlots) * kChunk; };

    // Waits for chunk j of a read-back and copies stripe t of it out of its slot.
    const auto take_out = [&](std::size_t j, int t) {
        if (!pr.wait([&] { return pr.posted > j; })) {
            return false;
        }
        const cudaError_t s = cudaEventSynchronize(ev.e[j % kSlots]);
        if (s != cudaSuccess) {
            pr.fail(s, "staged read-back");
            return false;
        }
        std::size_t a = 0, b = 0;
        stripe(chunks[j].len, t, nworkers, a, b);
        if (chunks[j].widen) {
            widen_stripe(chunks[j], slot(j), a, b);
        } else {
            std::memcpy(chunks[j].host + a, slot(j) + a, b - a);
        }
        return true;
    };
    // Of a read-back whose chunks all fit the ring, this thread is a worker too
    // once it has queued them, and each takes the next stripe that nobody has: the
    // copy does not wait for a thread that starts late.
    const bool shared = !upload && n <= static_cast<std::size_t>(kSlots);
    std::atomic<std::size_t> next{0};

    auto worker = [&](int t) {
        const cudaError_t e = cudaSetDevice(device);
        if (e != cudaSuccess) {
            pr.fail(e, "cudaSetDevice");
            return;
        }
        if (shared) {
            for (std::size_t k = next++; k < n * static_cast<std::size_t>(nworkers); k = next++) {
                if (!take_out(k / nworkers, static_cast<int>(k % nworkers))) {
                    return;
                }
            }
            return;
        }
        for (std::size_t j = 0; j < n; ++j) {
            if (upload) {
                std::size_t a = 0, b = 0;
                stripe(chunks[j].len, t, nworkers, a, b);
                // The slot is free once the DMA of chunk j - kSlots is done.
                if (j >= static_cast<std::size_t>(kSlots)) {
                    if (!pr.wait([&] { return pr.posted > j - kSlots; })) {
                        return;
                    }
                    const cudaError_t s = cudaEventSynchronize(ev.e[j % kSlots]);
                    if (s != cudaSuccess) {
                        pr.fail(s, "staged upload");
                        return;
                    }
                }
                std::memcpy(slot(j) + a, chunks[j].host + a, b - a);
            } else if (!take_out(j, t)) {
                return;
            }
            pr.mark_filled(j);
        }
    };

    std::vector<std::thread> threads;
    threads.reserve(nworkers);
    try {
        for (int t = shared ? 1 : 0; t < nworkers; ++t) {
            threads.emplace_back(worker, t);
        }
        if (!upload) {
            take_ring();
        }
    } catch (...) {
        pr.fail(cudaErrorUnknown, "staging threads");
        for (auto& th : threads) th.join();
        throw;
    }
    for (std::size_t j = 0; j < n; ++j) {
        if (upload) {
            if (!pr.wait([&] { return pr.filled[j] == nworkers; })) {
                break;
            }
        } else if (j >= static_cast<std::size_t>(kSlots)) {
            if (!pr.wait([&] { return pr.filled[j - kSlots] == nworkers; })) {
                break;
            }
        }
        const Chunk& c = chunks[j];
        cudaError_t e = upload ? cudaMemcpyAsync(c.device, slot(j), c.len, cudaMemcpyHostToDevice, stream)
                               : cudaMemcpyAsync(slot(j), c.device, c.len, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) {
            e = cudaEventRecord(ev.e[j % kSlots], stream);
        }
        if (e != cudaSuccess) {
            pr.fail(e, upload ? "staged upload" : "staged read-back");
            break;
        }
        pr.post(j);
    }
    if (shared) {
        worker(0);
    }
    for (auto& th : threads) th.join();
    if (pr.error == cudaSuccess && upload && n > 0) {
        // The DMAs run in stream order: the last one's event covers them all.
        const cudaError_t e = cudaEventSynchronize(ev.e[(n - 1) % kSlots]);
        if (e != cudaSuccess) {
            pr.fail(e, "staged upload");
        }
    }
    if (pr.error != cudaSuccess) {
        // Nothing may still read or write the ring when it is released.
        cudaStreamSynchronize(stream);
        throw CudaError{pr.error, pr.what};
    }
}

void copy(bool upload, const HostSpan* spans, int count, cudaStream_t stream, int device) {
    std::size_t total = 0;
    bool widen = false;
    for (int k = 0; k < count; ++k) {
        total += spans[k].bytes;
        if (spans[k].widen) {
            if (upload || spans[k].bytes % sizeof(float) != 0) {
                throw CudaError{cudaErrorInvalidValue, "widening copy (read-backs of binary32 values only)"};
            }
            widen = true;
        }
    }
    // Widening spans always take the ring: the host threads do the widening.
    if (total < kStagedCopyBytes && !widen) {
        const char* what = upload ? "upload" : "read-back";
        for (int k = 0; k < count; ++k) {
            const HostSpan& s = spans[k];
            if (s.bytes > 0) {
                check(upload ? cudaMemcpyAsync(s.device, s.host, s.bytes, cudaMemcpyHostToDevice, stream)
                             : cudaMemcpyAsync(s.host, s.device, s.bytes, cudaMemcpyDeviceToHost, stream),
                      what);
            }
        }
        check(cudaStreamSynchronize(stream), what);
        return;
    }
    std::vector<Chunk> chunks;
    chunks.reserve(total / kChunk + count);
    for (int k = 0; k < count; ++k) {
        auto* h = static_cast<unsigned char*>(spans[k].host);
        auto* d = static_cast<unsigned char*>(spans[k].device);
        const std::size_t scale = spans[k].widen ? 2 : 1;
        for (std::size_t off = 0; off < spans[k].bytes; off += kChunk) {
            chunks.push_back(Chunk{h + scale * off, d + off, std::min(kChunk, spans[k].bytes - off), spans[k].widen,
                                   spans[k].add});
        }
    }
    staged(upload, chunks, stream, device);
}

} // namespace

void copy_to_device(const HostSpan* spans, int count, cudaStream_t stream, int device) {
    copy(true, spans, count, stream, device);
}

void copy_to_host(const HostSpan* spans, int count, cudaStream_t stream, int device) {
    copy(false, spans, count, stream, device);
}

} // namespace orr
