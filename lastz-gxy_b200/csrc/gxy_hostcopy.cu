// gxy_hostcopy.cu -- copies between pageable host memory and the device.
//
// A copy of pageable memory goes through one staging buffer of the driver's, filled
// or emptied by one thread: 10 GB/s to the device, 7 from it into memory that is
// touched for the first time, where the link carries 50.  From 2 MB on the copy is
// cut into chunks that up to kCopyThreads threads (this one among them) take from a
// cursor; each has a stream and two pinned halves of its own, so that its chunk in
// one half crosses the link while it fills or empties the other, page faults
// included.  Chunks are taken 2 MB apart first: neighbours in one huge page would
// wait for one thread to clear it.  The arrays of 13.3 M bases (6.7 MB) into memory
// touched for the first time: 1.1 ms by the driver, 0.3 ms this way.
//
// The pinned memory (8 MB), streams, events and helper threads belong to the
// context, are made at its first such copy (or by host_copy_warm) and given back with it; a second copy at
// the same time takes the driver's path, as do smaller ones and memory that is
// pinned already.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>

#include "gxy_engine.cuh"

namespace gxy {

namespace {

constexpr size_t kChunk = 512u << 10;
constexpr size_t kStagedFrom = 2u << 20, kHugePage = 2u << 20;

cudaError_t prepare(HostCopy& h, int device) {
    if (h.pinned) return cudaSuccess;
    void* pinned = nullptr;
    cudaError_t e = cudaHostAlloc(&pinned, 2 * kCopyThreads * kChunk, cudaHostAllocPortable);
    // (A call that fails may leave anything in its handle: kept only when it succeeds.)
    if (e == cudaSuccess) h.pinned = static_cast<char*>(pinned);
    for (int i = 0; i < kCopyThreads && e == cudaSuccess; i++) {
        cudaStream_t st;
        e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        if (e == cudaSuccess) h.st[i] = st;
        for (int k = 0; k < 2 && e == cudaSuccess; k++) {
            cudaEvent_t ev;
            e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
            if (e == cudaSuccess) h.ev[i][k] = ev;
        }
    }
    if (e != cudaSuccess) {
        h.destroy();
        cudaGetLastError();
        return e;
    }
    const int want = (int)std::min<unsigned>(kCopyThreads, std::max(1u, std::thread::hardware_concurrency())) - 1;
    try {
        for (; h.n_helpers < want; h.n_helpers++) {
            const int me = h.n_helpers + 1;
            h.helper[h.n_helpers] = std::thread([&h, me, device] { h.help(me, device); });
        }
    } catch (...) {   // fewer helpers
    }
    return e;
}

bool pageable(const void* p) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

}  // namespace

void HostCopy::help(int me, int device) {
    cudaSetDevice(device);
    uint64_t done = 0;
    std::unique_lock<std::mutex> g(job_mu);
    for (;;) {
        cv.wait(g, [&] { return stop || generation != done; });
        if (stop) return;
        done = generation;
        if (me >= n_job) continue;
        const std::function<void(int)>* f = job;
        g.unlock();
        (*f)(me);
        g.lock();
        if (--running == 0) cv_done.notify_one();
    }
}

void HostCopy::run(const std::function<void(int)>& f, int threads) {
    {
        std::lock_guard<std::mutex> g(job_mu);
        job = &f;
        n_job = std::min(threads, n_helpers + 1);
        running = n_job - 1;
        generation++;
    }
    cv.notify_all();
    f(0);
    std::unique_lock<std::mutex> g(job_mu);
    cv_done.wait(g, [&] { return running == 0; });
    job = nullptr;
}

void HostCopy::destroy() {
    {
        std::lock_guard<std::mutex> g(job_mu);
        stop = true;
    }
    cv.notify_all();
    for (int i = 0; i < n_helpers; i++) helper[i].join();
    n_helpers = 0;
    stop = false;
    for (int i = 0; i < kCopyThreads; i++) {
        for (int k = 0; k < 2; k++) {
            if (ev[i][k]) cudaEventDestroy(ev[i][k]);
            ev[i][k] = nullptr;
        }
        if (st[i]) cudaStreamDestroy(st[i]);
        st[i] = nullptr;
    }
    if (pinned) cudaFreeHost(pinned);
    pinned = nullptr;
}

void host_copy_warm(gxy_ctx* ctx, uint64_t bytes) {
    if (bytes < kStagedFrom) return;
    std::lock_guard<std::mutex> hold(ctx->copy.mu);
    prepare(ctx->copy, ctx->device);   // (without it copies take the driver's path)
}

namespace {

struct Chunk {
    int piece;
    size_t at, bytes, turn;   // turn: its place in its huge page
};

// Through the pinned halves, by `threads` threads; the caller holds ctx->copy.mu.
cudaError_t staged_copy(gxy_ctx* ctx, const CopyPiece* pieces, const std::vector<Chunk>& chunks, int threads, bool to_host,
                        const std::function<void(size_t, size_t)>& seen) {
    std::atomic<size_t> next{0};
    std::atomic<int> failed{0};
    HostCopy& h = ctx->copy;
    auto copies = [&](int me) {
        char* half[2] = {h.pinned + 2 * me * kChunk, h.pinned + (2 * me + 1) * kChunk};
        char* dst[2] = {nullptr, nullptr};   // a half that waits to be emptied
        size_t len[2] = {0, 0};
        cudaError_t r = cudaSuccess;
        try {
            for (int k = 0; r == cudaSuccess && !failed.load(); k ^= 1) {
                const size_t c = next.fetch_add(1);
                const bool have = c < chunks.size();
                if (to_host) {
                    if (have) {
                        const CopyPiece& p = pieces[chunks[c].piece];
                        const size_t o = chunks[c].at;
                        len[k] = chunks[c].bytes;
                        dst[k] = static_cast<char*>(p.host) + o;
                        r = cudaMemcpyAsync(half[k], static_cast<const char*>(p.dev) + o, len[k], cudaMemcpyDeviceToHost, h.st[me]);
                        if (r == cudaSuccess) r = cudaEventRecord(h.ev[me][k], h.st[me]);
                    }
                    const int o = k ^ 1;
                    if (r == cudaSuccess && dst[o]) {
                        r = cudaEventSynchronize(h.ev[me][o]);
                        if (r == cudaSuccess) memcpy(dst[o], half[o], len[o]);
                        dst[o] = nullptr;
                    }
                    if (!have && !dst[k]) break;
                } else {
                    if (!have) break;
                    const CopyPiece& p = pieces[chunks[c].piece];
                    const size_t o = chunks[c].at, b = chunks[c].bytes;
                    if (len[k]) r = cudaEventSynchronize(h.ev[me][k]);
                    if (r != cudaSuccess) break;
                    memcpy(half[k], static_cast<const char*>(p.host) + o, b);
                    len[k] = b;
                    r = cudaMemcpyAsync(static_cast<char*>(p.dev) + o, half[k], b, cudaMemcpyHostToDevice, h.st[me]);
                    if (r == cudaSuccess) r = cudaEventRecord(h.ev[me][k], h.st[me]);
                    if (seen) seen(o, o + b);
                }
            }
        } catch (...) {
            r = cudaErrorMemoryAllocation;
        }
        const cudaError_t s = cudaStreamSynchronize(h.st[me]);   // the halves are free again
        if (r == cudaSuccess) r = s;
        if (r != cudaSuccess) {
            int none = 0;
            failed.compare_exchange_strong(none, (int)r);
        }
    };
    h.run(std::ref(copies), threads);   // (by reference: nothing is allocated)
    return (cudaError_t)failed.load();
}

}  // namespace

cudaError_t host_copy(gxy_ctx* ctx, const CopyPiece* pieces, int n, bool to_host, cudaStream_t st,
                      const std::function<void(size_t, size_t)>& seen) {
    size_t total = 0;
    for (int i = 0; i < n; i++) total += pieces[i].bytes;
    // (Only for copies of a size: asking what the memory and the host are takes 3 us.)
    std::unique_lock<std::mutex> hold(ctx->copy.mu, std::defer_lock);
    if (total >= kStagedFrom &&
        std::all_of(pieces, pieces + n, [](const CopyPiece& p) { return !p.bytes || pageable(p.host); })) {
        const int threads = (int)std::min<size_t>({(size_t)kCopyThreads, std::max<size_t>(1, std::thread::hardware_concurrency()),
                                                   total >> 19});
        if (threads >= 2 && hold.try_lock() && prepare(ctx->copy, ctx->device) == cudaSuccess) {
            std::vector<Chunk> chunks;
            try {
                for (int i = 0; i < n; i++) {
                    const size_t into = reinterpret_cast<uintptr_t>(pieces[i].host) % kHugePage;
                    for (size_t o = 0; o < pieces[i].bytes;) {
                        const size_t b = std::min(kChunk - (into + o) % kChunk, pieces[i].bytes - o);
                        chunks.push_back({i, o, b, (into + o) % kHugePage / kChunk});
                        o += b;
                    }
                }
                std::stable_sort(chunks.begin(), chunks.end(), [](const Chunk& x, const Chunk& y) { return x.turn < y.turn; });
            } catch (const std::bad_alloc&) {   // the driver's path needs nothing of the host
                chunks.clear();
            }
            if (!chunks.empty()) {
                // What st holds (the allocation, what fills it) comes first.
                const cudaError_t e = cudaStreamSynchronize(st);
                return e != cudaSuccess ? e : staged_copy(ctx, pieces, chunks, threads, to_host, seen);
            }
        }
    }
    for (int i = 0; i < n; i++) {
        if (!pieces[i].bytes) continue;
        const cudaError_t e = to_host ? cudaMemcpyAsync(pieces[i].host, pieces[i].dev, pieces[i].bytes, cudaMemcpyDeviceToHost, st)
                                      : cudaMemcpyAsync(pieces[i].dev, pieces[i].host, pieces[i].bytes, cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return e;
        if (seen) seen(0, pieces[i].bytes);
    }
    return to_host ? cudaStreamSynchronize(st) : cudaSuccess;
}

}  // namespace gxy
