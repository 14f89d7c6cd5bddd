// hostcopy.cu -- staged device-to-host copies (hostcopy.cuh).

#include "hostcopy.cuh"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>

namespace dnq {

namespace {

constexpr size_t kHostCopyMin = size_t(8) << 20;
constexpr size_t kChunk = size_t(2) << 20;
constexpr int kWorkers = 8;                      // at most
constexpr size_t kSlots = 2 * kWorkers * kChunk;  // 32 MiB: two slots per worker
constexpr int kKept = 2;                          // slot sets kept for later copies
// A slot set takes the driver 31 ms to lock and 3.5 to release, as long as the
// plain copies of about this many bytes take more than the staged ones (111 MB
// into fresh arrays: 17 to 27 ms plain, 4.2 staged).
constexpr size_t kWorth = size_t(192) << 20;

struct SlotPool {
    std::mutex mu;
    char* kept[kKept] = {};
    int made = 0;       // sets there are, kept or in use
    long contexts = 0;
    size_t plain = 0;   // bytes copied the plain way under these contexts
    // A slot set for a copy of n bytes, or null: the plain copy does it.  A set
    // is made only where it can be kept, and once the plain copies have cost as
    // much.
    char* take(size_t n) {
        std::unique_lock<std::mutex> lk(mu);
        for (auto& p : kept)
            if (p) {
                char* q = p;
                p = nullptr;
                return q;
            }
        if (contexts == 0 || made == kKept) return nullptr;
        plain += n;
        if (plain < kWorth) return nullptr;
        ++made;
        lk.unlock();   // other copies and contexts do not wait for the driver
        void* q = nullptr;
        if (cudaHostAlloc(&q, kSlots, cudaHostAllocPortable) == cudaSuccess)
            return static_cast<char*>(q);
        (void)cudaGetLastError();
        lk.lock();
        --made;
        return nullptr;   // no page-locked memory
    }
    void give(char* q) noexcept {
        {
            std::lock_guard<std::mutex> lk(mu);
            if (contexts > 0)
                for (auto& p : kept)
                    if (!p) {
                        p = q;
                        return;
                    }
            --made;
        }
        cudaFreeHost(q);
    }
};
// Never destroyed: a copy may run while the process ends.
SlotPool& pool() {
    static SlotPool* p = new SlotPool;
    return *p;
}

}  // namespace

void host_slots_hold() {
    SlotPool& P = pool();
    std::lock_guard<std::mutex> lk(P.mu);
    ++P.contexts;
}

void host_slots_drop() noexcept {
    SlotPool& P = pool();
    char* old[kKept] = {};
    {
        std::lock_guard<std::mutex> lk(P.mu);
        if (--P.contexts == 0) {
            for (int k = 0; k < kKept; ++k) {
                std::swap(old[k], P.kept[k]);
                if (old[k]) --P.made;
            }
            P.plain = 0;
        }
    }
    for (char* p : old)
        if (p) cudaFreeHost(p);
}

void HostCopies::add_bytes(void* dst, const void* src, size_t n) {
    cudaPointerAttributes at{};
    bool pageable = true;
    if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) (void)cudaGetLastError();
    else pageable = at.type == cudaMemoryTypeUnregistered;
    if (!pageable || n < kHostCopyMin) {
        DNQ_CUDA(cudaMemcpyAsync(dst, src, n, cudaMemcpyDefault, s_));
        return;
    }
    for (size_t o = 0; o < n; o += kChunk)
        pieces_.push_back(Piece{static_cast<char*>(dst) + o, static_cast<const char*>(src) + o,
                                std::min(kChunk, n - o)});
}

void HostCopies::run() {
    std::vector<Piece> todo;
    todo.swap(pieces_);
    size_t bytes = 0;
    for (const Piece& p : todo) bytes += p.n;
    char* slots = todo.empty() ? nullptr : pool().take(bytes);
    if (!slots) {
        for (const Piece& p : todo)
            DNQ_CUDA(cudaMemcpyAsync(p.dst, p.src, p.n, cudaMemcpyDeviceToHost, s_));
        DNQ_CUDA(cudaStreamSynchronize(s_));
        return;
    }
    // All copies are issued by this thread: a stream handle need not name the
    // same stream in another one (cudaStreamPerThread).  Chunk i fills slot
    // i % ns once chunk i - ns is copied out of it; the workers take the chunks
    // in order, wait for their events and copy on.
    const unsigned cores = std::thread::hardware_concurrency();
    const int nw = (int)std::max<size_t>(
        1, std::min<size_t>({(size_t)kWorkers, (size_t)(cores > 1 ? cores / 2 : 1), todo.size() / 2}));
    const size_t ns = 2 * (size_t)nw;
    cudaEvent_t ev[2 * kWorkers] = {};
    std::mutex mu;
    std::condition_variable filled, freed;
    size_t issued = 0;               // chunks issued
    size_t out[2 * kWorkers] = {};   // per slot: chunks copied out of it
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    bool stop = false;
    cudaError_t failed = cudaSuccess;
    std::atomic<size_t> next{0};
    auto work = [&]() noexcept {
        cudaError_t err = cudaSetDevice(dev);
        for (;;) {
            const size_t i = next++;
            if (i >= todo.size()) break;
            {
                std::unique_lock<std::mutex> lk(mu);
                if (err == cudaSuccess) filled.wait(lk, [&] { return issued > i || stop; });
                if (err != cudaSuccess || issued <= i) break;
            }
            const size_t q = i % ns;
            err = cudaEventSynchronize(ev[q]);
            if (err == cudaSuccess) std::memcpy(todo[i].dst, slots + q * kChunk, todo[i].n);
            std::lock_guard<std::mutex> lk(mu);
            if (err != cudaSuccess) break;
            ++out[q];
            freed.notify_one();
        }
        if (err != cudaSuccess) {
            std::lock_guard<std::mutex> lk(mu);
            failed = err;
            stop = true;
            filled.notify_all();
            freed.notify_one();
        }
    };
    for (size_t q = 0; q < ns && e == cudaSuccess; ++q)
        e = cudaEventCreateWithFlags(&ev[q], cudaEventDisableTiming);
    std::vector<std::thread> team;
    try {
        team.reserve(nw);
        while (e == cudaSuccess && (int)team.size() < nw) team.emplace_back(work);
    } catch (const std::exception&) {   // fewer threads: the chunks are shared out as they go
    }
    const bool alone = team.empty();   // no thread at all: plain copies
    for (size_t i = 0; i < todo.size() && e == cudaSuccess; ++i) {
        if (alone) {
            e = cudaMemcpyAsync(todo[i].dst, todo[i].src, todo[i].n, cudaMemcpyDeviceToHost, s_);
            continue;
        }
        const size_t q = i % ns;
        {
            std::unique_lock<std::mutex> lk(mu);
            freed.wait(lk, [&] { return out[q] == i / ns || stop; });
            if (stop) break;
        }
        e = cudaMemcpyAsync(slots + q * kChunk, todo[i].src, todo[i].n, cudaMemcpyDeviceToHost, s_);
        if (e == cudaSuccess) e = cudaEventRecord(ev[q], s_);
        std::lock_guard<std::mutex> lk(mu);
        if (e == cudaSuccess) issued = i + 1;
        else stop = true;
        filled.notify_all();
    }
    for (auto& t : team) t.join();
    const cudaError_t done = cudaStreamSynchronize(s_);   // no copy into a slot is left
    for (auto& x : ev)
        if (x) cudaEventDestroy(x);
    pool().give(slots);
    DNQ_CUDA(e);
    DNQ_CUDA(failed);
    DNQ_CUDA(done);
}

}  // namespace dnq
