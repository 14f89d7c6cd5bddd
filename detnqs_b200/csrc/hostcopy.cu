// hostcopy.cu -- staged device-to-host copies (hostcopy.cuh).

#include "hostcopy.cuh"

#include <atomic>
#include <algorithm>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>

namespace dnq {

namespace {

constexpr size_t kHostCopyMin = size_t(8) << 20;
constexpr size_t kChunk = size_t(2) << 20;
constexpr int kWorkers = 8;                      // at most
constexpr size_t kSlots = 2 * kWorkers * kChunk;  // 32 MiB: two slots per worker
constexpr int kKept = 2;                          // slot sets kept for later copies

struct SlotPool {
    std::mutex mu;
    char* kept[kKept] = {};
    long contexts = 0;
    char* take() {
        {
            std::lock_guard<std::mutex> lk(mu);
            for (auto& p : kept)
                if (p) {
                    char* q = p;
                    p = nullptr;
                    return q;
                }
        }
        void* q = nullptr;
        if (cudaHostAlloc(&q, kSlots, cudaHostAllocPortable) != cudaSuccess) {
            (void)cudaGetLastError();
            return nullptr;   // no page-locked memory: the plain copy does it
        }
        return static_cast<char*>(q);
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
        if (--P.contexts == 0)
            for (int k = 0; k < kKept; ++k) std::swap(old[k], P.kept[k]);
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
    char* slots = todo.empty() ? nullptr : pool().take();
    if (!slots) {
        for (const Piece& p : todo)
            DNQ_CUDA(cudaMemcpyAsync(p.dst, p.src, p.n, cudaMemcpyDeviceToHost, s_));
        DNQ_CUDA(cudaStreamSynchronize(s_));
        return;
    }
    int dev = 0;
    std::atomic<int> failed{(int)cudaGetDevice(&dev)};
    const unsigned cores = std::thread::hardware_concurrency();
    const int nw = (int)std::max<size_t>(
        1, std::min<size_t>({(size_t)kWorkers, (size_t)(cores > 1 ? cores / 2 : 1), todo.size() / 2}));
    // Worker w copies chunks w, w + nw, ...: the next one fills a slot on the
    // stream while the last one is copied out of the other.
    std::atomic<size_t> next{0};
    auto work = [&](int w) noexcept {
        cudaEvent_t ev[2] = {};
        cudaError_t e = cudaSetDevice(dev);
        for (auto& x : ev)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
        char* slot[2] = {slots + 2 * w * kChunk, slots + (2 * w + 1) * kChunk};
        const Piece* held[2] = {};
        int k = 0;
        for (;;) {
            const size_t i = e == cudaSuccess && !failed.load() ? next++ : todo.size();
            if (i < todo.size()) {
                held[k] = &todo[i];
                e = cudaMemcpyAsync(slot[k], todo[i].src, todo[i].n, cudaMemcpyDeviceToHost, s_);
                if (e == cudaSuccess) e = cudaEventRecord(ev[k], s_);
            } else {
                held[k] = nullptr;
            }
            k ^= 1;
            if (held[k] && e == cudaSuccess) {
                e = cudaEventSynchronize(ev[k]);
                if (e == cudaSuccess) std::memcpy(held[k]->dst, slot[k], held[k]->n);
            }
            if (e != cudaSuccess || (!held[0] && !held[1])) break;
            held[k] = nullptr;
        }
        if (e != cudaSuccess) failed = (int)e;
        for (auto& x : ev)
            if (x) cudaEventDestroy(x);
    };
    std::vector<std::thread> team;
    try {
        team.reserve(nw - 1);
        for (int w = 1; w < nw; ++w) team.emplace_back(work, w);
    } catch (const std::exception&) {   // fewer threads: the chunks are shared out as they go
    }
    work(0);
    for (auto& t : team) t.join();
    const cudaError_t done = cudaStreamSynchronize(s_);   // no copy into a slot is left
    pool().give(slots);
    DNQ_CUDA((cudaError_t)failed.load());
    DNQ_CUDA(done);
}

}  // namespace dnq
