// hostcopy.cuh -- large results to pageable host memory.
//
// The driver copies to pageable memory through one staging thread, which also
// takes the page faults of a fresh result array: 5 GB/s measured for the 220 MB
// of blocks of a 403-row proxy build.  Copies of kHostCopyMin bytes or more
// go through page-locked slots instead: the calling thread, the only one to use
// the caller's stream, keeps the GPU filling free slots while worker threads
// copy the chunks on (and fault them in).  106 MB of H_VP in 24 ms before, 5.6 ms
// now.
#pragma once

#include <vector>

#include "common.cuh"

namespace dnq {

// Device-to-host copies run together: add() them, then run() returns when
// all are done (after the work already on the stream).  Destinations that are
// device or page-locked memory, and small ones, go through cudaMemcpyAsync.
class HostCopies {
public:
    explicit HostCopies(cudaStream_t s) : s_(s) {}
    template <class T>
    void add(T* dst, const T* src, size_t count) {
        if (dst && count) add_bytes(dst, src, count * sizeof(T));
    }
    void run();

private:
    struct Piece {
        char* dst;
        const char* src;
        size_t n;
    };
    void add_bytes(void* dst, const void* src, size_t n);
    cudaStream_t s_;
    std::vector<Piece> pieces_;   // chunks of the staged copies
};

// Contexts alive: the page-locked slots kept between copies are released with
// the last of them, and none are made without one (locking and releasing them
// for every copy took get_ham_eff of 2e6 entries from 4.8 to 39 ms).
void host_slots_hold();
void host_slots_drop() noexcept;
struct HostSlots {
    HostSlots() { host_slots_hold(); }
    ~HostSlots() { host_slots_drop(); }
    HostSlots(const HostSlots&) = delete;
    HostSlots& operator=(const HostSlots&) = delete;
};

}  // namespace dnq
