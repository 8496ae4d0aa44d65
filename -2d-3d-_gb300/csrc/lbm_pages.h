// lbm_pages.h - bringing the pages of a host array that is about to be written whole into memory.
#pragma once

#include <sched.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <thread>
#include <vector>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23  // Linux 5.14; a kernel without it refuses, and the copy faults the pages in
#endif

namespace lbm {

// The memory node of the CPU that the calling thread is on.
inline unsigned memory_node() {
    unsigned cpu = 0, node = 0;
    getcpu(&cpu, &node);
    return node;
}

// Bring the pages of [dst, dst + bytes) into memory with a few threads.
// A copy into a fresh allocation otherwise takes one page fault after the other (GB300 host: 27
// GB/s, against 90 GB/s for the copy itself; lbm_get_state into fresh arrays before / after:
// 134 MB 6.6 / 4.0 ms, 453 MB 19 / 11 ms).
// Only whole pages inside the array are touched; where the kernel refuses (older kernels, other
// kinds of memory), the copy faults them as before.  A page lands on the node of the thread that
// touches it first, so a helper that runs on another node than the caller takes no part, and the
// pieces that it would have taken are left to the others and the caller.
inline void populate_pages(void* dst, size_t bytes) {
    // bytes of a piece: below, starting a thread costs what it saves.  More than four threads wait for
    // each other in the kernel (453 MB by 1 / 2 / 4 / 8 / 16 threads: 14.0 / 7.6 / 4.9 / 6.8 / 7.9 ms).
    constexpr size_t kEach = size_t(4) << 20;
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const uintptr_t b = ((uintptr_t)dst + page - 1) / page * page, e = ((uintptr_t)dst + bytes) / page * page;
    if (e <= b || e - b < kEach) return;
    // an array that is in memory already needs nothing (17 MB: 0.11 ms, 0.21 with the threads): look
    // at its first, middle and last page.  Each look costs such an array about 0.4 us (7 MB without / with
    // three / with eight: 50.2 / 52.1 / 53.8 us).
    int absent = 0;
    for (int k = 0; k < 3; ++k) {
        unsigned char in = 0;
        if (mincore((void*)(b + (e - b - page) / 2 * k / page * page), page, &in) != 0) return;
        absent += !(in & 1);
    }
    if (absent == 0) return;
    const size_t each = (kEach + page - 1) / page * page, pieces = (e - b + each - 1) / each;
    const unsigned node = memory_node();
    std::atomic<size_t> next{0};
    auto take = [&] {
        for (size_t t; (t = next++) < pieces;)
            madvise((void*)(b + t * each), std::min<size_t>(each, e - b - t * each), MADV_POPULATE_WRITE);
    };
    const size_t n = std::min<size_t>({4, (e - b) / kEach, std::max(1u, std::thread::hardware_concurrency())});
    std::vector<std::thread> others;
    try {
        others.reserve(n);
        for (size_t t = 1; t < n; ++t)
            others.emplace_back([&] {
                if (memory_node() == node) take();
            });
    } catch (...) {  // no more threads: the others take what is left
    }
    take();
    for (std::thread& t : others) t.join();
}

}  // namespace lbm
