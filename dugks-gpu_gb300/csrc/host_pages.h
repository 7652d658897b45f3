// Physical pages for a host array that a device copy is about to fill.
//
// A result array fresh from the allocator has no pages yet; the copy then waits while one
// thread faults in and clears them one by one.  60 MB state on GB300 (64 KB pages): 3.43 ms
// into a fresh array against 0.37 ms into one with pages; with the pages populated here by
// three threads, while the device packs the state, 2.52 ms (one thread 3.31, five 2.63, eight
// 3.18 ms).
#pragma once
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <thread>
#include <vector>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace dg {

constexpr size_t kPopulateBytes = size_t(4) << 20;  // a thread's least share: 0.2 ms of clearing, several times its start
constexpr int kPopulateThreads = 3;  // starting more waits for the address-space lock the first ones hold

// Populates the missing pages of [p, p + bytes), contents unchanged.  Does nothing where few
// are missing, and on kernels without MADV_POPULATE_WRITE (the copy then faults them in).
inline void populate_pages(void *p, size_t bytes) noexcept
{
    try {
        const size_t page = size_t(sysconf(_SC_PAGESIZE));
        const uintptr_t a = reinterpret_cast<uintptr_t>(p);
        const uintptr_t lo = (a + page - 1) / page * page, hi = (a + bytes) / page * page;
        if (hi < lo + kPopulateBytes) return;
        std::vector<unsigned char> in((hi - lo) / page);
        if (mincore(reinterpret_cast<void *>(lo), hi - lo, in.data())) return;
        const size_t missing = size_t(std::count_if(in.begin(), in.end(), [](unsigned char c) { return !(c & 1); }));
        const size_t n = std::min<size_t>({missing * page / kPopulateBytes, size_t(kPopulateThreads),
                                           size_t(std::max(1u, std::thread::hardware_concurrency()))});
        if (!n) return;
        auto share = [&](size_t t) {
            const size_t b = in.size() * t / n * page, e = in.size() * (t + 1) / n * page;
            (void)madvise(reinterpret_cast<void *>(lo + b), e - b, MADV_POPULATE_WRITE);
        };
        std::vector<std::thread> pool;
        pool.reserve(n - 1);
        try {
            for (size_t t = 1; t < n; ++t) pool.emplace_back(share, t);
        } catch (...) {
            // fewer threads: the copy faults in what they would have
        }
        share(0);
        for (auto &t : pool) t.join();
    } catch (...) {
    }
}

}  // namespace dg
