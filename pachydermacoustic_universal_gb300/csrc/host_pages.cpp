// host_pages.cpp -- gives freshly allocated host arrays their pages before a copy from the device.
#include <sys/mman.h>
#include <unistd.h>

#include <cerrno>

#include "engine.h"

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23  // Linux 5.14
#endif

// The kernel populates the pages that are not there as by a write that changes nothing, and a read of each page takes
// the fault of those that its NUMA balancing has unmapped meanwhile: left to the GPU, those make one download in
// five of the arena's 254 MB of pinned arrays 6 to 16 ms long instead of 3.  Where the kernel cannot populate, an
// atomic OR with nothing does it a page at a time; on Arm that faults twice a fresh page, as a read first.
// Memory that is not the process's own is left to the copy.
// 203 MB in 64 KB pages, fresh / there already, ms: 2.3 / 0.13 on four threads, a megabyte at a time; populated without
// asking 2.2 / 1.8; on 16 threads, which wait for one another's address space, 5.7; a store a page on 16 1.8 / 0.34;
// an atomic OR 10.9.
constexpr size_t kTouchBytes = size_t(1) << 20, kTouchThreads = 4;

void pach::touch_pages(const std::vector<std::pair<void *, size_t>> &ranges) {
    const size_t page = (size_t)std::max(4096l, sysconf(_SC_PAGESIZE));
    std::vector<std::pair<unsigned char *, size_t>> runs;  // first page, pages
    size_t total = 0;
    for (const auto &r : ranges) {
        if (!r.first || r.second < page) continue;  // too small to matter
        const uintptr_t a = reinterpret_cast<uintptr_t>(r.first), a0 = a / page * page;
        runs.emplace_back(reinterpret_cast<unsigned char *>(a0), (a + r.second - a0 + page - 1) / page);
        total += runs.back().second;
    }
    auto touch = [&](size_t a, size_t b) {
        size_t next = 0;
        for (const auto &r : runs) {
            const size_t first = next, i0 = std::max(a, first), i1 = std::min(b, first + r.second);
            next += r.second;
            if (i0 < i1) {
                unsigned char *p = r.first + (i0 - first) * page;
                std::vector<unsigned char> in(i1 - i0);
                if (mincore(p, (i1 - i0) * page, in.data())) continue;
                const bool there = std::all_of(in.begin(), in.end(), [](unsigned char c) { return c & 1; });
                const int e = !there && madvise(p, (i1 - i0) * page, MADV_POPULATE_WRITE) ? errno : 0;
                const bool old = e == EINVAL && madvise(p, page, MADV_NORMAL) == 0;  // mapped, but not to be populated
                if (e && !old) continue;
                for (size_t i = i0; i < i1; ++i, p += page) {
                    volatile unsigned char *q = p;
                    if (old) __atomic_fetch_or(q, 0, __ATOMIC_RELAXED);
                    else (void)*q;
                }
            }
        }
    };
    try {
        parallel_chunks(total, std::max<size_t>(1, kTouchBytes / page), touch, kTouchThreads);
    } catch (const std::exception &) {
        // no thread to be had: the copy faults the pages in
    }
}
