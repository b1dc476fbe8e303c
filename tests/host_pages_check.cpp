// Host check of touch_pages (csrc/host_pages.cpp): whatever the given ranges hold stays as it is, also while another
// thread writes to them; fresh memory gets its pages; ranges of odd addresses and sizes are not left.  Exit status 0
// when all hold.  Built and run by tests/test_host_pages.py (CPU only).
#include <sys/mman.h>
#include <unistd.h>

#include <atomic>
#include <cstdio>
#include <thread>

#include "../pachydermacoustic_universal_gb300/csrc/engine.h"

static unsigned char pattern(size_t i) { return (unsigned char)(1 + i * 2654435761u % 251); }

int main() {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = 40u << 20;
    int bad = 0;
    // fresh pages become resident, and read as zero
    unsigned char *f = (unsigned char *)mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (f == MAP_FAILED) return 2;
    pach::touch_pages({{f, n}});
    std::vector<unsigned char> in(n / page);
    if (mincore(f, n, in.data()) == 0)
        for (unsigned char r : in) bad += !(r & 1);
    std::printf("%d pages not resident\n", bad);
    // contents stay: several ranges, odd addresses and lengths, nulls, less than a page
    for (size_t i = 0; i < n; ++i) f[i] = pattern(i);
    pach::touch_pages({{f + 1, n - 1}, {nullptr, n}, {f + 12345, 3 * page + 7}, {f + 7, page - 1}, {f, 0}});
    int changed = 0;
    for (size_t i = 0; i < n; ++i) changed += f[i] != pattern(i);
    std::printf("%d bytes changed\n", changed);
    // a writer beside: no write of its own is lost
    std::atomic<bool> stop{false};
    std::thread toucher([&] {
        while (!stop) pach::touch_pages({{f, 8 * page}});
    });
    int lost = 0;
    volatile unsigned char *v = f;
    for (int k = 0; k < 2000000; ++k) {
        const size_t i = (size_t)(k & 7) * page;
        v[i] = (unsigned char)k;
        lost += v[i] != (unsigned char)k;
    }
    stop = true;
    toucher.join();
    std::printf("%d writes lost\n", lost);
    munmap(f, n);
    return bad || changed || lost;
}
