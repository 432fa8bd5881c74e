// Pages of a host array made before a copy into it (host code only).
#pragma once
#include <sched.h>
#include <sys/mman.h>
#include <unistd.h>

#include <stddef.h>
#include <stdint.h>

#include <atomic>
#include <thread>
#include <vector>

namespace ps3d {

// processors this process may run on
inline int allowed_cpus()
{
    cpu_set_t set;
    CPU_ZERO(&set);
    const int n = sched_getaffinity(0, sizeof(set), &set) ? 1 : CPU_COUNT(&set);
    return n < 1 ? 1 : n;
}

// Pages of a fresh host array (numpy's zeros, calloc) exist only after their
// first write, and the driver's copy into them faults page by page: 43 ms for
// the 51 MB of a 128^3 state, against 1 ms into pages that exist.  The pages
// are made first (MADV_POPULATE_WRITE keeps their contents; where the kernel
// lacks it, or for memory it does not take, the copy works as before).  The
// calling thread makes the first part; only if that is taken, and there is
// more, do others join it: at most seven, and no more than the process has
// processors.  From 8 MB on: smaller arrays come from heap pages that were in
// use before, and copy in well under a millisecond.  Returns the number of
// threads started.
inline int populate(void *p, size_t bytes)
{
    int started = 0;
#ifdef MADV_POPULATE_WRITE
    constexpr size_t MIN = (size_t)8 << 20, PART = (size_t)4 << 20;
    if (bytes < MIN) return 0;
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    char *a = (char *)(((uintptr_t)p + page - 1) / page * page);
    char *e = (char *)(((uintptr_t)p + bytes) / page * page);
    // an array that was written before has its pages: 16 of them tell
    bool fresh = false;
    for (int i = 0; i < 16 && !fresh; ++i) {
        unsigned char in = 1;
        char *q = a + (size_t)(e - a - 1) / 16 * i / page * page;
        fresh = mincore(q, page, &in) != 0 || !(in & 1);
    }
    if (!fresh) return 0;
    std::atomic<size_t> next{0};
    const auto part = [&] {  // makes the next part; false when there is none or it is refused
        const size_t o = next.fetch_add(PART), all = (size_t)(e - a);
        return o < all && madvise(a + o, all - o < PART ? all - o : PART, MADV_POPULATE_WRITE) == 0;
    };
    if (!part()) return 0;
    const auto work = [&] {
        while (part()) {}
    };
    const size_t left = ((size_t)(e - a) - 1) / PART;  // parts after the first
    int want = allowed_cpus() - 1;
    if (want > 7) want = 7;
    if ((size_t)want + 1 > left) want = (int)left - 1;
    std::vector<std::thread> t;
    try {
        for (; started < want; ++started) t.emplace_back(work);
    } catch (...) {  // no more threads: the ones that run do the work
    }
    work();
    for (std::thread &x : t) x.join();
#endif
    return started;
}

}  // namespace ps3d
