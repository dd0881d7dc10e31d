// host_pages.cpp -- pages of the callers' result arrays.
#include "host_pages.h"

#include <stdint.h>
#include <algorithm>
#include <thread>

#ifdef __linux__
#include <sys/mman.h>
#include <unistd.h>
#endif

namespace fpt {

#ifdef __linux__
// Whether an array has its memory: nine of its pages, spread from the first to
// the last, do.  A buffer that a program keeps from call to call, pinned or
// not, passes; a new one fails at the first or, where the first page lies in a
// huge page that the allocator touched, the second.
static bool pages_present(uintptr_t begin, size_t pages, size_t page) {
    constexpr size_t kProbes = 8;
    for (size_t k = 0; k <= kProbes; ++k) {
        unsigned char there = 0;
        if (mincore(reinterpret_cast<void *>(begin + (pages - 1) * k / kProbes * page), page, &there) != 0 || !(there & 1u)) return false;
    }
    return true;
}
#endif

// A result array that the caller has just allocated has no pages yet.  The copy
// from the device then takes a fault per page: 1 ms for the 41 MB of a 1080p
// frame, and up to 35 ms where the GPU takes the faults itself; into populated
// pages the copy takes 0.3 ms.  Between the launch of the kernels and the
// wait for them the host is idle, so the pages are populated there
// (MADV_POPULATE_WRITE: no byte changes, pages that are there are left alone,
// and on memory or kernels that do not know it the call fails and the copy
// faults as before).  Clearing pages is bound by one core's 20 GB/s: an array
// is shared between as many threads as it has full 4 MB, four at most.
// An array whose pages are there is left alone: the threads would be created
// for nothing (distances of 1M points into a kept array: Menger 288-305 us with
// them, 233-242 without; 1080p voxel frame of a 64^3 grid 486-571 and 464 us).
void populate_pages(std::initializer_list<HostRange> ranges) {
#ifdef __linux__
    constexpr int kPopulateWrite = 23;   // MADV_POPULATE_WRITE (Linux 5.14)
    constexpr size_t kPerThread = size_t(4) << 20;
    const size_t page = size_t(sysconf(_SC_PAGESIZE));
    for (const HostRange &r : ranges) {
        if (!r.data || r.bytes == 0) continue;
        const uintptr_t begin = (reinterpret_cast<uintptr_t>(r.data) + page - 1) / page * page;
        const uintptr_t end = (reinterpret_cast<uintptr_t>(r.data) + r.bytes) / page * page;
        if (end <= begin) continue;
        const size_t pages = (end - begin) / page;
        if (pages_present(begin, pages, page)) continue;
        const size_t parts = std::min<size_t>(4, std::max<size_t>(1, (end - begin) / kPerThread));
        auto part = [=](size_t k) {
            const uintptr_t a = begin + pages * k / parts * page, b = begin + pages * (k + 1) / parts * page;
            (void)madvise(reinterpret_cast<void *>(a), b - a, kPopulateWrite);
        };
        std::thread helpers[3];
        size_t started = 0;
        try {
            for (; started + 1 < parts; ++started) helpers[started] = std::thread(part, started + 1);
        } catch (...) {   // no thread to be had: the rest is done here
        }
        part(0);
        for (size_t k = started + 1; k < parts; ++k) part(k);
        for (size_t k = 0; k < started; ++k) helpers[k].join();
    }
#else
    (void)ranges;
#endif
}

}  // namespace fpt
