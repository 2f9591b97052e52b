// Fresh host memory made present by several host threads before a mesh is copied
// into it (no counterpart in the reference, whose vectors are filled by one
// thread).
//
// A new array of tens of megabytes has no pages yet; the copy back would bring
// them in one by one, on one thread, which clears each: 2.4 ms for the 52 MB mesh
// of a 256^3 noise volume, against 0.3 ms for the copy itself.  Memory that the
// allocator kept from an earlier array has its pages already (arrays of up to
// some 30 MB, call after call): what is missing is looked up first, and nothing is
// done for less than a piece (extract of 120^3 noise, 21 MB, again and again: 382 us
// with the faults of the first call only, 473 with helpers for pages that were
// there, 331 now; every mesh kept: 1,386, 766, 696).
//
// The helper threads live for one call and come from one budget for the whole
// process: callers on many threads share it instead of bringing up a team each,
// and none is left behind. Where none can be made (a limit on threads or address
// space) the caller does the work alone.
//
// What bounds it: the kernel's page allocation, where more threads get into each
// other's way. 16 Grace cores, 64 KB pages, 51 / 300 MB: 4 threads 0.67 / 3.4 ms,
// 16 kept ones 0.82 / 4.8, 16 made for the call 1.5 / 10.0.
#include <sys/mman.h>
#include <unistd.h>

#include <atomic>
#include <cstdint>
#include <thread>

#include "../../include/miniiso.h"

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23  // Linux 5.14
#endif

namespace {

constexpr int kMaxHelpers = 3;
std::atomic<int> g_helpers{0};  // of all calls under way

// The ranges cut into pieces of `piece` bytes, which the threads of a call take from `next`.
struct Pieces {
    int64_t n;
    void* const* ptrs;
    const int64_t* bytes;
    uintptr_t page, piece;
    std::atomic<int64_t> next{0};

    // Pages of range r; false: it has none.
    bool pages(int64_t r, uintptr_t& a, uintptr_t& e) const
    {
        if (!ptrs[r] || bytes[r] <= 0) return false;
        a = reinterpret_cast<uintptr_t>(ptrs[r]) & ~(page - 1);
        e = (reinterpret_cast<uintptr_t>(ptrs[r]) + (uintptr_t)bytes[r] + page - 1) & ~(page - 1);
        return true;
    }
    int64_t count(int64_t r) const
    {
        uintptr_t a = 0, e = 0;
        return pages(r, a, e) ? (int64_t)((e - a + piece - 1) / piece) : 0;
    }
    // Bytes of range r without a page, counted up to `enough`; 0 where the system cannot say.
    uintptr_t missing(int64_t r, uintptr_t enough) const
    {
        unsigned char present[4096];  // of 16 MB or more at a time
        uintptr_t a = 0, e = 0, n = 0;
        if (!pages(r, a, e)) return 0;
        for (uintptr_t p = a; p < e && n < enough;) {
            const uintptr_t most = sizeof present * page, len = e - p < most ? e - p : most;
            if (mincore(reinterpret_cast<void*>(p), len, present) != 0) return 0;
            for (uintptr_t q = 0; q < len / page; ++q) n += present[q] & 1 ? 0 : page;
            p += len;
        }
        return n;
    }
    // A thread's share: pieces in ascending order, so that one walk over the ranges finds them all.
    void work()
    {
        int64_t before = 0, q = next++;  // before: the pieces of the ranges before r
        for (int64_t r = 0; r < n; ++r) {
            const int64_t c = count(r);
            for (; q < before + c; q = next++) {
                uintptr_t a = 0, e = 0;
                (void)pages(r, a, e);
                const uintptr_t p = a + (uintptr_t)(q - before) * piece, end = e - p > piece ? p + piece : e;
                // what the memory holds stays as it is; a range that cannot be populated (an older kernel, device
                // memory) is left to the copy
                (void)madvise(reinterpret_cast<void*>(p), end - p, MADV_POPULATE_WRITE);
            }
            before += c;
        }
    }
};

// Takes up to `want` of the process's helpers.
int take_helpers(int64_t want)
{
    const int cpus = (int)std::thread::hardware_concurrency();
    const int limit = cpus - 1 < kMaxHelpers ? cpus - 1 : kMaxHelpers;
    int used = g_helpers.load();
    for (;;) {
        const int64_t room = limit - used, take = want < room ? want : room;
        if (take <= 0) return 0;
        if (g_helpers.compare_exchange_weak(used, used + (int)take)) return (int)take;
    }
}

}  // namespace

extern "C" {

iso_status iso_populate_host(int64_t n, void* const* ptrs, const int64_t* bytes)
{
    if (n < 0 || (n > 0 && (!ptrs || !bytes))) return ISO_ERR_INVALID_ARG;
    Pieces p;
    p.n = n;
    p.ptrs = ptrs;
    p.bytes = bytes;
    p.page = (uintptr_t)sysconf(_SC_PAGESIZE);
    p.piece = 1u << 20 > p.page ? 1u << 20 : p.page;  // a multiple of the page, cleared by one thread
    const uintptr_t enough = (kMaxHelpers + 1) * p.piece;  // a piece for every thread
    uintptr_t missing = 0;
    for (int64_t r = 0; r < n && missing < enough; ++r) missing += p.missing(r, enough);
    if (missing < p.piece) return ISO_OK;
    const int helpers = take_helpers((int64_t)(missing / p.piece) - 1);
    std::thread team[kMaxHelpers];
    int made = 0;
    try {
        for (; made < helpers; ++made) team[made] = std::thread([&p] { p.work(); });
    } catch (...) {  // no more threads to be had
    }
    p.work();
    for (int q = 0; q < made; ++q) team[q].join();
    g_helpers -= helpers;
    return ISO_OK;
}

}  // extern "C"
