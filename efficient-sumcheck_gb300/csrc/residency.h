// residency.h -- where a caller's table is, and how passes may read it there.
// Plain C++, so that the rules are compiled and tested without a GPU.
#pragma once
#include <cstddef>
#include <cstdint>
#include <unistd.h>

namespace effsc {

enum class Residency {
    device,     // device memory
    managed,    // managed memory: its pages may be on their way
    pinned,     // pinned or registered host memory
    pageable    // host memory as malloc or mmap gives it, a mapped file included
};

// Reads that arrive within the link's latency.  A pageable (or managed) page may
// first have to be brought in, from a file at worst.
constexpr bool prompt_reads(Residency r) { return r == Residency::device || r == Residency::pinned; }

// The limit of a tensor-core pass's waits on its own loads.  The pass that copies
// host tables (from_host) may meet pages that are not there yet.  Its blocks
// have at most some 400 tiles in flight, 1 KB in each of 32 places of two MSB
// tables (LSB: 16 KB in each table): 3200 pages of 4 KB, so 100 s are 30 ms for
// each of them one after the other, a disk's slowest.
constexpr uint64_t tc_wait_ns(bool from_host) { return from_host ? 100000000000ULL : 1000000000ULL; }

// Rounds that the first pass of the InnerProduct start runs on the tensor
// cores (k_gram.cu): 4 where the proof has five, else 3; 0: the general form
// of direct loads without waits (k_ip012.cu, 3 rounds).  `addresses`: the
// tables' and their copies', or-ed (16-byte loads and stores).  Tables that are
// not prompt are read once, by the first pass, when it also copies them
// (`copied`, with the limit above); where they are read in place by both, the
// direct loads do it.
constexpr int ip_start_rounds(size_t L, size_t num_rounds, uintptr_t addresses, bool prompt, bool copied, size_t tile_items) {
    const int nv = num_rounds >= 5 ? 4 : 3;
    const size_t items = L >> nv;
    return (!prompt && !copied) || (addresses & 15) || items % tile_items || items / tile_items >= ((size_t)1 << 31) ? 0 : nv;
}

// Copying host words by a kernel that reads them in place: pageable memory that
// the GPU reads through the host's own page tables (elsewhere each page
// faults or moves to the GPU), from 64 KB on (below, latency either way).
constexpr bool kernel_copies(Residency r, bool host_page_tables, size_t words, uintptr_t address) {
    return r == Residency::pageable && host_page_tables && words >= ((size_t)1 << 13) && (address & 7) == 0;
}

// Bring the pages of pageable memory in before a kernel reads them, by a read
// in each: on the host a missing page is a microsecond, from the GPU ten.
// (Resident pages: 20 us for 128 MB of 64 KB pages, madvise(MADV_POPULATE_READ) 73.)
inline void touch_pages(const void* p, size_t bytes) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const volatile char* c = (const volatile char*)p;
    for (size_t at = 0; at < bytes; at += page - ((uintptr_t)(c + at) & (page - 1))) (void)c[at];
}

// The caller's memory while kernels read it: once `pending`, the scope is not
// left without having waited for them, on the errors' ways out as well.
template <class Wait>
struct ReadsInPlace {
    Wait wait;               // returns an error code, 0 for none
    bool pending = false;
    explicit ReadsInPlace(Wait w) : wait(w) {}
    ReadsInPlace(const ReadsInPlace&) = delete;
    int finish() {
        const bool p = pending;
        pending = false;
        return p ? (int)wait() : 0;
    }
    ~ReadsInPlace() { finish(); }
};

}  // namespace effsc
