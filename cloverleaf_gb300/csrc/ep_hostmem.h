// ep_hostmem.h -- host-memory helpers of the calls on host buffers
// (ep_host.cpp; no CUDA).
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <atomic>
#include <memory>
#include <thread>
#include <vector>

namespace ep {

// Makes the pages of a result array resident from a few threads while the
// device computes, slab by slab, with MADV_POPULATE_WRITE: the contents stay
// as they are, so the array may overlap an input, and a call that fails before
// its download leaves it unchanged.  Pages of a fresh array that a
// device-to-host copy meets first are faulted in one by one through the host's
// page tables: a 4 MB download took 2.2 ms into a fresh array and 0.04 ms into
// a resident one, 205 MB 7.5 and 1.15 ms.  (An atomic addition of zero keeps
// the contents too, but maps the shared zero page first, whose replacement
// makes the device drop its translations: 24 us a page of 64 KB.)  205 MB take
// 2.2 ms on four threads; more stand in each other's way, 7.3 ms on eight.
// Where the kernel does not know the advice the pages are left to the copy.
// The copy follows slab by slab; smaller slabs let it start sooner (embeddings
// of 46 MB 1.59 ms with slabs of 32 MB, 1.51 with 8).  Arrays below THREADED,
// where starting threads costs more than they save, are made resident by
// wait(), on the OpenMP threads: 24 MB 0.98 ms, 1.10 with threads; 31 MB 1.17
// and 1.31; 36 MB 1.49 and 1.31.
class ResultPages {
public:
    static constexpr size_t SLAB = 8u << 20, THREADED = 32u << 20;

    ResultPages(void* p, size_t bytes);
    ~ResultPages();
    ResultPages(const ResultPages&) = delete;
    ResultPages& operator=(const ResultPages&) = delete;

    size_t slabs() const { return (bytes_ + SLAB - 1) / SLAB; }
    // Waits until slab i, bytes [i * SLAB, ...) of the array, is resident.
    void wait(size_t i);

private:
    static constexpr size_t THREADS = 4;

    void populate(size_t from, size_t to);
    void work();

    char* p_;
    size_t bytes_, page_, pieces_ = 0;
    bool later_ = false;                                // not started yet (small)
    std::atomic<size_t> next_{0};
    std::unique_ptr<std::atomic<uint32_t>[]> left_;     // pieces of each slab still to come
    std::vector<std::thread> threads_;
};

// Whether every id is below bound.
bool all_below(const uint32_t* ids, uint64_t n, uint64_t bound);

// Whether the n + 1 offsets do not decrease (several threads).
bool monotone(const uint64_t* off, uint64_t n);

}  // namespace ep
