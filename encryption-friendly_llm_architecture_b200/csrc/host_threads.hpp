// Work on host memory dealt to a few threads.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <thread>
#include <sys/mman.h>

constexpr int kCopyThreads = 4;
// work(begin, end) over [0, n) on up to `cap` threads (at most kCopyThreads), `words` doubles moved in all.  A thread that cannot be had
// (no room for it, no more of them) leaves its share to the caller, so nothing is thrown and every thread that has started is joined.
template <class F> void in_threads(int cap, size_t n, size_t words, F &&work) {
    const size_t per = (size_t)1 << 16; // words that are worth a thread
    const int k = (int)std::max<size_t>(1, std::min<size_t>({(size_t)std::min(cap, kCopyThreads), words / per, n}));
    auto part = [&](int t) { work(n * t / k, n * (t + 1) / k); };
    std::thread pool[kCopyThreads];
    int started = 1;
    try { for (; started < k; ++started) pool[started] = std::thread(part, started); } catch (...) {}
    part(0);
    for (int t = started; t < k; ++t) part(t);
    for (int t = 1; t < started; ++t) pool[t].join();
}

// Memory that results are about to be copied to: threads of their own ask the system for its pages, first ones first, while the device is at work, so
// that the copies do not stop at each of them (a page that is not there yet costs 0.7 us here).  What the memory holds stays; a system that cannot do it, or a thread that cannot be had,
// leaves the pages to the copies.  The threads are joined at the end of the scope.
class Pages {
    static constexpr int kMost = 2 * kCopyThreads;
    std::thread pool_[kMost];
    int started_ = 0, cap_;

public:
    explicit Pages(int cap) : cap_(std::min(cap, kCopyThreads)) {}
    Pages(const Pages &) = delete;
    ~Pages() { for (int t = 0; t < started_; ++t) pool_[t].join(); }
    void ask(const double *memory, std::size_t words) { // at most twice
        constexpr std::size_t kPage = 4096;
        const std::size_t first = ((std::uintptr_t)memory + kPage - 1) / kPage, last = (std::uintptr_t)(memory + words) / kPage;
        if (first >= last || last - first < 128) return;
        // pages of a call: from 4 MB on the system may give out pages of 2 MB, each of which one thread should ask for
        const std::size_t block = last - first < 1024 ? 64 : 512, base = first / block * block, blocks = (last - base + block - 1) / block;
        const int k = (int)std::min<std::size_t>((std::size_t)cap_, blocks);
        try {
            for (int t = 0; t < k && started_ < kMost; ++t, ++started_)
                pool_[started_] = std::thread([=] {
                    for (std::size_t b = (std::size_t)t; b < blocks; b += (std::size_t)k) {
                        const std::size_t from = std::max(first, base + b * block), to = std::min(last, base + (b + 1) * block);
                        if (madvise(reinterpret_cast<void *>(from * kPage), (to - from) * kPage, 23 /* MADV_POPULATE_WRITE */) != 0) return;
                    }
                });
        } catch (...) {}
    }
};
