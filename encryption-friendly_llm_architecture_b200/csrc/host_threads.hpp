// Work on host memory dealt to a few threads.
#pragma once
#include <algorithm>
#include <atomic>
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

// Memory that results are about to be copied to: up to `cap` threads, and the caller while it waits (help), ask the system for its pages, first ones first, while
// the device is at work, so that the copies do not stop at each of them (a page that is not there yet costs 0.5 to 0.7 us here).  What the memory holds stays; a
// system that cannot do it, or a thread that cannot be had, leaves the pages to the copies.  stop() joins the threads, as the end of the scope does, and leaves the rest to the copies
// and to the caller.
class Pages {
    static constexpr std::size_t kPage = 4096;
    struct Range { std::size_t first, last; }; // whole pages of an array
    Range range_[2] = {};
    std::size_t block_ = 0, blocks_ = 0; // pages of a block; blocks of all arrays, in turns
    int arrays_ = 1, started_ = 0, cap_;
    std::atomic<std::size_t> next_{0};
    std::atomic<bool> stop_{false};
    std::thread pool_[kCopyThreads];

    static Range pages_of(const double *memory, std::size_t words) {
        const Range r{((std::uintptr_t)memory + kPage - 1) / kPage, (std::uintptr_t)(memory + words) / kPage};
        return r.first < r.last ? r : Range{0, 0};
    }

public:
    explicit Pages(int cap) : cap_(std::max(0, std::min(cap, kCopyThreads))) {}
    Pages(const Pages &) = delete;
    ~Pages() { stop(); }
    // of one array, or of two that are written side by side; ends what was asked for before
    void ask(const double *memory, std::size_t words, const double *second = nullptr) {
        stop();
        blocks_ = 0;
        range_[0] = pages_of(memory, words);
        range_[1] = second ? pages_of(second, words) : Range{0, 0};
        arrays_ = second ? 2 : 1;
        const std::size_t most = std::max(range_[0].last - range_[0].first, range_[1].last - range_[1].first);
        if (most < 128) return;
        // pages of a call: from 4 MB on the system may give out pages of 2 MB, each of which one thread should ask for
        block_ = most < 1024 ? 64 : 512;
        blocks_ = (most + 2 * block_ - 2) / block_ * arrays_;
        next_ = 0;
        stop_ = false;
        try {
            for (; started_ < cap_ && (std::size_t)started_ < blocks_; ++started_) pool_[started_] = std::thread([this] { while (!stop_.load(std::memory_order_relaxed) && help()) {} });
        } catch (...) {}
    }
    bool help() { // the next block; false when there is none
        const std::size_t b = next_.fetch_add(1, std::memory_order_relaxed);
        if (b >= blocks_) return false;
        const Range &r = range_[b % arrays_];
        const std::size_t base = r.first / block_ * block_ + b / arrays_ * block_, from = std::max(r.first, base), to = std::min(r.last, base + block_);
        if (from < to && madvise(reinterpret_cast<void *>(from * kPage), (to - from) * kPage, 23 /* MADV_POPULATE_WRITE */) != 0) next_ = blocks_;
        return true;
    }
    void stop() {
        stop_ = true;
        for (int t = 0; t < started_; ++t) pool_[t].join();
        started_ = 0;
    }
};
