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

// Memory that results are about to be copied to: up to `cap` threads ask the system for its pages, first ones first, while the device is at work, so
// that the copies do not stop at each of them (a page that is not there yet costs 0.7 us here).  What the memory holds stays; a system that cannot do it, or a thread that cannot be had,
// leaves the pages to the copies.  The threads are joined at the end of the scope; until then running() of them are at work, and whoever counts threads deals
// so many fewer to the copies.
class Pages {
    static constexpr std::size_t kPage = 4096;
    std::thread pool_[kCopyThreads];
    std::atomic<int> running_{0};
    int started_ = 0, cap_;

    struct Range { std::size_t first, last; }; // whole pages of an array
    static Range pages_of(const double *memory, std::size_t words) {
        const Range r{((std::uintptr_t)memory + kPage - 1) / kPage, (std::uintptr_t)(memory + words) / kPage};
        return r.first < r.last ? r : Range{0, 0};
    }

public:
    explicit Pages(int cap) : cap_(std::max(0, std::min(cap, kCopyThreads))) {}
    Pages(const Pages &) = delete;
    ~Pages() { for (int t = 0; t < started_; ++t) pool_[t].join(); }
    int running() const { return running_.load(std::memory_order_acquire); }
    // of one array, or of two that are written side by side.  More calls share what is left of the cap.
    void ask(const double *memory, std::size_t words, const double *second = nullptr) {
        const Range r[2] = {pages_of(memory, words), second ? pages_of(second, words) : Range{0, 0}};
        const std::size_t most = std::max(r[0].last - r[0].first, r[1].last - r[1].first), arrays = second ? 2 : 1;
        if (most < 128) return;
        // pages of a call: from 4 MB on the system may give out pages of 2 MB, each of which one thread should ask for
        const std::size_t block = most < 1024 ? 64 : 512, blocks = (most + 2 * block - 2) / block;
        const int left = cap_ - started_, k = (int)std::min<std::size_t>((std::size_t)left, blocks * arrays);
        for (int t = 0; t < k; ++t) {
            running_.fetch_add(1, std::memory_order_relaxed);
            try {
                pool_[started_] = std::thread([=] {
                    for (std::size_t b = (std::size_t)t; b < blocks * arrays; b += (std::size_t)k) {
                        const Range &a = r[b % arrays];
                        const std::size_t base = a.first / block * block + b / arrays * block, from = std::max(a.first, base), to = std::min(a.last, base + block);
                        if (from < to && madvise(reinterpret_cast<void *>(from * kPage), (to - from) * kPage, 23 /* MADV_POPULATE_WRITE */) != 0) break;
                    }
                    running_.fetch_sub(1, std::memory_order_release);
                });
            } catch (...) {
                running_.fetch_sub(1, std::memory_order_relaxed);
                return;
            }
            ++started_;
        }
    }
};
