// Work on host memory dealt to a few threads.
#pragma once
#include <algorithm>
#include <cstddef>
#include <thread>

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
