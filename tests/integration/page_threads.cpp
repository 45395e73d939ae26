// Pages over a stand-in for the system call: no more threads than the cap; each page of one array or of two is asked for once, by threads or by the caller; after
// stop() no thread is at work, so that copies stay within a budget.  Prints what fails; 0 when nothing does.
#include "host_threads.hpp"

#include <chrono>
#include <cstdio>
#include <map>
#include <mutex>
#include <set>

static std::mutex lock;
static std::set<std::thread::id> threads;
static std::map<std::uintptr_t, int> asked;
static std::atomic<int> at_work{0}, most{0};
static std::atomic<bool> refuse{false};
static void work(int us) {
    const int now = ++at_work;
    for (int m = most; now > m && !most.compare_exchange_weak(m, now);) {}
    std::this_thread::sleep_for(std::chrono::microseconds(us));
    --at_work;
}
extern "C" int madvise(void *p, size_t n, int) noexcept {
    work(20);
    std::lock_guard<std::mutex> g(lock);
    threads.insert(std::this_thread::get_id());
    if (refuse) return -1;
    for (size_t i = 0; i < n / 4096; ++i) ++asked[(std::uintptr_t)p / 4096 + i];
    return 0;
}

static int bad = 0;
#define EXPECT(x) do { if (!(x)) { std::printf("line %d: %s (cap %d, %zu words)\n", __LINE__, #x, cap, words); ++bad; } } while (0)

int main() {
    const auto self = std::this_thread::get_id();
    for (int cap : {-1, 0, 1, 2, 3, 4, 9})
        for (size_t words : {size_t(512) * 100, size_t(512) * 128 + 511, size_t(512) * 700 + 3, size_t(512) * 5000 + 9})
            for (int arrays : {1, 2})
                for (bool helps : {false, true}) {
                    double *a = reinterpret_cast<double *>(std::uintptr_t(1) << 40) + 77, *b = a + words + 3000;
                    auto whole = [&](const double *x) { return (std::uintptr_t)(x + words) / 4096 - ((std::uintptr_t)x + 4095) / 4096; };
                    const int most_threads = std::max(0, std::min(cap, kCopyThreads));
                    const bool worth = std::max(whole(a), arrays > 1 ? whole(b) : 0) >= 128;
                    threads.clear(); asked.clear();
                    {
                        Pages pages(cap);
                        EXPECT(!pages.help());
                        pages.ask(a, words, arrays > 1 ? b : nullptr);
                        while (helps && pages.help()) {}
                    }
                    EXPECT((int)threads.size() <= most_threads + helps);
                    EXPECT(helps || !threads.count(self));
                    if (!worth) { EXPECT(asked.empty()); continue; }
                    for (const auto &p : asked) EXPECT(p.second == 1);
                    if (helps) EXPECT(asked.size() == whole(a) + (arrays > 1 ? whole(b) : 0));
                    for (const auto &p : asked) EXPECT((p.first * 4096 >= (std::uintptr_t)a && p.first * 4096 + 4096 <= (std::uintptr_t)(a + words)) || (arrays > 1 && p.first * 4096 >= (std::uintptr_t)b && p.first * 4096 + 4096 <= (std::uintptr_t)(b + words)));
                }
    for (int cap : {1, 2, 3, 4, 6}) { // pages, then copies, as a decryption does it: twice, with what the first round left
        const size_t words = size_t(512) * 4000;
        most = 0; threads.clear();
        {
            Pages pages(std::min(cap, kCopyThreads) - 1);
            for (int i = 0; i < 2; ++i) {
                pages.ask(reinterpret_cast<double *>(std::uintptr_t(1) << 40), words);
                for (int k = 0; k < 3; ++k) pages.help();
                pages.stop();
                EXPECT(at_work == 0);
                in_threads(cap, 4, words, [](size_t, size_t) { work(50); });
                pages.help();
            }
        }
        EXPECT(most <= cap);
    }
    refuse = true;
    asked.clear(); threads.clear();
    int cap = 3; size_t words = size_t(512) * 4000;
    { Pages pages(cap); pages.ask(reinterpret_cast<double *>(std::uintptr_t(1) << 40), words); while (pages.help()) {} }
    EXPECT(asked.empty() && threads.size() <= 4);
    return bad != 0;
}
