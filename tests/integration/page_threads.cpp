// Pages over a stand-in for the system call: no more threads than the cap, over all calls; each page of one array or of two is asked for once; running() counts
// the threads at work, so that copies beside them stay within a budget.  Prints what fails; 0 when nothing does.
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
    for (int cap : {-1, 0, 1, 2, 3, 4, 9})
        for (size_t words : {size_t(512) * 100, size_t(512) * 128 + 511, size_t(512) * 700 + 3, size_t(512) * 5000 + 9})
            for (int arrays : {1, 2, 3}) { // three: a call for two and a second call
                double *a = reinterpret_cast<double *>(std::uintptr_t(1) << 40) + 77, *b = a + words + 3000, *c = b + words + 3000;
                threads.clear(); asked.clear();
                {
                    Pages pages(cap);
                    pages.ask(a, words, arrays > 1 ? b : nullptr);
                    if (arrays > 2) pages.ask(c, words);
                    EXPECT(pages.running() >= 0 && pages.running() <= std::max(0, std::min(cap, kCopyThreads)));
                }
                EXPECT((int)threads.size() <= std::max(0, std::min(cap, kCopyThreads)));
                auto whole = [&](const double *x) { return (std::uintptr_t)(x + words) / 4096 - ((std::uintptr_t)x + 4095) / 4096; };
                const bool first_call = cap > 0 && std::max(whole(a), arrays > 1 ? whole(b) : 0) >= 128, any = first_call || (cap > 0 && arrays > 2 && whole(c) >= 128);
                EXPECT(threads.empty() == !any);
                for (const auto &p : asked) EXPECT(p.second == 1);
                if (first_call)
                    for (int i = 0; i < std::min(arrays, 2); ++i) {
                        const std::uintptr_t first = ((std::uintptr_t)(i ? b : a) + 4095) / 4096, last = (std::uintptr_t)((i ? b : a) + words) / 4096;
                        for (std::uintptr_t p = first; p < last; ++p) EXPECT(asked.count(p));
                    }
                size_t inside = 0;
                for (int i = 0; i < arrays; ++i) inside += whole(i == 0 ? a : i == 1 ? b : c);
                EXPECT(asked.size() <= inside);
            }
    for (int cap : {1, 2, 3, 4, 6}) { // pages and copies together, as a decryption does it
        const size_t words = size_t(512) * 4000;
        most = 0;
        {
            Pages pages(std::min(cap, kCopyThreads) - 1);
            pages.ask(reinterpret_cast<double *>(std::uintptr_t(1) << 40), words);
            for (int i = 0; i < 40; ++i) in_threads(cap - pages.running(), 4, words, [](size_t, size_t) { work(50); });
        }
        EXPECT(most <= cap);
    }
    refuse = true;
    threads.clear();
    int cap = 3; size_t words = size_t(512) * 4000;
    { Pages pages(cap); pages.ask(reinterpret_cast<double *>(std::uintptr_t(1) << 40), words); for (int i = 0; i < 2000 && pages.running(); ++i) std::this_thread::sleep_for(std::chrono::milliseconds(1)); EXPECT(pages.running() == 0); }
    return bad != 0;
}
