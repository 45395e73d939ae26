// in_threads while allocations fail: every element is worked on once, whichever of the threads cannot be started for want of memory.
#include "host_threads.hpp"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

static std::atomic<int> allowed{1 << 30}; // allocations that still succeed
void *operator new(std::size_t n) {
    if (allowed.fetch_sub(1) <= 0) throw std::bad_alloc();
    if (void *p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

int main() {
    int bad = 0;
    for (int cap : {1, 2, 4, 9})
        for (size_t n : {0, 1, 3, 4, 1000})
            for (size_t words : {size_t(0), size_t(1) << 16, size_t(1) << 20})
                for (int fail_at = 0; fail_at < 5; ++fail_at) {
                    std::vector<std::atomic<int>> seen(n);
                    allowed = fail_at;
                    in_threads(cap, n, words, [&](size_t a, size_t b) { for (; a < b; ++a) ++seen[a]; });
                    allowed = 1 << 30;
                    for (size_t i = 0; i < n; ++i)
                        if (seen[i] != 1) { std::printf("cap %d, %zu of %zu, %zu words, %d allocations: %d times\n", cap, i, n, words, fail_at, (int)seen[i]); bad = 1; }
                }
    return bad;
}
