// Pages: what the memory holds stays, whatever its alignment, length and protection.
#include "host_threads.hpp"

#include <cstdio>
#include <cstdlib>
#include <vector>

int main() {
    int bad = 0;
    for (size_t words : {size_t(0), size_t(1), size_t(511), size_t(512) * 127, size_t(512) * 129 + 5, size_t(512) * 1023, size_t(512) * 4096 + 77})
        for (size_t off : {size_t(0), size_t(1), size_t(2), size_t(300)}) {
            double *p = static_cast<double *>(std::malloc((words + off) * 8 + 8));
            for (size_t i = 0; i < words; i += 97) p[off + i] = (double)i;
            {
                Pages pages(4);
                pages.ask(p + off, words / 2);
                pages.ask(p + off + words / 2, words - words / 2);
                for (size_t i = 1; i < words; i += 97) p[off + i] = -(double)i; // the results arrive meanwhile
            }
            for (size_t i = 0; i < words; i += 97) bad |= p[off + i] != (double)i;
            for (size_t i = 1; i < words; i += 97) bad |= p[off + i] != -(double)i;
            std::free(p);
        }
    void *ro = mmap(nullptr, 1 << 20, PROT_READ, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0); // cannot be populated for writing: left alone
    { Pages pages(1); pages.ask(static_cast<const double *>(ro), (1 << 20) / 8); }
    return bad;
}
