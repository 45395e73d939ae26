// The twiddle values of a context: powers of psi and of its inverse at the bit-reversed slots, and nothing besides (which companions a transform
// multiplies by depends on the ring and on the prime, so they are made where the tables are).  Returns 0 when they are.
#include "host_ctx.hpp"

#include <cstdio>

int main() {
    const hbhost::HostParams prm{12, 3, 2, 3, 60, 42, 60, 32, 3.2, {1, 2, 3, 4}};
    const hbhost::HostCtx h(prm);
    int bad = 0;
    for (int i = 0; i < h.nprimes; ++i) {
        std::vector<hbhost::u64> f, iv;
        h.twiddles(i, f, iv);
        if (f.size() != (size_t)h.N || iv.size() != f.size()) { ++bad; continue; }
        for (int k = 0; k < h.N; k += 37) {
            unsigned slot = 0;
            for (int b = 0; b < h.logn; ++b) slot |= (unsigned)(k >> b & 1) << (h.logn - 1 - b);
            if (f[slot] != hbhost::powmod(h.psi_root[(size_t)i], (hbhost::u64)k, h.q[(size_t)i]) || hbhost::mulmod(f[slot], iv[slot], h.q[(size_t)i]) != 1) ++bad;
        }
    }
    std::printf("%d wrong\n", bad);
    return bad ? 1 : 0;
}
