// Shared memory of the conversions over every geometry a context may have: where the launch rules count on two CTAs of four-column strips (any
// number of sources) or of eight-column strips (up to four sources) per SM, two fit, and one of any shape fits a CTA.  Prints what does not.
#include "conv_shared.hpp"

#include <algorithm>
#include <cstdio>

using namespace hb;
static int bad = 0;
static void check(const char *what, std::size_t bytes, int ctas, int sources, int targets) {
    const std::size_t sm = 228 * 1024, cta = 227 * 1024, fixed = 1024 + 128; // what the system keeps per CTA, and static variables
    if (bytes + 128 > cta || ctas * (bytes + fixed) > sm) { std::printf("%s: %d sources, %d targets: %zu bytes, %d CTAs\n", what, sources, targets, bytes, ctas); ++bad; }
}

int main() {
    for (int special = 1; special <= 8; ++special)
        for (int alpha = 1; alpha <= 8; ++alpha)
            for (int limbs = 2; limbs + special <= 32; ++limbs) {
                auto conversion = [&](int sources, std::size_t consts, int targets) {
                    check("4 x 4", strip_bytes(4, sources + 4) + consts, 2, sources, targets);
                    check("4 x 8", strip_bytes(4, sources + 8) + consts, 1, sources, targets);
                    if (sources <= 4) check("8 x 2", strip_bytes(8, sources + 2) + consts, 2, sources, targets);
                    else check("8 x 4", strip_bytes(8, sources + 4) + consts, 1, sources, targets);
                };
                const int own = std::min(alpha, limbs);
                std::size_t digits = 0; // the largest of the digits of one level, of which the last may be short
                for (int n = 1; n <= own; ++n) digits = std::max(digits, conv_const_bytes(n, limbs + special - n));
                conversion(own, std::max(digits, conv_const_bytes(own, limbs + special - own)), limbs + special - own);
                conversion(special, conv_const_bytes(special, limbs), limbs);
                if (special < 8) conversion(special + 1, conv_const_bytes(special + 1, limbs - 1), limbs - 1);
            }
    return bad ? 1 : 0;
}
