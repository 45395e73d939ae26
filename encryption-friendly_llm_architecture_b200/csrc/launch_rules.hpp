// Rules of dispatch that depend on sizes alone.
#pragma once

namespace hb {

// Part sums: up to how many polynomials the masks are streamed once per pair of polynomials (k_prod_parts_few); beyond, and never for one or two parts, they
// are kept (k_prod_parts).  Either kernel works for nothing where its sizes are not filled: the streamed one multiplies 2, 4, 8 or 17 terms, the other has
// six parts a CTA.  Calls with a mask of its own for every product (the same masks for all parts stay in L2 and make streaming look up to 20 %
// quicker), level 7, us, streamed / kept, terms x parts:
//   up to 4 terms   4 x 4, 12 polynomials 382 / 487, 84 2378 / 2368; 4 x 6, 24 0.99 of kept, 48 1.03; 1 x 8, 84 3618 / 3819; 4 x 9, 96 0.95
//   up to 8         8 x 6, 12 0.93, 16 0.97, 24 1.06; 8 x 12, 12 1116 / 1397, 24 0.98, 48 1.04; 5 x 12, 16 0.96, 24 1.02; 5 x 8, 48 0.95, 84 1.01
//   more            9 x 6, 12 913 / 796; 9 x 4, 84 4391 / 2964; 16 x 12, 12 1713 / 1884, 16 1.02, 32 4423 / 3791; 9 x 12, 12 1.02; 16 x 8, 16 0.93, 32 1.06;
//                   9 x 8, 12 0.91, 16 1.02; up to ten polynomials 0.9 to 1.07 in one group of parts
// No call of 12 to 192 polynomials that it streams takes over 1.02 of the time with kept masks; levels 3 and 12 lie within 0.05 of these ratios.
constexpr int streamed_polynomials(int terms, int parts) {
    const int groups = (parts + 5) / 6;
    const bool room = 2 * parts <= 9 * groups; // a quarter or more of the kept kernel's places for parts are empty
    if (terms <= 4) return room ? 96 : 24;
    if (terms <= 8) return groups == 1 ? 12 : room ? 48 : 16;
    if (groups == 1) return 10;
    return terms >= 12 ? (room ? 16 : 12) : room ? 12 : 10;
}

} // namespace hb
