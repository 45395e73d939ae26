// Rules of dispatch that depend on sizes alone.
#pragma once

namespace hb {

// Strip width and groups of a launch over `units` (polynomial, conversion) pairs.  At most two units: narrow strips and many groups, so that
// all sources and all targets of a unit are worked on at once.  Up to twelve: narrow strips, two CTAs per SM, for the last wave.
// Beyond: strips of eight columns (64-byte runs) and two groups, two CTAs per SM, whose barriers and loads cover each other, as long as their
// strips fit (four sources); otherwise four groups and one CTA.  Calls, us, (4 x 8) / (4 x 4) / (8 x 2): decompositions of level 7, 2 units 47 / 45 / 58,
// divisions 53 / 59 / 62, 4 units 88 / 81 / 94, 10 units 175 / 163 / 171, 18 units 279 / 260 / 256, 40 units 594 / 546 / 533; decompositions of level 2, 17
// units 111 / 92 / 83, of level 12, 24 units 280 / 260 / 254.  Launches, us, (8 x 4) / (8 x 2): 192 polynomials of the division at level 6 696 / 604,
// the conversions of 256 products at level 8 3174 / 2719 and 2079 / 1797.
// The wide strips lose where few SMs have one CTA more than the others: 15, 16, 19 and 20 units leave a tenth to a half of the SMs with it,
// and a CTA with four sources and many targets is long.  Calls, us, (4 x 4) / (8 x 2): divisions of level 7, 16 units 234 / 238, 20 units 289 / 293, of
// level 6 169 / 171 and 206 / 208.  Up to five targets it does not show (divisions of level 5, 16 units 157 / 155, 20 units 190 / 188), nor with the
// three sources of a ModDown (level 7, 206 / 205 and 253 / 252); decompositions of level 12 go either way (179 / 180 and 222 / 221).
// The line at twelve was drawn when the narrow strips were ahead up to there; now (8 x 2) is from seven units on, except at 10, 14, 16 and 20 of the
// division (decompositions of level 2, 8 units 56 / 51; divisions of level 3, 8 units 84 / 76, of level 7, 8 units 134 / 131, 14 units 216 / 219).
// More than four sources, (4 x 4) / (8 x 4): divisions of seven sources 32 units 425 / 434, 40 units 520 / 536; of eight 48 units 1120 / 1140;
// a digit of seven limbs 40 units 425 / 411.
//
// mma: up to four sources, primes of LongPm, and two CTAs find room with their constants (conv_mma).  Its strips have eight columns, so few units fill the GPU
// badly: two groups and two CTAs per SM hold nine units at once, four groups and one CTA four and a half; a group without a target waits for the
// others, and with two sources there is little to multiply.  Digits of several plans even out, a single conversion does not: there the number of its targets
// decides; and it matters what runs before and after.  Calls, us, the strips / conv_mma with two groups / with four:
//   3, 4 units       decompositions of level 8, one member 40 / 51 / 37; divisions of level 7 75 / 87 / 73, of level 5 (five targets fill the second round of
//                    four groups with one) 52.0 / 61.1 / 53.0
//   5, 6             decompositions of level 6 53 / 52 / 54, hoisted rotations with their ModDown of level 8 101 / 107 / 107
//   7 to 9           decompositions of level 12 89 / 83 / 85; divisions of level 1 54 / 49 / 53, of level 12 188 / 193 / 182; rotations with their ModDown of
//                    level 8 0.97 / 0.99 of the strips, of level 12 1.02 / 0.99
//   12               decompositions of level 12 137 / 124 / 131, as part of a rotation (ks_rows follows) 1.00 / 0.98 of the strips; divisions of level 4
//                    111 / 108 / 109, of level 12 275 / 288 / 267
//   17, 18           decompositions of level 8 136 / 131 / 144; divisions of level 8 275 / 269 / 260; ModDowns of level 7 208 / 215 / 216
//   from 24          decompositions of level 12, 48 units 436 / 420 / 451, of level 3 (two sources on average) 148 / 151 / 167; divisions of level 8, 96 units
//                    1313 / 1288 / 1336, of level 3, 28 units 195 / 201 / 203; ModDowns of level 8, 96 units 1068 / 1059 / 1133, of level 5, 24 units 218 / 222 / 234
//   two sources      (six or seven digits) decompositions of level 7, 120 units 611 / 636 / 707, 9 units at level 3 45 / 42 / 45
// Over all levels, 1 to 48 members and contexts of two to four sources no call takes over 1.02 of the time with the strips.
enum StripShape { kStrip8x1, kStrip8x2, kStrip8x4, kStrip4x4, kStrip4x8, kMma2, kMma4 };
enum class Conversion { kDigits, kDigitsOnce, kModDown, kDivision }; // kDigitsOnce: of digits that go to ks_rows; kDivision: by P and a prime of Q
// `plans` conversions of at most max_ns sources, `sources` in all, and `targets` each on average, for units / plans polynomials
constexpr StripShape conv_shape(Conversion what, int units, int max_ns, int targets, int plans, int sources, bool mma) {
    if (mma) {
        const bool one = plans == 1, division = what == Conversion::kDivision, down = what == Conversion::kModDown;
        if ((units == 3 || units == 4) && !(division && targets == 5)) return kMma4;
        if (units >= 7 && units <= 9) return (division && targets >= 7) || (down && targets >= (max_ns >= 3 ? 12 : 9)) ? kMma4 : kMma2;
        if (units == 12) return ((division || down) && targets >= 5) || (what == Conversion::kDigitsOnce && targets >= 6) ? kMma4 : kMma2;
        if (max_ns >= 3 && (units >= 24 || ((units == 17 || units == 18) && !(one && max_ns == 3))) &&
            (one ? targets >= (max_ns == 3 ? 7 : 4) : targets >= 6 || 2 * sources >= 5 * plans))
            return kMma2;
    }
    if (units <= 2) return kStrip4x8;
    if (units <= 12) return kStrip4x4;
    if (max_ns > 4) return units <= 32 ? kStrip4x4 : kStrip8x4;
    const int more = units * 32 % 148; // SMs with one CTA more
    return units <= 20 && max_ns == 4 && targets > 5 && more >= 148 / 10 && more < 148 / 2 ? kStrip4x4 : kStrip8x2;
}

// Key switches of digits used once, with limbs of Q and P together: whether their row passes and inner products go through one kernel (ks_rows), and the
// members a CTA takes there.  Rotations, us, three kernels / ks_rows with one member a CTA / with two:
//   one member      level 12 (four digits) 121 / 113, level 7 (three) 93 / 91, level 6 (two) 68 / 82; three digits of six limbs in all 65 / 74
//   two digits      level 6, 2 members 98 / 102 / 104, 3 members 136 / 141 / 144, 12 members 397 / 400 / 394, 17 members 531 / 538 / 535; five limbs in all, 2 members 68 / 80 / 80
//   three, four     level 12, 2 members 190 / 172 / 171, 24 members 1540 / 1510 / 1494; level 8, 12 members 556 / 561 / 546; level 7, 5 members 254 / 251 / 260
// Over contexts of two to seven digits and 1 to 33 members no rotation takes over 1.03 of the time with three kernels.
constexpr bool one_kernel_switch(int digits, int limbs, int members) {
    if (digits < 2 || digits > 4) return false; // more do not fit the registers
    if (digits == 2) return limbs >= 7 && members >= 4 && members % 2 == 0;
    return members > 1 || digits * limbs >= 30;
}
constexpr int switch_members(int batch) { return batch >= 4 && (batch % 2 == 0 || batch > 8) ? 2 : 1; } // an odd one leaves half a CTA without work

// Part sums: up to how many polynomials the masks are streamed once per pair of polynomials (k_prod_parts_few); beyond, and never for one or two parts, they
// are kept (k_prod_parts).  Either kernel works for nothing where its sizes are not filled: the streamed one multiplies 2, 4, 8 or 17 terms, the other has
// six parts a CTA; from nine terms on the line goes by the products of either.  Calls with a mask of its own for every product (the same masks for all parts
// stay in L2 and make streaming look up to 20 % quicker; absent masks change nothing), streamed / kept at level 7, us or ratio, terms x parts:
//   up to 4 terms   4 x 4, 12 polynomials 382 / 487, 84 2378 / 2368; 4 x 6, 24 0.99, 48 1.03; 1 x 8, 84 3618 / 3819; 4 x 9, 96 0.95
//   up to 8         8 x 6, 12 0.93, 16 0.97, 24 1.06; 5 x 4, 16 1.01; 8 x 12, 12 1116 / 1397, 24 0.98, 48 1.04; 5 x 12, 24 1.02; 5 x 8, 48 1.00, 84 1.01;
//                   8 x 13, 84 0.94; 8 x 7, 96 0.91; 5 x 9, 48 1.04
//   more            9 x 6, 12 913 / 796; 9 x 4, 84 4391 / 2964; 9 x 8, 12 0.91, 16 1.02; 12 x 12, 12 0.98, 14 1.04; 16 x 8, 16 0.93, 24 1.01; 16 x 12, 12 1713 / 1884,
//                   16 1.02, 32 4423 / 3791; 13 x 13, 22 0.97, 28 1.00; 16 x 16, 22 1.01, 24 1.02; 17 x 17, 16 0.90, 24 0.99, 36 1.06, 48 1.10; up to ten
//                   polynomials 0.9 to 1.07 in one group of parts
// Over 2200 calls at levels 3 to 12, 12 to 192 polynomials, none that it streams takes over 1.025 of the time with kept masks; all together take 1.002 of what the
// quicker kernel of each call would.
constexpr int streamed_polynomials(int terms, int parts) {
    const int groups = (parts + 5) / 6, empty = 6 * groups - parts; // empty: places for parts that the kept kernel has and does not need
    if (terms <= 4) return 2 * empty >= 3 * groups ? 96 : 24;
    if (terms <= 8) {
        if (groups == 1) return parts <= 4 ? 16 : 12;
        return 2 * empty >= 5 * groups ? 96 : 3 * empty >= 5 * groups ? 12 * terms : 2 * empty >= 3 * groups ? 48 : 24;
    }
    const int line = groups == 1 ? 10 : (groups == 2 ? 16 : 22) * 6 * groups * terms / (17 * parts);
    return line > 10 ? line : 10;
}

} // namespace hb
