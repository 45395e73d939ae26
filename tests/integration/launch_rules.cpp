// The rules of dispatch against calls that were timed with both kernels: a rule takes none that loses more than a fiftieth.  Prints those that it does.
#include "launch_rules.hpp"

#include <algorithm>
#include <cstdio>

using namespace hb;
static int bad = 0;

struct PartSums { int terms, parts, polys, kept, streamed; }; // us at level 7, a mask of its own for every product
static const PartSums part_sums[] = {
    {4, 4, 12, 487, 382},    {4, 4, 84, 2368, 2378},  {1, 8, 12, 778, 550},     {1, 8, 84, 3819, 3618},   {2, 8, 84, 4047, 3968},   {8, 12, 12, 1397, 1116}, {8, 12, 84, 7107, 7520},
    {8, 17, 16, 2388, 2014}, {8, 7, 48, 3123, 2689},  {9, 6, 12, 796, 913},     {9, 6, 16, 926, 1195},    {9, 3, 84, 2647, 3792},   {9, 4, 84, 2964, 4391},  {9, 4, 32, 1270, 1764},
    {10, 4, 84, 3080, 4513}, {12, 4, 64, 2567, 3685}, {12, 12, 16, 1985, 2133}, {14, 6, 32, 1826, 2581},  {14, 4, 48, 2162, 2973},  {16, 4, 84, 3754, 5439}, {16, 6, 32, 1910, 2702},
    {16, 5, 32, 1746, 2421}, {17, 5, 48, 2580, 3667}, {17, 6, 48, 2826, 4088},  {16, 12, 12, 1884, 1713}, {16, 12, 32, 3791, 4423}, {16, 12, 84, 9129, 11130}, {17, 13, 16, 3011, 2454},
    {17, 17, 48, 8062, 8798},
    {17, 17, 16, 3399, 3067}, {17, 17, 22, 4272, 4162}, {17, 17, 36, 6312, 6669}, {17, 17, 48, 7972, 8783}, {16, 16, 16, 3102, 2894}, {16, 16, 32, 5241, 5617}, {13, 13, 20, 3046, 2853},
    {13, 13, 36, 4822, 5040}, {12, 12, 16, 1979, 2154}, {17, 13, 28, 4585, 4185}, {17, 9, 28, 3134, 3184}, {8, 13, 84, 8667, 8116}, {8, 7, 96, 5899, 5344}, {5, 9, 64, 4054, 4226},
    {8, 3, 16, 610, 556}, {5, 5, 16, 704, 734}, {8, 12, 24, 2266, 2214}, {8, 12, 48, 4168, 4329},
};

struct Call { int units, max_ns, targets, plans, sources; Conversion what; double us[3]; }; // strips, conv_mma with two groups, with four
constexpr Conversion kDigits = Conversion::kDigits, kDigitsOnce = Conversion::kDigitsOnce, kModDown = Conversion::kModDown, kDivision = Conversion::kDivision;
static const Call conversions[] = {
    {18, 3, 7, 1, 3, kDivision, {263.0, 283.7, 266.3}}, {18, 3, 8, 1, 3, kDivision, {285.3, 306.2, 286.4}}, {8, 2, 13, 1, 2, kModDown, {177.4, 189.5, 176.7}},
    {18, 2, 6, 1, 2, kModDown, {160.7, 171.5, 175.1}}, {18, 2, 8, 1, 2, kModDown, {205.8, 218.2, 219.6}}, {8, 3, 12, 1, 3, kDivision, {216.9, 229.1, 212.3}},
    {8, 2, 11, 1, 2, kModDown, {148.0, 156.3, 146.8}}, {24, 2, 6, 1, 2, kModDown, {215.3, 227.2, 237.1}}, {32, 2, 6, 4, 6, kDigits, {155.0, 162.6, 173.8}},
    {60, 2, 8, 5, 8, kDigits, {320.2, 333.9, 366.7}}, {120, 2, 8, 5, 8, kDigits, {610.5, 635.6, 706.8}}, {96, 2, 6, 4, 6, kDigits, {413.3, 430.2, 482.3}},
    {240, 2, 8, 5, 8, kDigits, {1188.5, 1236.3, 1384.3}}, {64, 2, 6, 4, 6, kDigits, {283.8, 294.9, 329.3}}, {192, 2, 6, 4, 6, kDigits, {795.0, 825.8, 939.8}},
    {8, 3, 10, 1, 3, kDivision, {182.0, 188.9, 178.7}}, {40, 2, 8, 5, 8, kDigits, {224.6, 232.2, 252.6}}, {28, 4, 3, 1, 4, kDivision, {194.8, 201.2, 203.0}},
    {240, 2, 9, 5, 9, kDigits, {1302.3, 1343.6, 1502.0}}, {45, 2, 8, 5, 8, kDigits, {247.6, 255.4, 280.5}}, {18, 3, 8, 1, 3, kModDown, {208.4, 214.8, 215.6}},
    {36, 2, 6, 4, 6, kDigits, {170.2, 175.4, 193.6}}, {18, 3, 7, 1, 3, kModDown, {178.7, 184.1, 186.2}}, {336, 2, 13, 7, 13, kDigits, {2425.6, 2497.0, 2727.4}},
    {30, 2, 8, 5, 8, kDigits, {177.7, 182.9, 197.8}}, {120, 2, 9, 5, 9, kDigits, {668.7, 688.2, 764.9}}, {80, 2, 8, 5, 8, kDigits, {422.6, 434.9, 482.6}},
    {60, 2, 9, 5, 9, kDigits, {349.1, 358.9, 394.2}}, {48, 2, 6, 4, 6, kDigits, {223.5, 229.7, 257.5}}, {12, 2, 4, 3, 4, kDigits, {58.4, 56.8, 60.0}},
    {80, 2, 9, 5, 9, kDigits, {462.8, 475.4, 526.4}}, {84, 2, 13, 7, 13, kDigits, {641.6, 658.9, 716.4}}, {4, 4, 6, 2, 6, kDigits, {37.5, 44.7, 34.2}},
    {27, 4, 9, 3, 10, kDigits, {212.5, 201.8, 220.8}}, {48, 4, 10, 3, 11, kDigits, {391.4, 369.7, 403.1}}, {3, 4, 9, 3, 10, kDigits, {43.4, 53.8, 38.9}},
    {96, 4, 12, 4, 13, kDigits, {826.3, 784.0, 851.2}}, {8, 4, 4, 1, 4, kDivision, {81.2, 75.5, 77.9}}, {8, 3, 12, 4, 11, kDigits, {91.0, 83.6, 87.9}},
    {36, 4, 12, 4, 13, kDigits, {329.7, 313.0, 337.8}}, {4, 3, 12, 4, 11, kDigits, {47.9, 63.0, 45.5}}, {8, 4, 1, 1, 4, kDivision, {54.3, 49.3, 53.2}},
    {8, 3, 5, 2, 3, kDigits, {52.8, 46.0, 50.3}}, {8, 2, 3, 1, 2, kDigits, {44.5, 38.9, 41.6}}, {8, 4, 12, 4, 13, kDigits, {94.2, 86.0, 88.5}},
    {72, 4, 10, 3, 11, kDigits, {559.7, 526.6, 581.0}}, {12, 3, 6, 2, 4, kDigits, {82.7, 73.5, 79.1}}, {8, 2, 3, 1, 2, kModDown, {66.0, 59.6, 64.7}},
    {30, 4, 10, 3, 11, kDigits, {257.9, 243.2, 261.3}}, {3, 3, 9, 3, 8, kDigits, {40.8, 51.8, 38.2}}, {12, 4, 10, 3, 11, kDigitsOnce, {262.4, 258.1, 255.2}},
    {8, 2, 8, 1, 2, kModDown, {114.7, 115.0, 113.7}}, {8, 3, 9, 1, 3, kModDown, {231.6, 223.9, 229.4}}, {4, 3, 5, 1, 3, kModDown, {58.1, 66.3, 56.9}},
    {8, 3, 10, 1, 3, kModDown, {134.9, 133.5, 133.2}}, {8, 4, 8, 1, 4, kModDown, {123.7, 121.8, 120.9}}, {8, 3, 7, 1, 3, kModDown, {164.7, 158.2, 161.2}},
    {12, 4, 6, 2, 6, kDigitsOnce, {207.3, 203.9, 206.1}}, {8, 3, 8, 1, 3, kModDown, {116.0, 114.3, 113.3}}, {12, 4, 8, 3, 8, kDigitsOnce, {213.1, 211.6, 212.5}},
    {12, 4, 12, 4, 13, kDigitsOnce, {248.9, 249.9, 244.8}}, {8, 3, 10, 1, 3, kModDown, {247.2, 239.3, 244.4}}, {8, 3, 11, 1, 3, kModDown, {142.1, 141.7, 140.1}},
    {8, 3, 8, 1, 3, kModDown, {215.3, 207.5, 211.7}},
};

struct Switch { int digits, limbs, members; double us[3]; }; // three kernels, one with a member a CTA, with two
static const Switch switches[] = {
    {2, 4, 2, {57.6, 71.4, 71.2}}, {2, 5, 2, {67.7, 79.6, 79.7}}, {3, 6, 1, {64.6, 73.5, 73.5}}, {2, 4, 3, {83.8, 94.0, 93.6}}, {3, 7, 1, {72.3, 80.0, 80.0}},
    {2, 7, 2, {84.9, 91.4, 90.4}}, {2, 4, 9, {144.5, 142.5, 155.3}}, {2, 7, 2, {81.3, 86.4, 85.9}}, {2, 5, 9, {169.4, 168.4, 179.0}}, {2, 8, 2, {86.8, 91.7, 91.9}},
    {2, 5, 3, {93.7, 98.3, 97.4}}, {3, 6, 5, {161.9, 155.4, 169.1}}, {2, 4, 4, {84.7, 88.9, 88.2}}, {2, 10, 3, {135.6, 141.1, 143.5}}, {3, 7, 5, {180.8, 171.2, 188.1}},
    {2, 4, 11, {175.7, 177.8, 182.7}}, {4, 15, 3, {256.5, 236.5, 255.1}}, {4, 9, 3, {174.2, 160.8, 166.6}}, {2, 8, 5, {172.7, 168.6, 171.2}}, {2, 9, 6, {208.3, 206.0, 202.9}},
    {2, 10, 12, {396.6, 400.2, 393.6}}, {3, 12, 2, {132.9, 129.7, 130.3}}, {3, 13, 5, {297.1, 289.7, 300.5}}, {3, 14, 6, {347.1, 347.6, 339.4}}, {4, 15, 12, {785.1, 764.1, 756.0}},
    {2, 10, 1, {68.4, 81.6, 81.6}}, {4, 16, 1, {121.4, 113.4, 113.4}}, {3, 11, 1, {93.2, 90.8, 90.8}}, {2, 10, 17, {531.4, 538.4, 534.8}}, {4, 16, 24, {1540.1, 1510.0, 1494.2}},
};

int main() {
    for (const Switch &c : switches) {
        const bool one = one_kernel_switch(c.digits, c.limbs, c.members);
        const double us = c.us[one ? switch_members(c.members) : 0];
        if (us > c.us[0] * 1.02 || us > 1.05 * std::min({c.us[0], c.us[1], c.us[2]}))
            std::printf("key switch of %d digits, %d limbs, %d members: %.1f us of %.1f / %.1f / %.1f\n", c.digits, c.limbs, c.members, us, c.us[0], c.us[1], c.us[2]), ++bad;
    }
    for (const Call &c : conversions) {
        const StripShape s = conv_shape(c.what, c.units, c.max_ns, c.targets, c.plans, c.sources, true);
        const double us = c.us[s == kMma2 ? 1 : s == kMma4 ? 2 : 0];
        if (us > c.us[0] * 1.02 || us > 1.06 * std::min({c.us[0], c.us[1], c.us[2]}))
            std::printf("%d units of %d plans, %d sources at most, %d targets: shape %d, %.1f us of %.1f / %.1f / %.1f\n", c.units, c.plans, c.max_ns, c.targets, (int)s, us, c.us[0], c.us[1], c.us[2]), ++bad;
        if (const StripShape w = conv_shape(c.what, c.units, c.max_ns, c.targets, c.plans, c.sources, false); w == kMma2 || w == kMma4) std::printf("conv_mma where it must not be\n"), ++bad;
    }
    for (const PartSums &c : part_sums) {
        const bool streamed = c.polys <= streamed_polynomials(c.terms, c.parts);
        if (streamed ? c.streamed > c.kept * 1.02 : c.kept > c.streamed * 1.06)
            std::printf("part sums of %d terms, %d parts, %d polynomials: %s, %d us kept, %d streamed\n", c.terms, c.parts, c.polys, streamed ? "streamed" : "kept", c.kept, c.streamed), ++bad;
    }
    return bad ? 1 : 0;
}
