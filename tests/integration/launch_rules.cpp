// The rules of dispatch against calls that were timed with both kernels: a rule takes none that loses more than a fiftieth.  Prints those that it does.
#include "launch_rules.hpp"

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
};

int main() {
    for (const PartSums &c : part_sums) {
        const bool streamed = c.polys <= streamed_polynomials(c.terms, c.parts);
        if (streamed ? c.streamed > c.kept * 1.02 : c.kept > c.streamed * 1.25)
            std::printf("part sums of %d terms, %d parts, %d polynomials: %s, %d us kept, %d streamed\n", c.terms, c.parts, c.polys, streamed ? "streamed" : "kept", c.kept, c.streamed), ++bad;
    }
    return bad ? 1 : 0;
}
