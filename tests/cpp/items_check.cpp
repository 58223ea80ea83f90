// Items::point numbers every point of a box once, whatever its shape, and FastDiv is
// the integer division over its whole range: exhaustive over small boxes, random
// divisors and the numerators on both sides of their multiples.
#include <cstdio>
#include <vector>

#include "fhd_items.h"

using namespace fhd;

int main() {
    long bad = 0, points = 0;
    for (int nx = 1; nx < 140; nx += nx < 40 ? 1 : 7)
        for (int ny = 1; ny < 12; ++ny)
            for (int nz = 1; nz < 9; ++nz) {
                const Items t = make_items(nx, ny, nz);
                std::vector<char> seen(t.n, 0);
                for (int q = 0; q < t.n; ++q) {
                    int i, j, k;
                    t.point(q, i, j, k);
                    if (i < 0 || i >= nx || j < 0 || j >= ny || k < 0 || k >= nz || seen[i + nx * (j + ny * k)]++) ++bad;
                    ++points;
                }
            }
    uint64_t x = 88172645463325252ull;
    for (int r = 0; r < 5000000; ++r) {
        x ^= x << 13;
        x ^= x >> 7;
        x ^= x << 17;
        const uint32_t d = (uint32_t)(x >> 40) % (1u << ((x >> 3) % 31)) + 1, q = (uint32_t)(x >> 5) & 0x7fffffffu;
        const FastDiv f = fast_div(d);
        const uint32_t m = q / d * d;
        if (f.div(q) != q / d || f.div(m) != m / d || (m && f.div(m - 1) != (m - 1) / d)) ++bad;
        if (f.div(0x7fffffffu) != 0x7fffffffu / d) ++bad;
    }
    // the largest numerators of the smallest and largest divisors
    for (uint32_t d : {1u, 2u, 3u, 0x40000000u, 0x7ffffffeu, 0x7fffffffu})
        for (uint32_t q : {0u, 1u, 0x7ffffffdu, 0x7ffffffeu, 0x7fffffffu})
            if (fast_div(d).div(q) != q / d) ++bad;
    std::printf("%ld wrong of %ld points and 5000000 divisors\n", bad, points);
    return bad != 0;
}
