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
    // offsets_fit against the last element's offset, at sizes around the line (16 words of a
    // four-species cell record: 510^3 the largest cube, whose 14 components of prim fit too)
    for (int s : {500, 509, 510, 511, 512, 520})
        for (int comps : {4, 7, 14, 16})
            for (int g : {0, 1, 2}) {
                const int n[3] = {s, s, s};
                const uint64_t e = s + 2 * g, last = e * e * e * comps - 1;
                if (offsets_fit(n, g, comps) != (last <= 0x7fffffffull)) ++bad;
            }
    const int big[3] = {1 << 30, 1 << 30, 1 << 30}, c510[3] = {510, 510, 510}, c511[3] = {511, 511, 511};
    if (offsets_fit(big, 0, 1) || !offsets_fit(c510, 1, 16) || offsets_fit(c511, 1, 16) || !offsets_fit(c511, 2, 14)) ++bad;
    std::printf("%ld wrong of %ld points and 5000000 divisors\n", bad, points);
    return bad != 0;
}
