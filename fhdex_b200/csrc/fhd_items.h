// fhd_items.h — work items of a kernel as points of a box.  Plain C++ on the host (the
// CPU test runs this same code).
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define FHD_ITEMS_HD __host__ __device__ __forceinline__
#else
#define FHD_ITEMS_HD inline
#endif

namespace fhd {

// Division of a 31-bit item number by a run constant: q / d = (q * m) >> s with
// m = floor(2^(31+l) / d) + 1, l = ceil(log2 d), s = 31 + l (Granlund and Montgomery,
// "Division by invariant integers using multiplication", PLDI 1994: exact for
// 0 <= q < 2^31, as m*d - 2^(31+l) lies in (0, 2^l]).  Three instructions against
// about twenty for a division by a value the compiler does not know.
struct FastDiv {
    uint32_t m, s;
    FHD_ITEMS_HD uint32_t div(uint32_t q) const { return (uint32_t)(((uint64_t)q * m) >> s); }
};
inline FastDiv fast_div(uint32_t d) {
    uint32_t l = 0;
    while (((uint64_t)1 << l) < d) ++l;
    FastDiv f;
    f.m = (uint32_t)((((uint64_t)1 << (31 + l)) / d) + 1);
    f.s = 31 + l;
    return f;
}

// Items 0 .. nx*ny*nz - 1 of a box as points, x fastest.  (Numbering patches of 32 points
// by four rows, so that a block finds the row below in L1, was measured slower: 25.3
// against 24.4 ms per step at 256^3 argon FP64.)
struct Items {
    int nx, nxy, n;      // row, plane, all points (below 2^31)
    FastDiv dx, dxy;
    FHD_ITEMS_HD void point(int q, int& i, int& j, int& k) const {
        k = (int)dxy.div((uint32_t)q);
        const int r = q - k * nxy;
        j = (int)dx.div((uint32_t)r);
        i = r - j * nx;
    }
};
inline Items make_items(int nx, int ny, int nz) {
    Items t;
    t.nx = nx;
    t.nxy = nx * ny;
    t.n = nx * ny * nz;
    t.dx = fast_div((uint32_t)nx);
    t.dxy = fast_div((uint32_t)(nx * ny));
    return t;
}

// Whether 32-bit offsets (component or word times stride, plus the point) reach every
// element of a field of n cells grown by g, with comps components or words per cell.
inline bool offsets_fit(const int n[3], int g, int comps) {
    int64_t e = comps;
    for (int d = 0; d < 3; ++d) {
        e *= n[d] + 2 * (int64_t)g;
        if (e > (int64_t)INT32_MAX + 1) return false;
    }
    return true;
}

}  // namespace fhd
