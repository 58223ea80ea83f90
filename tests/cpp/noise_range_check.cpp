// The stress kernel's per-point function over every point of its launch, run on the host:
// the edge noise fields have no ghosts and allocations of their own, so that a fetch
// beyond one of them ends the program (built with the address sanitizer).  Modes: W (the
// flux operator, unpacked, with flux outputs) and A + w B (a step with injected noise,
// packed); the noise of every valid edge has to arrive.
#include <cstdio>
#include <vector>

#include "fhd_kernels.cuh"

using namespace fhd;

namespace {

std::vector<std::vector<double>> store;   // 16-byte aligned by operator new

// a fab of cells (or nodes) -g .. n - 1 + nodal + g, nc components of words of T
template <class T>
Arr4<T> fab(const int n[3], const int (&nodal)[3], int g, int nc, double value) {
    int e[3];
    for (int d = 0; d < 3; ++d) e[d] = n[d] + nodal[d] + 2 * g;
    const size_t values = (size_t)e[0] * e[1] * e[2] * nc * sizeof(T) / sizeof(double);
    store.emplace_back(values, value);
    Arr4<T> a;
    a.sy = e[0];
    a.sz = e[0] * e[1];
    a.sn = e[0] * e[1] * e[2];
    a.p = reinterpret_cast<T*>(store.back().data()) + g * (1 + a.sy + a.sz);
    return a;
}

constexpr int CELL[3] = {0, 0, 0}, ALL[3] = {1, 1, 1};
constexpr int FACE[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
constexpr int EDGE[3][3] = {{1, 1, 0}, {1, 0, 1}, {0, 1, 1}};

template <int NZ, bool PACK, bool AUX>
long run(const int n[3]) {
    constexpr int NS = 2;
    StageArgs<NS, double, NZ, PACK> a{};
    RunParams& P = a.P;
    P.ns = NS;
    P.dim = 3;
    P.volinv = P.dtinv = P.k_B = 1.0;
    for (int d = 0; d < 3; ++d) {
        P.n[d] = n[d];
        P.dx[d] = P.rdx[d] = 1.0;
        a.F.vel[d] = fab<const double>(n, FACE[d], 1, 1, 0.0);
        a.F.mom[d] = fab<const double>(n, FACE[d], 1, 1, 0.0);
        a.noise.a.fa[d] = a.noise.a.fb[d] = fab<const double>(n, FACE[d], 0, NS + 1, 0.0);
        a.noise.a.ea[d] = fab<const double>(n, EDGE[d], 0, 1, 1.0 + d);
        a.noise.a.eb[d] = fab<const double>(n, EDGE[d], 0, 1, 1.0);
        a.noise.a.ca[d] = a.noise.a.cb[d] = fab<const double>(n, CELL, 1, 1, 0.0);
    }
    a.noise.w = 0.5;
    a.F.cons = fab<const double>(n, CELL, 1, 5 + NS, 1.0);
    a.F.pT = 4;
    a.F.pr = fab<const double>(n, CELL, 1, 6 + 2 * NS, 1.0);
    a.mc = fab<double>(n, CELL, 1, 3, 0.0);
    StageAux<AUX> x{};
    if constexpr (AUX) {
        for (int d = 0; d < 3; ++d) x.cf[d] = fab<double>(n, CELL, 1, 1, 0.0);
        const int e[6] = {0, 1, 0, 2, 1, 2};   // edgeflux_x {xy, xz}, _y {xy, yz}, _z {xz, yz}
        for (int q = 0; q < 6; ++q) x.ef[q] = fab<double>(n, EDGE[e[q]], 0, 1, 0.0);
    }
    if constexpr (PACK) {
        const Arr4<double2> r = fab<double2>(n, CELL, 1, RecLayout<NS, double>::NV, 1.0);
        a.F.q = Rec<NS, double>{r.p, r.sy, r.sz, r.sn};
        a.S.ct = fab<double2>(n, CELL, 1, 3, 0.0);
        a.S.et = fab<double2>(n, ALL, 0, 3, 0.0);
        a.S.me = fab<double2>(n, ALL, 0, 3, 0.0);
    } else {
        a.F.eta = a.F.zeta = a.F.kappa = fab<const double>(n, CELL, 1, 1, 1.0);
        a.S.ct = fab<double>(n, CELL, 1, 6, 0.0);
        a.S.et = fab<double>(n, ALL, 0, 6, 0.0);
        a.S.me = fab<double>(n, ALL, 0, 6, 0.0);
    }
    a.it_taus = make_items(n[0] + 2, n[1] + 2, n[2] + 2);
    for (int q = 0; q < a.it_taus.n; ++q) taus_point<NS, double, NZ, false, AUX>(a, q, x);
    // the stochastic stress of a valid edge of a uniform gas: sqrt(2) times its noise
    long bad = 0;
    for (int e = 0; e < 3; ++e) {
        const double w = NZ == NZ_W ? 1.0 + e : 1.5 + e;
        for (int k = 0; k < n[2] + EDGE[e][2]; ++k)
            for (int j = 0; j < n[1] + EDGE[e][1]; ++j)
                for (int i = 0; i < n[0] + EDGE[e][0]; ++i) {
                    double s;
                    if constexpr (PACK) s = a.S.et(i, j, k, e).x;
                    else s = a.S.et(i, j, k, 2 * e);
                    if (!(std::abs(s - std::sqrt(2.0) * w) < 1e-14 * w)) ++bad;
                }
    }
    store.clear();
    return bad;
}

}  // namespace

int main() {
    const int boxes[][3] = {{1, 1, 1}, {5, 4, 3}, {3, 5, 4}, {4, 3, 5}, {8, 8, 8}};
    long bad = 0;
    for (const auto& n : boxes) bad += run<NZ_W, false, true>(n) + run<NZ_AB, true, false>(n) + run<NZ_AB, false, false>(n);
    std::printf("%ld wrong stresses\n", bad);
    return bad != 0;
}
