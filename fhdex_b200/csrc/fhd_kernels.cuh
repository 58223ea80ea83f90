// fhd_kernels.cuh — sm_100a kernels of the staggered RK3 step.
//
//   k_cellprep  per stage: conservedToPrimitiveStag + calculateTransportCoeffs for
//               every cell once (cells grown by 1, face velocities grown by 1)
//   k_taus      per stage: stochastic + deterministic stresses on cells and edges
//               (k_taus_staged: small boxes)
//   k_faces     per stage: stochastic + diffusive + hyperbolic conservative face
//               fluxes of the three directions
//   k_update    per stage: flux divergence, momentum update and the SSP-RK3
//               combination, with the results' periodic ghosts (k_update_split: the
//               smallest boxes)
//   k_convert   end of step / drop-in conversion (prim, vel, cons 1..3)
//   k_ghosts    periodic FillBoundary of several fabs in one launch
//   k_transport, k_aux_*  drop-in operators (transport coefficients, flux MultiFabs)
//   k_noise_*   Philox noise fills;  k_init_uniform  InitConsVarStag prob_type 1
#pragma once
#include "fhd_flux.cuh"
#include "fhd_transport_alt.cuh"

namespace fhd {

// Every kernel here has internal linkage (static): the FP64 and the mixed units both
// instantiate the kernels that do not depend on the precision (e.g. k_convert_b<NS>)
// under the same name.  With external linkage a launch could reach the other unit's
// device code, and which one depends on the order the modules are loaded in.

enum { ST_OK = 0, ST_MASSFRAC = 2, ST_NONFINITE = 3, ST_TIMEOUT = 5 };

FHD_D void flag(int* status, int code) {
    if (status) atomicCAS(status, 0, code);
}

// ===================================================================================
// cellprep: U^s -> (T, p, Y, X), coefficients, face velocities
// ===================================================================================
template <int NS, class R>
struct alignas(16) PrepArgs {
    DevParams P;
    Arr4<const double> cons;
    Arr4<const double> mom[3];
    Arr4<double> vel[3];
    Arr4<double> pr;   // view starting at the T component: T, p, Y[NS], X[NS]
    Arr4<R> eta, zeta, kappa, chi, D;
    // packed pipeline: the cell records, else q null; which of prim (1: p, 2: T, p, Y, X)
    // and whether the coefficient fields are written
    Vec<R>* q;
    int qsy, qsz, qsn;
    int prim, coef;
    Items it;          // cells [-1, n + 1]^3
    int* status;
};

template <int NS, class R>
FHD_D int cellprep_count(const PrepArgs<NS, R>& a) { return a.it.n; }

template <int NS, class R>
FHD_D void cellprep_point(const PrepArgs<NS, R>& a, int q) {
    const DevParams& P = a.P;
    int i, j, k;
    a.it.point(q, i, j, k);
    --i; --j; --k;
    const double rho = a.cons(i, j, k, 0);
    // low face velocities (conservedPrimitiveConversionsStag.cpp:61-67)
    a.vel[0](i, j, k) = 2 * a.mom[0](i, j, k) / (rho + a.cons(i - 1, j, k, 0));
    a.vel[1](i, j, k) = 2 * a.mom[1](i, j, k) / (rho + a.cons(i, j - 1, k, 0));
    a.vel[2](i, j, k) = 2 * a.mom[2](i, j, k) / (rho + a.cons(i, j, k - 1, 0));
    if (i > P.n[0] || j > P.n[1] || k > P.n[2]) return;
    double rY[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) rY[n] = a.cons(i, j, k, 5 + n);
    Prim<NS> q2;
    const bool fin = cons_to_prim<NS>(P, rho, a.cons(i, j, k, 4), rY, a.mom[0](i, j, k), a.mom[0](i + 1, j, k),
                                      a.mom[1](i, j, k), a.mom[1](i, j + 1, k), a.mom[2](i, j, k),
                                      a.mom[2](i, j, k + 1), q2);
    if (!fin) flag(a.status, ST_NONFINITE);
    if (a.prim) a.pr(i, j, k, 1) = q2.p;
    if (a.prim > 1) {
        a.pr(i, j, k, 0) = q2.T;
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            a.pr(i, j, k, 2 + n) = q2.Y[n];
            a.pr(i, j, k, 2 + NS + n) = q2.X[n];
        }
    }
    R Yr[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) Yr[n] = R(q2.Y[n]);
    // The cell record, each word as soon as its components are known (the ones of Y and
    // X alone before the transport model: fewer values live through it)
    using L = RecLayout<NS, R>;
    R v[L::NV * L::V];
    Vec<R>* const o = a.q + (i + j * a.qsy + k * a.qsz);
    auto early = [](int w) { return NS > 1 && w * L::V >= L::Y && (w + 1) * L::V <= L::CHI; };
    if constexpr (NS > 1) {
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            v[L::Y + n] = R(q2.Y[n]);
            v[L::X + n] = R(q2.X[n]);
        }
#pragma unroll
        for (int w = 0; w < L::NV; ++w)
            if (early(w) && a.q) o[w * a.qsn] = vmake(v + w * L::V);
    }
    Coeffs<NS, R> c;
    if (!transport_gio<NS, R>(P, R(rho), R(q2.T), R(q2.p), Yr, c)) flag(a.status, ST_MASSFRAC);
    if (a.q) {
        v[L::T] = R(q2.T);
        v[L::ETA] = c.eta;
        v[L::KAPPA] = c.kappa;
        v[L::PR] = R(q2.p);
        if constexpr (NS > 1) {
#pragma unroll
            for (int n = 0; n < NS; ++n) v[L::CHI + n] = c.chi[n];
#pragma unroll
            for (int n = 0; n < NS * NS; ++n) v[L::D + n] = c.D[n];
        }
#pragma unroll
        for (int n = L::N; n < L::NV * L::V; ++n) v[n] = R(0.);
#pragma unroll
        for (int w = 0; w < L::NV; ++w)
            if (!early(w)) o[w * a.qsn] = vmake(v + w * L::V);
    }
    if (!a.coef) return;
    a.eta(i, j, k) = c.eta;
    a.kappa(i, j, k) = c.kappa;
    a.zeta(i, j, k) = c.zeta;
#pragma unroll
    for (int n = 0; n < NS; ++n) a.chi(i, j, k, n) = c.chi[n];
#pragma unroll
    for (int n = 0; n < NS * NS; ++n) a.D(i, j, k, n) = c.D[n];
}

// Register cap of the cell kernel: 64 registers up to two species (8 blocks of
// 128, no spills); with three or four species the Giovangigli solves need ~164
// registers in FP64 and ~93 in FP32, so cap at 128 (4 blocks, 40 B of spills in
// FP64) and 80 (6 blocks, no spills) to raise occupancy.
template <int NS, class R>
constexpr int cellprep_min_blocks() { return NS <= 2 ? 8 : (sizeof(R) == 8 ? 4 : 6); }

template <int NS, class R>
static __global__ void __launch_bounds__(128, cellprep_min_blocks<NS, R>()) k_cellprep(PrepArgs<NS, R> a) {
    const int tot = cellprep_count(a);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += gridDim.x * blockDim.x) cellprep_point(a, q);
}

// centre momentum flux with the particle reservoir's rule: a ghost cell beyond a
// bc_mass 4 side of direction d takes the stochastic and diffusive part of the cell
// inside it (recomputed here with that cell's own noise)
template <int NS, class R, int NZ, bool WL, class FT>
FHD_D double cen_total_res(const RunParams& P, const FT& F, const Noise<NZ>& nz, const CellTaus<R>& t,
                           int d, int i, int j, int k) {
    if constexpr (WL) {
        const int x = d == 0 ? i : (d == 1 ? j : k);
        const int side = x < 0 ? 2 * d : (x > P.n[d] - 1 ? 2 * d + 1 : -1);
        if (side >= 0 && P.bc_mass[side] == 4) {
            int c[3] = {i, j, k};
            c[d] += (side & 1) ? -1 : 1;
            const CellTaus<R> tin = cell_taus<NS, R, NZ, WL>(P, F, nz, c[0], c[1], c[2]);
            return cen_total<NS, R, WL>(P, F, t, d, i, j, k, &tin);
        }
    }
    return cen_total<NS, R, WL>(P, F, t, d, i, j, k);
}

// ===================================================================================
// stage pipeline: k_taus -> k_faces -> k_update
// ===================================================================================
// Scratch of one stage (owned by the context):
//   ct: cell stresses on the cells grown by 1, comps 0-2 stochastic xx,yy,zz,
//       3-5 deterministic xx,yy,zz
//   et: edge stresses on the points [0, n]^3, comps (s,d) of xy, xz, yz at 0-1, 2-3, 4-5
//   ff[d]: conservative face fluxes (rho, rhoE, rhoY) of direction d on [0, n]^3
//   mc: total centre momentum fluxes (cenflux x, y, z) on the cells grown by 1
//   me: total edge momentum fluxes on [0, n]^3 in the reference's order
//       edgeflux_x[0..1], edgeflux_y[0..1], edgeflux_z[0..1]
// PACK (periodic boxes): the same values in words of two; ct and et hold (s, d), me the
// two totals of edge E (edgey_u, edgex_v; edgez_u, edgex_w; edgez_v, edgey_w), ff
// (rho, rhoE), (rhoY_0, rhoY_1), ... with a last odd component by itself (fl).
template <int NS, class R, bool PACK>
struct StageScratch {
    Arr4<R> ct, et;
    Arr4<double> ff[3], me;
    FHD_D void put_ct(int i, int j, int k, int d, R s, R dd) const {
        ct(i, j, k, d) = s;
        ct(i, j, k, 3 + d) = dd;
    }
    FHD_D void put_et(int E, int i, int j, int k, const Taus<R>& t) const {
        et(i, j, k, 2 * E) = t.s;
        et(i, j, k, 2 * E + 1) = t.d;
    }
    // component of edgeflux_x[0..1], _y, _z that total q of edge E is
    static FHD_D int me_comp(int E, int q) { return q == 0 ? (E == 0 ? 2 : (E == 1 ? 4 : 5)) : (E == 0 ? 0 : (E == 1 ? 1 : 3)); }
    FHD_D bool has_me() const { return me.p != nullptr; }
    FHD_D void put_me(int E, int i, int j, int k, double va, double vb) const {
        me(i, j, k, me_comp(E, 0)) = va;
        me(i, j, k, me_comp(E, 1)) = vb;
    }
    FHD_D double get_me(int E, int q, int i, int j, int k) const { return me(i, j, k, me_comp(E, q)); }
    FHD_D bool has_ff(int d) const { return ff[d].p != nullptr; }
    FHD_D void put_ff(int d, int i, int j, int k, const double (&f)[2 + NS]) const {
#pragma unroll
        for (int c = 0; c < 2 + NS; ++c) ff[d](i, j, k, c) = f[c];
    }
    // Fluxes in words: word w holds components cw .. cw + n - 1 (n = 1, PACK 2); their
    // differences of the faces above and below (i, j, k) in direction d
    static constexpr int NW = 2 + NS;
    static FHD_D int first(int w) { return w; }
    static FHD_D int count(int) { return 1; }
    FHD_D void ff_diff(int w, int d, int i, int j, int k, double (&f)[2]) const {
        f[0] = ff[d](i + (d == 0), j + (d == 1), k + (d == 2), w) - ff[d](i, j, k, w);
    }
};
template <int NS, class R>
struct StageScratch<NS, R, true> {
    static constexpr int NP = (2 + NS) / 2;     // whole words of a face's fluxes
    Arr4<Pair<R>> ct, et;
    Arr4<double2> ff[3], me;
    Arr4<double> fl[3];
    FHD_D void put_ct(int i, int j, int k, int d, R s, R dd) const { ct(i, j, k, d) = pmake(s, dd); }
    FHD_D void put_et(int E, int i, int j, int k, const Taus<R>& t) const { et(i, j, k, E) = pmake(t.s, t.d); }
    FHD_D bool has_me() const { return true; }
    FHD_D void put_me(int E, int i, int j, int k, double va, double vb) const { me(i, j, k, E) = make_double2(va, vb); }
    FHD_D double get_me(int E, int q, int i, int j, int k) const {
        const double2& v = me(i, j, k, E);
        return q ? v.y : v.x;
    }
    FHD_D bool has_ff(int) const { return true; }
    FHD_D void put_ff(int d, int i, int j, int k, const double (&f)[2 + NS]) const {
#pragma unroll
        for (int c = 0; c < NP; ++c) ff[d](i, j, k, c) = make_double2(f[2 * c], f[2 * c + 1]);
        if constexpr (NS % 2) fl[d](i, j, k) = f[1 + NS];
    }
    static constexpr int NW = NP + NS % 2;
    static FHD_D int first(int w) { return 2 * w; }
    static FHD_D int count(int w) { return w < NP ? 2 : 1; }
    FHD_D void ff_diff(int w, int d, int i, int j, int k, double (&f)[2]) const {
        const int ip = i + (d == 0), jp = j + (d == 1), kp = k + (d == 2);
        if (w < NP) {
            const double2 h = ff[d](ip, jp, kp, w), l = ff[d](i, j, k, w);
            f[0] = h.x - l.x;
            f[1] = h.y - l.y;
        } else {
            f[0] = fl[d](ip, jp, kp) - fl[d](i, j, k);
        }
    }
};

// What the face kernel reads, as one pointer per component at point (0,0,0) of its
// fab and the strides of the fabs: an operand is then pointer + offset, with the
// offset shared by the components of a fab.  FaceDir: what depends on the face
// direction (the same code serves the three).
template <int NS, class R, bool PACK>
struct FaceIn {
    const double *T, *p, *Y[NS], *X[NS];          // prim
    const double *E, *rY[NS];                     // cons 4, 5..
    const R *kappa, *chi[NS], *D[NS * NS];
    int psy, psz, csy, csz, ksy, ksz, hsy, hsz, dsy, dsz;   // prim, cons, kappa, chi, D
    int tsy, tsz, esy, esz;                       // ct, et
};
template <int NS, class R>
struct FaceIn<NS, R, true> {
    const double *T, *p, *Y[NS];                  // prim, for the hyperbolic part
    const double *E, *rY[NS];
    int psy, psz, csy, csz, tsy, tsz, esy, esz;
};
template <int NS, class R, bool PACK>
struct FaceDir {
    const double *u, *m;                          // vel[d], mom[d]
    int usy, usz, msy, msz;
    const std::conditional_t<PACK, Pair<R>, R>*cs, *cd;   // ct comps d, 3 + d (PACK: cs the pair)
    struct Family {                               // edge family f (first, second transverse direction)
        const std::conditional_t<PACK, Pair<R>, R>*s, *d; // et comps (s, d) (PACK: s the pair)
        const double* v;                          // transverse velocity
        int eq, vsy, vsz, vq, vd;                 // et: step to position 1; v: strides, steps to position 1 and across the face
    } f[2];
    int pd, cd_, kd, hd, dd, td, qd;              // steps across the face in prim, cons, kappa, chi, D, ct, records
    Items it;
};

template <int NS, class R, int NZ, bool PACK = false>
struct alignas(16) StageArgs {
    RunParams P;
    std::conditional_t<PACK, FieldsPack<NS, R>, Fields<NS, R>> F;   // stage-input state U^s + derived fields
    Noise<NZ> noise;
    StageScratch<NS, R, PACK> S;
    Arr4<double> mc;
    Arr4<const double> cons0;    // U^0 (for the RK combination)
    Arr4<const double> mom0[3];
    Arr4<double> cons_o;         // U^{s+1}
    Arr4<double> mom_o[3];
    Arr4<const double> src;      // source (nprimvars comps) or p == nullptr
    FaceIn<NS, R, PACK> fi;
    FaceDir<NS, R, PACK> fd[3];
    Items it_taus, it_upd;       // cells [-1, n]^3, points [0, n]^3
    int stage;                   // 1, 2, 3
    int img;                     // packed: ghost width of the periodic images the update stores (0: none)
};

// stresses on cells (grown by 1) and edges; one thread per point of [-1, n]^3
template <int NS, class R, int NZ, bool PACK>
FHD_D int taus_count(const StageArgs<NS, R, NZ, PACK>& a) { return a.it_taus.n; }

// The flux MultiFabs of a caller that wants them (the reference's by-products, and the
// flux operator's outputs): the stress kernel has every edge and centre total and the
// face kernel every face flux in registers when it stores its stage's scratch, so
// AUX writes them from there.  Computing them in kernels of their own recomputed six
// stresses with their noise for every face.
template <bool AUX>
struct StageAux {
    Arr4<double> ff[3];   // faceflux (nvars+4 comps)
    Arr4<double> ef[6];   // edgeflux_x[0..1], edgeflux_y[0..1], edgeflux_z[0..1]
    Arr4<double> cf[3];   // cenflux (1 ghost)
};
template <>
struct StageAux<false> {};

// ---- staged operands ---------------------------------------------------------------
// In a box of a few waves the stress kernel's time is one thread's: registers hold only a
// few of a point's 32 operands at a time, so it waits for memory several times in turn,
// then draws its noise.  Staged, a thread issues all of them at once as asynchronous
// copies into its own column of shared memory, draws the noise meanwhile, waits once and
// computes from there (launch_stage_part_t has the figures and the size up to which it is
// used; more registers without it gave 38.5 us for 38.6).  A column is read by its own
// thread alone, so cp.async.wait_all orders it and no barrier is needed.
template <int N>
FHD_D void stage_copy(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(src), "n"(N) : "memory");
}
FHD_D void stage_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

constexpr int kStagedThreads = 128;

// stress kernel: (T, eta) words of the point's cell and the six below it that its edges
// touch, its pressure, and four values of each face velocity and momentum
template <int NS, class R>
struct TausStage {
    static constexpr bool f64 = sizeof(R) == 8;
    static constexpr int n16 = 7 + (f64 ? 1 : 0), n8 = 24 + (f64 ? 0 : 1);
    static constexpr int bytes = (n16 * 16 + n8 * 8) * kStagedThreads;
};
template <int NS, class R>
struct FieldsStaged {
    // values of one face field: (0), one above in its own direction, one below in the
    // first and in the second of the other two
    struct Face {
        const double* s;
        int d, i, j, k;
        FHD_D static int slot(int d, int dx, int dy, int dz) {
            if (dx + dy + dz > 0) return 1;
            if (dx < 0) return 2;
            if (dy < 0) return d == 0 ? 2 : 3;
            return dz < 0 ? 3 : 0;
        }
        FHD_D double operator()(int a, int b, int c) const { return s[slot(d, a - i, b - j, c - k) * kStagedThreads]; }
    };
    const Vec<R>* s16;   // the thread's columns
    const double* s8;
    int i, j, k;
    R zr;
    Face vel[3], mom[3];
    FHD_D FieldsStaged(const unsigned char* smem, int i_, int j_, int k_, R zr_) : i(i_), j(j_), k(k_), zr(zr_) {
        s16 = reinterpret_cast<const Vec<R>*>(smem) + threadIdx.x;
        s8 = reinterpret_cast<const double*>(smem + TausStage<NS, R>::n16 * 16 * kStagedThreads) + threadIdx.x;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            vel[d] = Face{s8 + 4 * d * kStagedThreads, d, i, j, k};
            mom[d] = Face{s8 + (12 + 4 * d) * kStagedThreads, d, i, j, k};
        }
    }
    FHD_D R word(int a, int b, int c, int e) const {
        return vget(s16[((i - a) + 2 * (j - b) + 4 * (k - c)) * kStagedThreads], e);
    }
    FHD_D R T(int a, int b, int c) const { return word(a, b, c, RecLayout<NS, R>::T); }
    FHD_D R eta(int a, int b, int c) const { return word(a, b, c, RecLayout<NS, R>::ETA); }
    FHD_D R zeta(int a, int b, int c) const { return zr * eta(a, b, c); }
    FHD_D double p(int, int, int) const {
        if constexpr (sizeof(R) == 8) return vget(s16[7 * kStagedThreads], RecLayout<NS, R>::PR % 2);
        else return s8[24 * kStagedThreads];
    }
};
template <int NS, class R>
FHD_D void taus_issue(const FieldsPack<NS, R>& F, unsigned char* smem, int i, int j, int k, bool edges) {
    constexpr int B = kStagedThreads;
    Vec<R>* s16 = reinterpret_cast<Vec<R>*>(smem) + threadIdx.x;
    double* s8 = reinterpret_cast<double*>(smem + TausStage<NS, R>::n16 * 16 * B) + threadIdx.x;
    const int oq = F.q.at(i, j, k);
    stage_copy<16>(s16, F.q.p + oq);
    if constexpr (sizeof(R) == 8) stage_copy<16>(s16 + 7 * B, F.q.p + oq + F.q.sn);
    else stage_copy<8>(s8 + 24 * B, &F.pr(i, j, k, F.pT + 1));
#pragma unroll
    for (int d = 0; d < 3; ++d) {
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const Arr4<const double>& f = m ? F.mom[d] : F.vel[d];
            double* s = s8 + (12 * m + 4 * d) * B;
            const double* g = &f(i, j, k);
            stage_copy<8>(s, g);
            stage_copy<8>(s + B, g + (d == 0 ? 1 : (d == 1 ? f.sy : f.sz)));
            if (edges) {
                stage_copy<8>(s + 2 * B, g - (d == 0 ? f.sy : 1));
                stage_copy<8>(s + 3 * B, g - (d == 2 ? f.sy : f.sz));
            }
        }
    }
    if (edges) {
#pragma unroll
        for (int c = 1; c < 7; ++c)
            stage_copy<16>(s16 + c * B, F.q.p + oq - ((c & 1) + ((c >> 1) & 1) * F.q.sy + (c >> 2) * F.q.sz));
    }
}

// both edge totals of edge E into the stage's scratch (absent: the flux operator) and
// the flux fabs
template <int E, bool AUX, class A>
FHD_D void put_edge(const A& a, const StageAux<AUX>& x, int i, int j, int k, double va, double vb) {
    if (!AUX || a.S.has_me()) a.S.put_me(E, i, j, k, va, vb);
    if constexpr (AUX) {
        constexpr int ca = E == 0 ? 2 : (E == 1 ? 4 : 5), cb = E == 0 ? 0 : (E == 1 ? 1 : 3);
        x.ef[ca](i, j, k) = va;
        x.ef[cb](i, j, k) = vb;
    }
}

// stress and edge totals of edge E at point (i, j, k)
template <int NS, class R, int NZ, int E, bool WL, bool AUX, bool PACK, class FT>
FHD_D void taus_edge(const StageArgs<NS, R, NZ, PACK>& a, const FT& F, const StageAux<AUX>& x, double w, int i, int j,
                     int k) {
    const RunParams& P = a.P;
    const int hadv = P.advection_type >= 0;
    const Taus<R> e = edge_taus_w<NS, R, NZ, E, WL>(P, F, w, i, j, k);
    a.S.put_et(E, i, j, k, e);
    double ea, eb;
    edge_adv<NS, R, E, WL>(P, F, i, j, k, ea, eb);
    put_edge<E>(a, x, i, j, k, WL ? edge_total_w<R, E>(P, e, ea, hadv, i, j, k) : edge_total<R>(e, ea, hadv),
                WL ? edge_total_w<R, E>(P, e, eb, hadv, i, j, k) : edge_total<R>(e, eb, hadv));
}

// WL: walls (the wall variants of the edge stresses, advective edge fluxes and
// StochFluxStag's factors on the edge totals)
// STAGED: the operands come through shared memory (smem, TausStage)
template <int NS, class R, int NZ, bool WL = false, bool AUX = false, bool STAGED = false, bool PACK = false>
FHD_D void taus_point(const StageArgs<NS, R, NZ, PACK>& a, int q, const StageAux<AUX>& x = StageAux<AUX>(),
                      unsigned char* smem = nullptr) {
    const RunParams& P = a.P;
    int i, j, k;
    a.it_taus.point(q, i, j, k);
    --i; --j; --k;
    const bool edges = i >= 0 && j >= 0 && k >= 0;
    double wc[3] = {0.0, 0.0, 0.0}, we[3] = {0.0, 0.0, 0.0};
    if constexpr (STAGED) taus_issue<NS, R>(a.F, smem, i, j, k, edges);
    if (NZ != NZ_OFF) a.noise.cen_and_yz_edge(P, i, j, k, edges, wc, we[2]);
    auto work = [&](const auto& F) {
        const CellTaus<R> t = cell_taus_w<NS, R, NZ, WL>(P, F, wc, i, j, k);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            a.S.put_ct(i, j, k, d, t.s[d], t.d[d]);
            const double c = cen_total_res<NS, R, NZ, WL>(P, F, a.noise, t, d, i, j, k);
            if (!AUX || a.mc.p) a.mc(i, j, k, d) = c;
            if constexpr (AUX) x.cf[d](i, j, k) = c;
        }
        if (!edges) return;
        if (NZ != NZ_OFF && !STAGED) a.noise.xy_xz_edges(P, i, j, k, we[0], we[1]);
        if (k < P.n[2]) taus_edge<NS, R, NZ, 0, WL>(a, F, x, we[0], i, j, k);
        if (j < P.n[1]) taus_edge<NS, R, NZ, 1, WL>(a, F, x, we[1], i, j, k);
        if (i < P.n[0]) taus_edge<NS, R, NZ, 2, WL>(a, F, x, we[2], i, j, k);
    };
    if constexpr (STAGED) {
        if (NZ != NZ_OFF && edges) a.noise.xy_xz_edges(P, i, j, k, we[0], we[1]);
        stage_wait();
        work(FieldsStaged<NS, R>(smem, i, j, k, a.F.zr));
    } else {
        work(a.F);
    }
}

// Packed, beyond the sizes of k_taus_staged: bound by the latency of its loads, where 48
// registers (40 warps per SM; a few spilled values) beat 64 (32 warps): 510 against 529 us
// per step at 128^3 argon FP64, 654 at 80.  (0: no minimum.)
template <int NS, class R, int NZ, bool WL = false, bool AUX = false, bool PACK = false>
static __global__ void __launch_bounds__(256, PACK ? 5 : 0) k_taus(StageArgs<NS, R, NZ, PACK> a, StageAux<AUX> x) {
    const int tot = taus_count(a);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += gridDim.x * blockDim.x)
        taus_point<NS, R, NZ, WL, AUX>(a, q, x);
}

template <int NS, class R, int NZ>
static __global__ void __launch_bounds__(kStagedThreads, 5) k_taus_staged(StageArgs<NS, R, NZ, true> a) {
    extern __shared__ __align__(16) unsigned char stage_smem[];
    const int tot = taus_count(a);
    for (int q = blockIdx.x * kStagedThreads + threadIdx.x; q < tot; q += gridDim.x * kStagedThreads)
        taus_point<NS, R, NZ, false, false, true>(a, q, StageAux<false>{}, stage_smem);
}

// operands of one face of a direction known only at run time (face_flux)
template <int NS, class R, int NZ, bool PACK>
struct FaceRun {
    using L = RecLayout<NS, R>;
    const StageArgs<NS, R, NZ, PACK>& a;
    int d, op, oc, ok, oh, od, ot, oe, ou, om, ov[2];   // (ok: records when PACK)
    FHD_D FaceRun(const StageArgs<NS, R, NZ, PACK>& a_, int d_, int i, int j, int k) : a(a_), d(d_) {
        const auto& fi = a.fi;
        const auto& f = a.fd[d];
        op = i + j * fi.psy + k * fi.psz;
        oc = i + j * fi.csy + k * fi.csz;
        if constexpr (PACK) {
            ok = a.F.q.at(i, j, k);
        } else {
            ok = i + j * fi.ksy + k * fi.ksz;
            oh = i + j * fi.hsy + k * fi.hsz;
            od = i + j * fi.dsy + k * fi.dsz;
        }
        ot = i + j * fi.tsy + k * fi.tsz;
        oe = i + j * fi.esy + k * fi.esz;
        ou = i + j * f.usy + k * f.usz;
        om = i + j * f.msy + k * f.msz;
        ov[0] = i + j * f.f[0].vsy + k * f.f[0].vsz;
        ov[1] = i + j * f.f[1].vsy + k * f.f[1].vsz;
    }
    FHD_D const FaceDir<NS, R, PACK>& f() const { return a.fd[d]; }
    FHD_D int dir() const { return d; }
    FHD_D R rec(int s, int c) const { return a.F.q.get(s ? ok : ok - f().qd, c); }
    FHD_D auto T(int s) const {
        if constexpr (PACK) return rec(s, L::T);
        else return a.fi.T[s ? op : op - f().pd];
    }
    FHD_D auto p(int s) const {
        if constexpr (PACK) return rec(s, L::PR);
        else return a.fi.p[s ? op : op - f().pd];
    }
    FHD_D auto Y(int s, int n) const {
        if constexpr (PACK) return rec(s, L::Y + n);
        else return a.fi.Y[n][s ? op : op - f().pd];
    }
    FHD_D auto X(int s, int n) const {
        if constexpr (PACK) return rec(s, L::X + n);
        else return a.fi.X[n][s ? op : op - f().pd];
    }
    // T, p and Y in FP64 for the hyperbolic part
    FHD_D double Td(int s) const { return a.fi.T[s ? op : op - f().pd]; }
    FHD_D double pd(int s) const {
        if constexpr (PACK && sizeof(R) == 8) return rec(s, L::PR);
        else return a.fi.p[s ? op : op - f().pd];
    }
    FHD_D double Yd(int s, int n) const { return a.fi.Y[n][s ? op : op - f().pd]; }
    FHD_D double cons(int s, int n) const {
        const int o = s ? oc : oc - f().cd_;
        if (n == 4) return a.fi.E[o];
        if (n >= 5) return a.fi.rY[n - 5][o];
        return a.F.cons.p[o];
    }
    FHD_D R kappa(int s) const {
        if constexpr (PACK) return rec(s, L::KAPPA);
        else return a.fi.kappa[s ? ok : ok - f().kd];
    }
    FHD_D R chi(int s, int n) const {
        if constexpr (PACK) return rec(s, L::CHI + n);
        else return a.fi.chi[n][s ? oh : oh - f().hd];
    }
    FHD_D R Dc(int s, int n) const {
        if constexpr (PACK) return rec(s, L::D + n);
        else return a.fi.D[n][s ? od : od - f().dd];
    }
    FHD_D double u() const { return f().u[ou]; }
    FHD_D double m() const { return f().m[om]; }
    FHD_D Taus<R> cell(int s) const {
        const int o = s ? ot : ot - f().td;
        Taus<R> t;
        if constexpr (PACK) {
            const Pair<R> v = f().cs[o];
            t.s = v.x;
            t.d = v.y;
        } else {
            t.s = f().cs[o];
            t.d = f().cd[o];
        }
        return t;
    }
    FHD_D Taus<R> edge(int q, int pos) const {
        const int o = pos ? oe + f().f[q].eq : oe;
        Taus<R> t;
        if constexpr (PACK) {
            const Pair<R> v = f().f[q].s[o];
            t.s = v.x;
            t.d = v.y;
        } else {
            t.s = f().f[q].s[o];
            t.d = f().f[q].d[o];
        }
        return t;
    }
    FHD_D double vt(int q, int pos, int s) const {
        const auto& v = f().f[q];
        return v.v[ov[q] + (pos ? v.vq : 0) - (s ? 0 : v.vd)];
    }
};

template <int NS, class R, int NZ, bool PACK>
FHD_D int faces_count(const StageArgs<NS, R, NZ, PACK>& a, int d) { return a.fd[d].it.n; }

// conservative flux of face q of direction d
template <int NS, class R, int NZ, bool WL = false, bool AUX = false, bool PACK = false>
FHD_D void faces_point(const StageArgs<NS, R, NZ, PACK>& a, int d, int q, const StageAux<AUX>& aux = StageAux<AUX>()) {
    int i, j, k;
    a.fd[d].it.point(q, i, j, k);
    const FaceRun<NS, R, NZ, PACK> x(a, d, i, j, k);
    const FaceFlux<NS> f = face_flux<NS, R, NZ, WL>(a.P, a.F, a.noise, x, i, j, k);
    if (!AUX || a.S.has_ff(d)) a.S.put_ff(d, i, j, k, f.cons);
    if constexpr (AUX) {
        const Arr4<double>& o = aux.ff[d];
        o(i, j, k, 0) = f.cons[0];
        o(i, j, k, 1) = 0.0;
        o(i, j, k, 2) = 0.0;
        o(i, j, k, 3) = 0.0;
        o(i, j, k, 4) = f.cons[1];
#pragma unroll
        for (int s = 0; s < NS; ++s) o(i, j, k, 5 + s) = f.cons[2 + s];
#pragma unroll
        for (int c = 0; c < 4; ++c) o(i, j, k, 5 + NS + c) = f.aux[c];
    }
}

// The faces of the three directions in one launch, block b on direction b % 3: the
// blocks working at one time then read the same cells for all three directions, so
// the second and third find them in L2, and a small box keeps three times as many SMs
// busy as one launch per direction.
// MINB = minimum resident blocks requested from the register allocator.
template <int NS, class R, int NZ, int BS, int MINB, bool WL = false, bool AUX = false, bool PACK = false>
static __global__ void __launch_bounds__(BS, MINB) k_faces(StageArgs<NS, R, NZ, PACK> a, int per, StageAux<AUX> x) {
    const int d = blockIdx.x % 3;
    const int tot = faces_count(a, d);
    for (int q = (blockIdx.x / 3) * BS + threadIdx.x; q < tot; q += per * BS)
        faces_point<NS, R, NZ, WL, AUX>(a, d, q, x);
}

// Periodic ghosts from the kernel that computes the values (FillBoundary fused into its
// producer): a point within g of a face of the box also stores its values at the ghost
// points they wrap to, instead of a launch per stage that reads and writes them again
// (argon FP64 per step, before and after: 32^3 125 and 117 us, 64^3 423 and 403 us, 128^3
// 2760 and 2732 us).  With n > 2 g (image_width) that is at most one shift per direction.
// image_shift: that shift of index i in a direction of n cells (0: no image)
FHD_D int image_shift(int i, int n, int g, int nodal) {
    return i >= nodal && i < g + nodal ? n : (i >= n - g && i < n ? -n : 0);
}
// put(di, dj, dk) for the point itself, (0, 0, 0), and each of its images
template <class F>
FHD_D void images(int sx, int sy, int sz, F&& put) {
    for (int dk = 0;; dk = sz) {
        for (int dj = 0;; dj = sy) {
            put(0, dj, dk);
            if (sx) put(sx, dj, dk);
            if (dj == sy) break;
        }
        if (dk == sz) break;
    }
}

// RK3 stage combination (timeStepStag.cpp:439-528, 771-861, 1106-1202): one thread
// per point of [0, n]^3 updates the cell there (if valid) and the faces there
template <int NS, class R, int NZ, bool PACK>
FHD_D int update_count(const StageArgs<NS, R, NZ, PACK>& a) { return a.it_upd.n; }

// SPLIT: one part of it alone, 0 the cell, 1 + d the face of direction d
template <bool SPLIT = false, int NS, class R, int NZ, bool PACK>
FHD_D void update_point(const StageArgs<NS, R, NZ, PACK>& a, int q, int part = 0) {
    const RunParams& P = a.P;
    const auto& F = a.F;
    const double dt = P.dt;
    const int st = a.stage;
    {
        int i, j, k;
        a.it_upd.point(q, i, j, k);
        const bool cell = i < P.n[0] && j < P.n[1] && k < P.n[2];
        if (cell && (!SPLIT || part == 0)) {
            using S = std::remove_const_t<std::remove_reference_t<decltype(a.S)>>;
            double on[2 + NS];
#pragma unroll
            for (int w = 0; w < S::NW; ++w) {
                double fx[2], fy[2], fz[2];
                a.S.ff_diff(w, 0, i, j, k, fx);
                a.S.ff_diff(w, 1, i, j, k, fy);
                a.S.ff_diff(w, 2, i, j, k, fz);
#pragma unroll
                for (int e = 0; e < S::count(w); ++e) {
                    const int c = S::first(w) + e;
                    const int n = (c == 0) ? 0 : 3 + c;  // conserved component index
                    const double div = divc(P, fx[e], P.dx[0], P.rdx[0]) + divc(P, fy[e], P.dx[1], P.rdx[1]) +
                                       divc(P, fz[e], P.dx[2], P.rdx[2]);
                    const double src = a.src.p ? a.src(i, j, k, n) : 0.0;
                    const double u0 = a.cons0(i, j, k, n);
                    double v;
                    if (st == 1) v = u0 - dt * (div) + dt * src;
                    else if (st == 2) v = 0.25 * (3.0 * u0 + F.cons(i, j, k, n) - dt * (div) + dt * src);
                    else v = (2. / 3.) * (0.5 * u0 + F.cons(i, j, k, n) - dt * (div) + dt * src);
                    on[c] = v;
                }
            }
            // gravity work on the energy with the stage-input momenta
            const double gfac = (st == 1) ? 0.5 * dt : (st == 2) ? 0.5 * 0.25 * dt : 0.5 * (2. / 3.) * dt;
            on[1] += gfac * (P.grav[0] * (F.mom[0](i + 1, j, k) + F.mom[0](i, j, k)) +
                             P.grav[1] * (F.mom[1](i, j + 1, k) + F.mom[1](i, j, k)) +
                             P.grav[2] * (F.mom[2](i, j, k + 1) + F.mom[2](i, j, k)));
            auto put = [&](int di, int dj, int dk) {
#pragma unroll
                for (int c = 0; c < 2 + NS; ++c) a.cons_o(i + di, j + dj, k + dk, (c == 0) ? 0 : 3 + c) = on[c];
            };
            if constexpr (PACK)
                images(image_shift(i, P.n[0], a.img, 0), image_shift(j, P.n[1], a.img, 0),
                       image_shift(k, P.n[2], a.img, 0), put);
            else
                put(0, 0, 0);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int e0 = d == 0, e1 = d == 1, e2 = d == 2;
            if (SPLIT && part != 1 + d) continue;
            if (i >= P.n[0] + e0 || j >= P.n[1] + e1 || k >= P.n[2] + e2) continue;
            // momentum flux differences (timeStepStag.cpp:452-482): centre and edge
            // totals stored by k_taus
            double t1, t2, t3;
            if (d == 0) {
                t1 = a.mc(i, j, k, 0) - a.mc(i - 1, j, k, 0);
                t2 = a.S.get_me(0, 0, i, j + 1, k) - a.S.get_me(0, 0, i, j, k);   // edgey_u
                t3 = a.S.get_me(1, 0, i, j, k + 1) - a.S.get_me(1, 0, i, j, k);   // edgez_u
            } else if (d == 1) {
                t1 = a.S.get_me(0, 1, i + 1, j, k) - a.S.get_me(0, 1, i, j, k);   // edgex_v
                t2 = a.mc(i, j, k, 1) - a.mc(i, j - 1, k, 1);
                t3 = a.S.get_me(2, 0, i, j, k + 1) - a.S.get_me(2, 0, i, j, k);   // edgez_v
            } else {
                t1 = a.S.get_me(1, 1, i + 1, j, k) - a.S.get_me(1, 1, i, j, k);   // edgex_w
                t2 = a.S.get_me(2, 1, i, j + 1, k) - a.S.get_me(2, 1, i, j, k);   // edgey_w
                t3 = a.mc(i, j, k, 2) - a.mc(i, j, k - 1, 2);
            }
            const double rsum = F.cons(i - e0, j - e1, k - e2, 0) + F.cons(i, j, k, 0);
            const double m0 = a.mom0[d](i, j, k);
            double v;
            if (st == 1) {
                v = m0 - divc(P, dt * t1, P.dx[0], P.rdx[0]) - divc(P, dt * t2, P.dx[1], P.rdx[1]) -
                    divc(P, dt * t3, P.dx[2], P.rdx[2]) + 0.5 * dt * P.grav[d] * rsum;
            } else if (st == 2) {
                v = 0.25 * 3.0 * m0 + 0.25 * F.mom[d](i, j, k) - divc(P, 0.25 * dt * t1, P.dx[0], P.rdx[0]) -
                    divc(P, 0.25 * dt * t2, P.dx[1], P.rdx[1]) - divc(P, 0.25 * dt * t3, P.dx[2], P.rdx[2]) +
                    0.5 * 0.25 * dt * P.grav[d] * rsum;
            } else {
                v = (2. / 3.) * (0.5 * m0 + F.mom[d](i, j, k)) - divc(P, (2. / 3.) * dt * t1, P.dx[0], P.rdx[0]) -
                    divc(P, (2. / 3.) * dt * t2, P.dx[1], P.rdx[1]) - divc(P, (2. / 3.) * dt * t3, P.dx[2], P.rdx[2]) +
                    0.5 * (2. / 3.) * dt * P.grav[d] * rsum;
            }
            auto put = [&](int di, int dj, int dk) { a.mom_o[d](i + di, j + dj, k + dk) = v; };
            if constexpr (PACK)
                images(image_shift(i, P.n[0], a.img, e0), image_shift(j, P.n[1], a.img, e1),
                       image_shift(k, P.n[2], a.img, e2), put);
            else
                put(0, 0, 0);
        }
    }
}

// MINB: 16 blocks of 128 (32 registers, full occupancy; packed 12 or 10) where the kernel
// streams from HBM; 4 for a small box that is not packed (launch_update)
template <int NS, class R, int NZ, int MINB, bool PACK>
static __global__ void __launch_bounds__(128, MINB) k_update(StageArgs<NS, R, NZ, PACK> a) {
    const int tot = update_count(a);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += gridDim.x * blockDim.x) update_point(a, q);
}

// one part of a point per thread, block b on part b % 4
template <int NS, class R, int NZ>
static __global__ void __launch_bounds__(128, 6) k_update_split(StageArgs<NS, R, NZ, true> a) {
    const int q = (blockIdx.x / 4) * 128 + threadIdx.x;
    if (q < update_count(a)) update_point<true>(a, q, blockIdx.x % 4);
}

// ===================================================================================
// conservedToPrimitiveStag on valid cells/faces (conservedPrimitiveConversionsStag.cpp)
// ===================================================================================
template <int NS>
struct alignas(16) ConvArgs {
    RunParams P;
    Items it;
    Arr4<double> prim;   // reference layout (nprimvars comps)
    Arr4<double> vel[3];
    Arr4<double> cons;   // comps 1..3 rewritten
    Arr4<const double> mom[3];
    int* status;
    int img;             // ghost width of the periodic images to store too (0: none)
};

template <int NS>
FHD_D int convert_count(const ConvArgs<NS>& a) { return a.it.n; }

// IMG: with the periodic images (a.img).  A step's conversion stores them; the operator's,
// and those of boxes whose ghosts are filled apart, have none, and hold no value for them:
// 48 registers for two species and 54 for four against 72 and 96, 114 against 138 us and
// 138 against 189 at 128^3.
template <bool IMG, int NS>
FHD_D void convert_point(const ConvArgs<NS>& a, int q) {
    const RunParams& P = a.P;
    auto put = [](int sx, int sy, int sz, auto&& f) {
        if constexpr (IMG) images(sx, sy, sz, f);
        else f(0, 0, 0);
    };
    {
        int i, j, k;
        a.it.point(q, i, j, k);
        const Arr4<double>& cons = a.cons;
        const double rho = cons(i, j, k, 0);
        const Arr4<const double>&mx = a.mom[0], &my = a.mom[1], &mz = a.mom[2];
        // face velocities (:61-67); the last cell in a direction also owns face n_cells
        const double vxl = 2 * mx(i, j, k) / (rho + cons(i - 1, j, k, 0));
        const double vyl = 2 * my(i, j, k) / (rho + cons(i, j - 1, k, 0));
        const double vzl = 2 * mz(i, j, k) / (rho + cons(i, j, k - 1, 0));
        const double vxh = 2 * mx(i + 1, j, k) / (cons(i + 1, j, k, 0) + rho);
        const double vyh = 2 * my(i, j + 1, k) / (cons(i, j + 1, k, 0) + rho);
        const double vzh = 2 * mz(i, j, k + 1) / (cons(i, j, k + 1, 0) + rho);
        const int g = IMG ? a.img : 0;
        const int s0 = image_shift(i, P.n[0], g, 0), s1 = image_shift(j, P.n[1], g, 0), s2 = image_shift(k, P.n[2], g, 0);
        put(image_shift(i, P.n[0], g, 1), s1, s2,
            [&](int di, int dj, int dk) { a.vel[0](i + di, j + dj, k + dk) = vxl; });
        put(s0, image_shift(j, P.n[1], g, 1), s2,
            [&](int di, int dj, int dk) { a.vel[1](i + di, j + dj, k + dk) = vyl; });
        put(s0, s1, image_shift(k, P.n[2], g, 1),
            [&](int di, int dj, int dk) { a.vel[2](i + di, j + dj, k + dk) = vzl; });
        // (the node of the high side has images in the other two directions alone)
        if (i == P.n[0] - 1) put(0, s1, s2, [&](int, int dj, int dk) { a.vel[0](i + 1, j + dj, k + dk) = vxh; });
        if (j == P.n[1] - 1) put(s0, 0, s2, [&](int di, int, int dk) { a.vel[1](i + di, j + 1, k + dk) = vyh; });
        if (k == P.n[2] - 1) put(s0, s1, 0, [&](int di, int dj, int) { a.vel[2](i + di, j + dj, k + 1) = vzh; });
        const double vc[3] = {0.5 * (vxl + vxh), 0.5 * (vyl + vyh), 0.5 * (vzl + vzh)};
        const double mc[3] = {0.5 * (mx(i, j, k) + mx(i + 1, j, k)), 0.5 * (my(i, j, k) + my(i, j + 1, k)),
                              0.5 * (mz(i, j, k) + mz(i, j, k + 1))};
        auto flow = [&](int di, int dj, int dk) {
            double* u = &cons(i + di, j + dj, k + dk);
            double* w = &a.prim(i + di, j + dj, k + dk);
            w[0] = rho;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                u[(1 + d) * cons.sn] = mc[d];
                w[(1 + d) * a.prim.sn] = vc[d];
            }
        };
        if constexpr (!IMG) flow(0, 0, 0);   // (their registers are free for the rest)
        double rY[NS];
#pragma unroll
        for (int n = 0; n < NS; ++n) rY[n] = cons(i, j, k, 5 + n);
        Prim<NS> q2;
        if (!cons_to_prim<NS>(P, rho, cons(i, j, k, 4), rY, mx(i, j, k), mx(i + 1, j, k), my(i, j, k), my(i, j + 1, k),
                              mz(i, j, k), mz(i, j, k + 1), q2))
            flag(a.status, ST_NONFINITE);
        put(s0, s1, s2, [&](int di, int dj, int dk) {
            if constexpr (IMG) flow(di, dj, dk);
            double* w = &a.prim(i + di, j + dj, k + dk);
            w[4 * a.prim.sn] = q2.T;
            w[5 * a.prim.sn] = q2.p;
#pragma unroll
            for (int n = 0; n < NS; ++n) {
                w[(6 + n) * a.prim.sn] = q2.Y[n];
                w[(6 + NS + n) * a.prim.sn] = q2.X[n];
            }
        });
    }
}

template <int NS, bool IMG>
static __global__ void __launch_bounds__(128) k_convert(ConvArgs<NS> a) {
    const int tot = convert_count(a);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += gridDim.x * blockDim.x) convert_point<IMG>(a, q);
}

// ===================================================================================
// periodic FillBoundary of up to 16 fabs in one launch
// ===================================================================================
struct GhostFab {
    double* p;        // point (0,0,0)
    int g, vhi[3];    // ghost width; valid upper index per direction
    int sy, sz, sn;
    int c0, nc;       // component range
    int npts;         // ghost points of one component
    int n[3];         // cells of the box (period)
    // periodic directions (walls elsewhere).  mode 0 (FillBoundary): a ghost point
    // is filled only when it lies outside the valid box in periodic directions
    // alone; mode 1 (noise fields whose wall ghosts hold their own values): the
    // periodic coordinates are wrapped and the wall coordinates kept.
    int per[3];
    int mode;
    int zsl, ysl;     // points of the two z slabs (all x, y) and of the two y slabs (valid z)
    int nx, vy, vz;   // row length with ghosts; valid rows and planes
    FastDiv dpts, dzp, dnx, dyp, dxp, dvy;   // by npts, nx*(vy+2g), nx, nx*vz, vy*vz, vy
};
struct GhostArgs {
    GhostFab f[16];
    int nf;
};

// host: the ghost fill of components c0 .. c0+nc-1 of a fab of the box (a fab has fewer
// than 2^31 values, so every index here is 32-bit and the divisions are FastDiv: with
// 64-bit ones the fill of a statistics update took 39 us at 144x112x96, see fill_ghosts)
inline GhostFab make_ghost(void* data, const int lo[3], const int hi[3], const int nodal[3], int c0, int nc,
                           const int ncell[3], const int* periodic, int mode) {
    GhostFab f;
    f.g = -lo[0];
    const int ex = hi[0] - lo[0] + 1, ey = hi[1] - lo[1] + 1, ez = hi[2] - lo[2] + 1;
    f.sy = ex;
    f.sz = ex * ey;
    f.sn = ex * ey * ez;
    f.p = static_cast<double*>(data) + f.g * (1 + f.sy + f.sz);
    f.c0 = c0;
    f.nc = nc;
    for (int d = 0; d < 3; ++d) {
        f.vhi[d] = ncell[d] - 1 + nodal[d];
        f.n[d] = ncell[d];
        f.per[d] = periodic ? periodic[d] : 1;
    }
    f.mode = mode;
    f.nx = ex;
    f.vy = f.vhi[1] + 1;
    f.vz = f.vhi[2] + 1;
    f.zsl = 2 * f.g * ex * ey;
    f.ysl = 2 * f.g * ex * f.vz;
    f.npts = f.zsl + f.ysl + 2 * f.g * f.vy * f.vz;
    auto div = [](int d) { return fast_div((uint32_t)(d > 0 ? d : 1)); };
    f.dpts = div(f.npts);
    f.dzp = div(ex * ey);
    f.dnx = div(ex);
    f.dyp = div(ex * f.vz);
    f.dxp = div(f.vy * f.vz);
    f.dvy = div(f.vy);
    return f;
}

FHD_D void ghost_point(const GhostFab& f, int q) {
    const int g = f.g;
    const int cc = (int)f.dpts.div((uint32_t)q);
    int r = q - cc * f.npts;
    int s[3];
    if (r < f.zsl) {
        const int kk = (int)f.dzp.div((uint32_t)r);
        r -= kk * f.sz;
        const int jj = (int)f.dnx.div((uint32_t)r);
        s[0] = r - jj * f.nx - g;
        s[1] = jj - g;
        s[2] = kk < g ? kk - g : f.vz + (kk - g);
    } else if (r < f.zsl + f.ysl) {
        r -= f.zsl;
        const int jj = (int)f.dyp.div((uint32_t)r);
        r -= jj * f.nx * f.vz;
        const int kk = (int)f.dnx.div((uint32_t)r);
        s[0] = r - kk * f.nx - g;
        s[1] = jj < g ? jj - g : f.vy + (jj - g);
        s[2] = kk;
    } else {
        r -= f.zsl + f.ysl;
        const int ii = (int)f.dxp.div((uint32_t)r);
        r -= ii * f.vy * f.vz;
        const int kk = (int)f.dvy.div((uint32_t)r);
        s[0] = ii < g ? ii - g : f.vhi[0] + 1 + (ii - g);
        s[1] = r - kk * f.vy;
        s[2] = kk;
    }
    double* base = f.p + (f.c0 + cc) * f.sn;
    double* dst = base + s[0] + s[1] * f.sy + s[2] * f.sz;
    bool wrapped = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (s[d] >= 0 && s[d] <= f.vhi[d]) continue;
        if (!f.per[d]) {
            if (f.mode == 0) return;
            continue;
        }
        wrapped = true;
        while (s[d] < 0) s[d] += f.n[d];
        while (s[d] > f.vhi[d]) s[d] -= f.n[d];
    }
    if (!wrapped) return;
    *dst = base[s[0] + s[1] * f.sy + s[2] * f.sz];
}

static __global__ void __launch_bounds__(256) k_ghosts(GhostArgs a) {
    const int fidx = blockIdx.y;
    if (fidx >= a.nf) return;
    const GhostFab& f = a.f[fidx];
    const int tot = f.npts * f.nc;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += gridDim.x * blockDim.x) ghost_point(f, q);
}

// OverrideSync: nodal point n_cells <- point 0 (per nodal direction)
struct SyncArgs {
    double* p;
    int lo;
    int nodal[3];   // nodal and periodic (a wall direction has no duplicate points)
    int n[3];
    int64_t sy, sz, sn;
    int nc;
};
static __global__ void k_override_sync(SyncArgs a) {
    const int g = -a.lo;
    const int VX = a.n[0] + a.nodal[0], VY = a.n[1] + a.nodal[1], VZ = a.n[2] + a.nodal[2];
    const int64_t tot = (int64_t)VX * VY * VZ * a.nc;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < tot; q += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(q % VX), j = (int)((q / VX) % VY), k = (int)((q / ((int64_t)VX * VY)) % VZ);
        const int c = (int)(q / ((int64_t)VX * VY * VZ));
        int si = i, sj = j, sk = k;
        bool dup = false;
        if (a.nodal[0] && i == a.n[0]) { si = 0; dup = true; }
        if (a.nodal[1] && j == a.n[1]) { sj = 0; dup = true; }
        if (a.nodal[2] && k == a.n[2]) { sk = 0; dup = true; }
        if (!dup) continue;
        const int64_t b = (int64_t)c * a.sn;
        a.p[b + (i + g) + (j + g) * a.sy + (k + g) * a.sz] = a.p[b + (si + g) + (sj + g) * a.sy + (sk + g) * a.sz];
    }
}

// ===================================================================================
// drop-in operators
// ===================================================================================
template <int NS>
struct TransArgs {
    DevParams P;
    Arr4<const double> prim;
    Arr4<double> eta, zeta, kappa, chi, D;
    Items it;          // the box grown by ng
    int ng;
    int* status;
};

// ALT: the Valk/Waldmann or HCB binary model (runs with these models take this
// kernel), else Giovangigli's.  One kernel with both models in it took 255 registers and
// 620 B of spills for four species (160 registers for two); apart, Giovangigli's has
// the cell kernel's register budget (cellprep_min_blocks).
template <int NS, bool ALT>
FHD_D void transport_body(const TransArgs<NS>& a) {
    const DevParams& P = a.P;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < a.it.n; q += gridDim.x * blockDim.x) {
        int i, j, k;
        a.it.point(q, i, j, k);
        i -= a.ng; j -= a.ng; k -= a.ng;
        double Y[NS];
#pragma unroll
        for (int n = 0; n < NS; ++n) Y[n] = a.prim(i, j, k, 6 + n);
        Coeffs<NS, double> c;
        if constexpr (ALT) {
            const int st = transport_alt<NS>(P, a.prim(i, j, k, 0), a.prim(i, j, k, 4), a.prim(i, j, k, 5), Y, c);
            if (st) flag(a.status, st);
        } else if (!transport_gio<NS, double>(P, a.prim(i, j, k, 0), a.prim(i, j, k, 4), a.prim(i, j, k, 5), Y, c)) {
            flag(a.status, ST_MASSFRAC);
        }
        a.eta(i, j, k) = c.eta;
        a.kappa(i, j, k) = c.kappa;
        a.zeta(i, j, k) = c.zeta;
#pragma unroll
        for (int n = 0; n < NS; ++n) a.chi(i, j, k, n) = c.chi[n];
#pragma unroll
        for (int n = 0; n < NS * NS; ++n) a.D(i, j, k, n) = c.D[n];
    }
}

template <int NS>
static __global__ void __launch_bounds__(128, cellprep_min_blocks<NS, double>()) k_transport(TransArgs<NS> a) {
    transport_body<NS, false>(a);
}
template <int NS>
static __global__ void __launch_bounds__(128) k_transport_alt(TransArgs<NS> a) {
    transport_body<NS, true>(a);
}

// stresses recomputed on the fly (operator path)
template <int NS, class R, int NZ, bool WL = false>
struct DirectTaus {
    const RunParams* P;
    const Fields<NS, R>* F;
    const Noise<NZ>* nz;
    FHD_D CellTaus<R> cell(int i, int j, int k) const { return cell_taus<NS, R, NZ, WL>(*P, *F, *nz, i, j, k); }
    template <int E>
    FHD_D Taus<R> edge(int i, int j, int k) const { return edge_taus<NS, R, NZ, E, WL>(*P, *F, *nz, i, j, k); }
};

template <int NS, class R, int NZ>
struct AuxArgs {
    RunParams P;
    Fields<NS, R> F;
    Noise<NZ> noise;
    Arr4<double> ff[3];   // faceflux (nvars+4 comps)
    Arr4<double> ef[6];   // edgeflux_x[0..1], edgeflux_y[0..1], edgeflux_z[0..1]
    Arr4<double> cf[3];   // cenflux (1 ghost)
};

// faceflux[d] on valid faces; items enumerate the three face boxes back to back
template <int NS, class R, int NZ, bool WL = false>
static __global__ void __launch_bounds__(128) k_aux_faces(AuxArgs<NS, R, NZ> a) {
    const RunParams& P = a.P;
    const int* N = P.n;
    const int64_t nxf = (int64_t)(N[0] + 1) * N[1] * N[2], nyf = (int64_t)N[0] * (N[1] + 1) * N[2],
                  nzf = (int64_t)N[0] * N[1] * (N[2] + 1);
    const DirectTaus<NS, R, NZ, WL> tg{&P, &a.F, &a.noise};
    using TG = DirectTaus<NS, R, NZ, WL>;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nxf + nyf + nzf; q += (int64_t)gridDim.x * blockDim.x) {
        int d, i, j, k;
        if (q < nxf) { d = 0; i = (int)(q % (N[0] + 1)); j = (int)((q / (N[0] + 1)) % N[1]); k = (int)(q / ((int64_t)(N[0] + 1) * N[1])); }
        else if (q < nxf + nyf) { const int64_t r = q - nxf; d = 1; i = (int)(r % N[0]); j = (int)((r / N[0]) % (N[1] + 1)); k = (int)(r / ((int64_t)N[0] * (N[1] + 1))); }
        else { const int64_t r = q - nxf - nyf; d = 2; i = (int)(r % N[0]); j = (int)((r / N[0]) % N[1]); k = (int)(r / ((int64_t)N[0] * N[1])); }
        FaceFlux<NS> f;
        if (d == 0) f = face_flux<NS, R, NZ, WL>(P, a.F, a.noise, FaceGen<NS, R, 0, TG>{a.F, tg, i, j, k}, i, j, k);
        else if (d == 1) f = face_flux<NS, R, NZ, WL>(P, a.F, a.noise, FaceGen<NS, R, 1, TG>{a.F, tg, i, j, k}, i, j, k);
        else f = face_flux<NS, R, NZ, WL>(P, a.F, a.noise, FaceGen<NS, R, 2, TG>{a.F, tg, i, j, k}, i, j, k);
        const Arr4<double>& o = a.ff[d];
        o(i, j, k, 0) = f.cons[0];
        o(i, j, k, 1) = 0.0;
        o(i, j, k, 2) = 0.0;
        o(i, j, k, 3) = 0.0;
        o(i, j, k, 4) = f.cons[1];
#pragma unroll
        for (int s = 0; s < NS; ++s) o(i, j, k, 5 + s) = f.cons[2 + s];
#pragma unroll
        for (int c = 0; c < 4; ++c) o(i, j, k, 5 + NS + c) = f.aux[c];
    }
}

// edge fluxes (6 fabs) on valid edges and centre fluxes on cells grown by 1
template <int NS, class R, int NZ, bool WL = false>
static __global__ void __launch_bounds__(128) k_aux_edges_cen(AuxArgs<NS, R, NZ> a) {
    const RunParams& P = a.P;
    const int* N = P.n;
    const int64_t nxy = (int64_t)(N[0] + 1) * (N[1] + 1) * N[2], nxz = (int64_t)(N[0] + 1) * N[1] * (N[2] + 1),
                  nyz = (int64_t)N[0] * (N[1] + 1) * (N[2] + 1), nc = (int64_t)(N[0] + 2) * (N[1] + 2) * (N[2] + 2);
    const int hadv = P.advection_type >= 0;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nxy + nxz + nyz + nc; q += (int64_t)gridDim.x * blockDim.x) {
        double ea, eb;
        if (q < nxy) {
            const int i = (int)(q % (N[0] + 1)), j = (int)((q / (N[0] + 1)) % (N[1] + 1)), k = (int)(q / ((int64_t)(N[0] + 1) * (N[1] + 1)));
            const Taus<R> t = edge_taus<NS, R, NZ, 0, WL>(P, a.F, a.noise, i, j, k);
            edge_adv<NS, R, 0, WL>(P, a.F, i, j, k, ea, eb);
            a.ef[2](i, j, k) = WL ? edge_total_w<R, 0>(P, t, ea, hadv, i, j, k) : edge_total<R>(t, ea, hadv);  // edgey_u
            a.ef[0](i, j, k) = WL ? edge_total_w<R, 0>(P, t, eb, hadv, i, j, k) : edge_total<R>(t, eb, hadv);  // edgex_v
        } else if (q < nxy + nxz) {
            const int64_t r = q - nxy;
            const int i = (int)(r % (N[0] + 1)), j = (int)((r / (N[0] + 1)) % N[1]), k = (int)(r / ((int64_t)(N[0] + 1) * N[1]));
            const Taus<R> t = edge_taus<NS, R, NZ, 1, WL>(P, a.F, a.noise, i, j, k);
            edge_adv<NS, R, 1, WL>(P, a.F, i, j, k, ea, eb);
            a.ef[4](i, j, k) = WL ? edge_total_w<R, 1>(P, t, ea, hadv, i, j, k) : edge_total<R>(t, ea, hadv);  // edgez_u
            a.ef[1](i, j, k) = WL ? edge_total_w<R, 1>(P, t, eb, hadv, i, j, k) : edge_total<R>(t, eb, hadv);  // edgex_w
        } else if (q < nxy + nxz + nyz) {
            const int64_t r = q - nxy - nxz;
            const int i = (int)(r % N[0]), j = (int)((r / N[0]) % (N[1] + 1)), k = (int)(r / ((int64_t)N[0] * (N[1] + 1)));
            const Taus<R> t = edge_taus<NS, R, NZ, 2, WL>(P, a.F, a.noise, i, j, k);
            edge_adv<NS, R, 2, WL>(P, a.F, i, j, k, ea, eb);
            a.ef[5](i, j, k) = WL ? edge_total_w<R, 2>(P, t, ea, hadv, i, j, k) : edge_total<R>(t, ea, hadv);  // edgez_v
            a.ef[3](i, j, k) = WL ? edge_total_w<R, 2>(P, t, eb, hadv, i, j, k) : edge_total<R>(t, eb, hadv);  // edgey_w
        } else {
            const int64_t r = q - nxy - nxz - nyz;
            const int i = (int)(r % (N[0] + 2)) - 1, j = (int)((r / (N[0] + 2)) % (N[1] + 2)) - 1,
                      k = (int)(r / ((int64_t)(N[0] + 2) * (N[1] + 2))) - 1;
            const CellTaus<R> t = cell_taus<NS, R, NZ, WL>(P, a.F, a.noise, i, j, k);
#pragma unroll
            for (int d = 0; d < 3; ++d) a.cf[d](i, j, k) = cen_total_res<NS, R, NZ, WL>(P, a.F, a.noise, t, d, i, j, k);
        }
    }
}

// ===================================================================================
// noise fills and initial state
// ===================================================================================
// MultiFabFillRandomNormal body: value = mean + sd*z on the valid region, with z
// from the counter (canonical point, field = fid0 + comp, stream) -> periodic
// duplicates are equal (OverrideSync); ghosts by k_ghosts afterwards.
// MultiFabFillRandomUniform body (use_b = 2): a uniform in [0, 1) with 53 random
// bits, 27 from the first and 26 from the second word of one Philox call on the
// counter (canonical point, field = fid0 + comp, stream).
struct NoiseFillArgs {
    RunParams P;
    Arr4<double> f;
    int vx, vy, vz;   // extents of the filled box
    int ox, oy, oz;   // its low corner (0, or -1 to take the ghost layer of a wall direction)
    int c0, nc;
    double mean, sd;
    uint32_t fid0;
    int use_b;        // 0: z_A of the field's pair, 1: z_B, 2: the uniform
};

FHD_D double uniform53(uint32_t w0, uint32_t w1) {
    return ((double)(w0 >> 5) * 67108864.0 + (double)(w1 >> 6)) * (1.0 / 9007199254740992.0);
}
static __global__ void k_noise_fill(NoiseFillArgs a) {
    const int64_t tot = (int64_t)a.vx * a.vy * a.vz * a.nc;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < tot; q += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(q % a.vx) + a.ox, j = (int)((q / a.vx) % a.vy) + a.oy,
                  k = (int)((q / ((int64_t)a.vx * a.vy)) % a.vz) + a.oz;
        const int c = (int)(q / ((int64_t)a.vx * a.vy * a.vz));
        if (a.use_b == 2) {
            uint32_t w[4] = {canon(a.P, i, j, k), a.fid0 + (uint32_t)c, (uint32_t)a.P.step, (uint32_t)(a.P.step >> 32)};
            philox4x32_10(w, a.P.key0, a.P.key1);
            a.f(i, j, k, a.c0 + c) = uniform53(w[0], w[1]);
            continue;
        }
        float za, zb;
        normal_pair(a.P.key0, a.P.key1, canon(a.P, i, j, k), a.fid0 + (uint32_t)c, a.P.step, za, zb);
        a.f(i, j, k, a.c0 + c) = a.mean + a.sd * (double)(a.use_b ? zb : za);
    }
}

struct InitArgs {
    double* cu;       // the fab's first element
    int64_t sn, npts; // component stride; points of one component (whole fab incl. ghosts)
    int nvars, ns;
    double rho0, rhoE, rhoY[MAXS];
};
static __global__ void k_init_uniform(InitArgs a) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < a.npts; q += (int64_t)gridDim.x * blockDim.x) {
        double* p = a.cu + q;
        p[0] = a.rho0;
        p[a.sn] = 0.0;
        p[2 * a.sn] = 0.0;
        p[3 * a.sn] = 0.0;
        p[4 * a.sn] = a.rhoE;
        for (int s = 0; s < a.ns; ++s) p[(5 + s) * a.sn] = a.rhoY[s];
    }
}

// ===================================================================================
// batched launches: one launch covers the work items of every member of an
// ensemble; block b belongs to the member m with bpref[m] <= b < bpref[m+1].  After the
// nmem + 1 prefixes come the members of blocks 0, 64, 128, ...: a block starts there and
// steps to its own (boxes of 64 and more blocks: at most one step), where a binary
// search made log2(members) dependent loads before the block could start.
// ===================================================================================
FHD_D int member_of(const int* __restrict__ bpref, int nmem) {
    const int b = blockIdx.x;
    int m = __ldg(bpref + nmem + 1 + (b >> 6));
    while (__ldg(bpref + m + 1) <= b) ++m;
    return m;
}

// The member's argument block, copied once per block into shared memory (every
// thread of a block belongs to the same member): the bodies then read pointers,
// strides and run constants with shared loads on demand instead of holding what
// they read from global memory in registers.
template <class A>
FHD_D const A& member_args(const A* __restrict__ args, int m) {
    static_assert(sizeof(A) % 16 == 0, "argument blocks are copied in 16-byte words");
    __shared__ A sa;
    const uint4* src = reinterpret_cast<const uint4*>(args + m);
    uint4* dst = reinterpret_cast<uint4*>(&sa);
    for (int w = threadIdx.x; w < (int)(sizeof(A) / 16); w += blockDim.x) dst[w] = src[w];
    __syncthreads();
    return sa;
}

template <int NS, class R>
static __global__ void __launch_bounds__(128, cellprep_min_blocks<NS, R>()) k_cellprep_b(const PrepArgs<NS, R>* __restrict__ args,
                                                    const int* __restrict__ bpref, int nmem) {
    const int m = member_of(bpref, nmem);
    const PrepArgs<NS, R>& a = member_args(args, m);
    const int q = (blockIdx.x - bpref[m]) * blockDim.x + threadIdx.x;
    if (q < cellprep_count(a)) cellprep_point(a, q);
}

// 64 registers (8 blocks of 128 per SM): uncapped, the FP32 kernel took 96 and ran 20 warps per SM
template <int NS, class R, int NZ>
static __global__ void __launch_bounds__(128, 8) k_taus_b(const StageArgs<NS, R, NZ, true>* __restrict__ args,
                                                const int* __restrict__ bpref, int nmem) {
    const int m = member_of(bpref, nmem);
    const StageArgs<NS, R, NZ, true>& a = member_args(args, m);
    const int q = (blockIdx.x - bpref[m]) * blockDim.x + threadIdx.x;
    if (q < taus_count(a)) taus_point(a, q);
}

// Register cap of the batched face kernel: MINB resident blocks of 128 threads
// (8: 64 registers, 6: 80, 4: 128), picked per batch by its autotuner.
template <int NS, class R, int NZ, int MINB>
static __global__ void __launch_bounds__(128, MINB) k_faces_b(const StageArgs<NS, R, NZ, true>* __restrict__ args,
                                                   const int* __restrict__ bpref, int nmem, int d) {
    const int m = member_of(bpref, nmem);
    const StageArgs<NS, R, NZ, true>& a = member_args(args, m);
    const int q = (blockIdx.x - bpref[m]) * blockDim.x + threadIdx.x;
    if (q < faces_count(a, d)) faces_point(a, d, q);
}

// 64 registers (8 blocks per SM; fewer spill)
template <int NS, class R, int NZ>
static __global__ void __launch_bounds__(128, 8) k_update_b(const StageArgs<NS, R, NZ, true>* __restrict__ args,
                                                  const int* __restrict__ bpref, int nmem) {
    const int m = member_of(bpref, nmem);
    const StageArgs<NS, R, NZ, true>& a = member_args(args, m);
    const int q = (blockIdx.x - bpref[m]) * blockDim.x + threadIdx.x;
    if (q < update_count(a)) update_point(a, q);
}

template <int NS>
static __global__ void __launch_bounds__(128) k_convert_b(const ConvArgs<NS>* __restrict__ args,
                                                   const int* __restrict__ bpref, int nmem) {
    const int m = member_of(bpref, nmem);
    const ConvArgs<NS>& a = member_args(args, m);
    const int q = (blockIdx.x - bpref[m]) * blockDim.x + threadIdx.x;
    if (q < convert_count(a)) convert_point<true>(a, q);
}

static __global__ void __launch_bounds__(256) k_ghosts_b(const GhostFab* __restrict__ fabs,
                                                         const int* __restrict__ bpref, int nfab) {
    const int m = member_of(bpref, nfab);
    const GhostFab& f = fabs[m];
    const int q = (blockIdx.x - bpref[m]) * blockDim.x + threadIdx.x;
    if (q < f.npts * f.nc) ghost_point(f, q);
}

// ===================================================================================
// persistent batched step: one launch runs every phase of one RK3 step for every
// member.  Phases per member: for each stage cellprep, stresses, faces x / y / z,
// update, ghost fill; then the conversion, its ghost fill and the step counter (no ghost
// fills when the update and the conversion store the images).
// Work is cut into chunks of `chunk` items; a unit is one member's (or one ghost
// fab's) part of a phase.  Blocks take chunks in order from one counter (phase-
// major over members) and, before working on a chunk of phase p > 0, wait until
// every chunk of the member's phase p - 1 is done.  A block only ever waits on
// chunks taken before its own, by blocks that are running, so the order cannot
// deadlock; every wait is still bounded in time (limit_ns): on expiry the block
// marks the member FHD_ERR_TIMEOUT, raises the abort flag and all blocks stop
// taking work.
// ===================================================================================
FHD_D unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// bounded wait for every chunk of member m's phase p; 1 when done, 0 on abort or expiry
FHD_D int wait_phase(const PersistArgs& a, int m, int p) {
    volatile const unsigned int* d = a.done + (size_t)m * a.nphase + p;
    const unsigned int target = a.need[(size_t)m * a.nphase + p];
    const unsigned long long t0 = global_ns();
    for (;;) {
        if (*d >= target) {
            __threadfence();
            return 1;
        }
        if (*reinterpret_cast<volatile int*>(a.abort)) return 0;
        if (global_ns() - t0 > a.limit_ns) {
            atomicCAS(a.status + m, 0, ST_TIMEOUT);
            atomicExch(a.abort, 1);
            return 0;
        }
        __nanosleep(256);
    }
}

template <int NS, class R, int NZ>
struct PersistBytes {
    static constexpr size_t a = sizeof(PrepArgs<NS, R>), b = sizeof(StageArgs<NS, R, NZ, true>), c = sizeof(ConvArgs<NS>),
                            d = sizeof(GhostFab);
    static constexpr size_t m1 = a > b ? a : b, m2 = c > d ? c : d;
    static constexpr size_t value = ((m1 > m2 ? m1 : m2) + 7) / 8 * 8;
};

template <int NS, class R, int NZ, int MINB>
static __global__ void __launch_bounds__(128, MINB) k_batch_persist(PersistArgs a) {
    __shared__ __align__(16) unsigned long long sbuf[PersistBytes<NS, R, NZ>::value / 8];
    __shared__ int s_unit, s_go, s_end;
    __shared__ long long s_chunk;
    for (;;) {
        if (threadIdx.x == 0) {
            long long I = -1;
            if (!*reinterpret_cast<volatile int*>(a.abort)) I = (long long)atomicAdd(a.next, 1u);
            const int end = I < 0 || I >= a.total;
            int u = 0, go = 0;
            if (!end) {
                int lo = 0, hi = a.nunits;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (a.units[mid].first <= I) lo = mid;
                    else hi = mid;
                }
                u = lo;
                const PUnit& pu = a.units[u];
                go = pu.phase == 0 ? 1 : wait_phase(a, pu.member, pu.phase - 1);
                s_chunk = I - pu.first;
            }
            s_unit = u;
            s_go = go;
            s_end = end;
        }
        __syncthreads();
        if (s_end) break;
        const PUnit& pu = a.units[s_unit];
        const int kind = pu.kind;
        if (s_go) {
            if (kind != PK_STEP) {
                const size_t bytes = kind == PK_PREP ? sizeof(PrepArgs<NS, R>)
                                     : kind == PK_CONVERT ? sizeof(ConvArgs<NS>)
                                     : kind == PK_GHOST ? sizeof(GhostFab) : sizeof(StageArgs<NS, R, NZ, true>);
                const unsigned long long* src = static_cast<const unsigned long long*>(pu.args);
                for (int w = threadIdx.x; w < (int)((bytes + 7) / 8); w += blockDim.x) sbuf[w] = src[w];
            }
            __syncthreads();
            const int64_t q0 = s_chunk * a.chunk;
            const int64_t q1 = q0 + a.chunk < pu.items ? q0 + a.chunk : pu.items;
            const int64_t q = q0 + threadIdx.x;
            const int st = blockDim.x;
            switch (kind) {
                case PK_PREP: {
                    const auto& A = *reinterpret_cast<const PrepArgs<NS, R>*>(sbuf);
                    for (int64_t x = q; x < q1; x += st) cellprep_point(A, (int)x);
                } break;
                case PK_TAUS: {
                    const auto& A = *reinterpret_cast<const StageArgs<NS, R, NZ, true>*>(sbuf);
                    for (int64_t x = q; x < q1; x += st) taus_point(A, (int)x);
                } break;
                case PK_FACEX: {
                    const auto& A = *reinterpret_cast<const StageArgs<NS, R, NZ, true>*>(sbuf);
                    for (int64_t x = q; x < q1; x += st) faces_point(A, 0, (int)x);
                } break;
                case PK_FACEY: {
                    const auto& A = *reinterpret_cast<const StageArgs<NS, R, NZ, true>*>(sbuf);
                    for (int64_t x = q; x < q1; x += st) faces_point(A, 1, (int)x);
                } break;
                case PK_FACEZ: {
                    const auto& A = *reinterpret_cast<const StageArgs<NS, R, NZ, true>*>(sbuf);
                    for (int64_t x = q; x < q1; x += st) faces_point(A, 2, (int)x);
                } break;
                case PK_UPDATE: {
                    const auto& A = *reinterpret_cast<const StageArgs<NS, R, NZ, true>*>(sbuf);
                    for (int64_t x = q; x < q1; x += st) update_point(A, (int)x);
                } break;
                case PK_CONVERT: {
                    const auto& A = *reinterpret_cast<const ConvArgs<NS>*>(sbuf);
                    for (int64_t x = q; x < q1; x += st) convert_point<true>(A, (int)x);
                } break;
                case PK_GHOST: {
                    const auto& G = *reinterpret_cast<const GhostFab*>(sbuf);
                    for (int64_t x = q; x < q1; x += st) ghost_point(G, (int)x);
                } break;
                default:
                    if (threadIdx.x == 0) a.steps[pu.member] += 1;
                    break;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && s_go && pu.phase != a.hold_phase) {
            __threadfence();
            atomicAdd(a.done + (size_t)pu.member * a.nphase + pu.phase, 1u);
        }
    }
}

static __global__ void k_steps_set(uint64_t* step, uint64_t v) { *step = v; }

static __global__ void k_steps_inc(uint64_t* steps, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) steps[i] += 1;
}

}  // namespace fhd
