// fhd_launch.cuh — templated launchers included by each kernel translation unit.
#pragma once
#include <atomic>

#include "fhd_host.h"
#include "fhd_kernels.cuh"
#include "fhd_fused.cuh"
#include "fhd_walls.cuh"

namespace fhd {

template <class T>
inline Arr4<T> view(const fhd_fab& f, int comp0 = 0) {
    Arr4<T> a;
    const int64_t nx = f.hi[0] - f.lo[0] + 1, ny = f.hi[1] - f.lo[1] + 1, nz = f.hi[2] - f.lo[2] + 1;
    a.sy = nx;
    a.sz = nx * ny;
    a.sn = nx * ny * nz;
    a.p = f.data ? static_cast<T*>(f.data) + comp0 * a.sn - (f.lo[0] + f.lo[1] * nx + f.lo[2] * nx * ny) : nullptr;
    return a;
}

// Grid of a grid-stride kernel: as many blocks as the SMs hold at once (the kernel's
// occupancy at this block size, queried once per kernel and block size), so that
// every block runs from the start and all finish together instead of leaving a
// partly filled last wave; fewer when there is less work.
inline int device_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) {
            cudaGetLastError();
            sms = 148;
        }
    }
    return sms;
}

template <auto K>
inline int resident_blocks(int block) {
    static int cache[3] = {0, 0, 0};  // block sizes 128, 256, other
    const int slot = block == 128 ? 0 : (block == 256 ? 1 : 2);
    if (slot == 2 || !cache[slot]) {
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, K, block, 0) != cudaSuccess || nb < 1) {
            cudaGetLastError();
            nb = 1;
        }
        if (slot == 2) return nb * device_sms();
        cache[slot] = nb * device_sms();
    }
    return cache[slot];
}

template <auto K>
inline int resident_grid(int64_t items, int block) {
    int64_t g = (items + block - 1) / block;
    const int cap = resident_blocks<K>(block);
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

// Blocks per direction of the face kernel: together as many as the SMs hold at once, each
// over several chunks of its direction.  Quasi-1-D and 2-D runs (dim < 3): a block per chunk.
// Their transverse faces cost next to nothing, so the blocks of those directions end early
// and would leave the others' on a third (two thirds) of the SMs: faces per step, 256^3
// argon, 1-D 6.9 against 12.9 ms, 2-D 10.2 against 12.9; 128x96x80 with four species, 1-D 1.29
// against 2.74, 2-D 2.16 against 2.82.
template <auto K>
inline int face_grid(const int N[3], int block, int dim) {
    int64_t most = 0;
    for (int d = 0; d < 3; ++d) {
        const int64_t f = (int64_t)(N[0] + (d == 0)) * (N[1] + (d == 1)) * (N[2] + (d == 2));
        if (f > most) most = f;
    }
    int64_t g = (most + block - 1) / block;
    const int cap = resident_blocks<K>(block) / 3;
    if (dim == 3 && g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

// opts a kernel into dynamic shared memory above 48 KiB on the current device, once per
// device, and returns the blocks its SMs hold at once with it (0: not available)
template <auto K>
inline int staged_blocks(int block, int bytes) {
    static std::atomic<int> blocks[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return 0; }
    int nb = blocks[dev].load(std::memory_order_relaxed);
    if (!nb) {
        if (cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, K, block, bytes) != cudaSuccess || nb < 1) {
            cudaGetLastError();
            return 0;
        }
        nb *= device_sms();
        blocks[dev].store(nb, std::memory_order_relaxed);
    }
    return nb;
}

inline int grid_for(int64_t items, int block, int cap = 148 * 32) {
    int64_t g = (items + block - 1) / block;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

inline int cuda_rc(cudaError_t e) { return e == cudaSuccess ? FHD_OK : FHD_ERR_CUDA; }

template <int NS, class R>
Fields<NS, R> make_fields(const StageCall& c) {
    Fields<NS, R> F;
    F.cons = view<const double>(c.cons_s);
    for (int d = 0; d < 3; ++d) {
        F.mom[d] = view<const double>(c.mom_s[d]);
        F.vel[d] = view<const double>(c.vel[d]);
    }
    F.pr = view<const double>(c.pr);
    F.pT = c.pT;
    F.eta = view<const R>(c.eta);
    F.zeta = view<const R>(c.zeta);
    F.kappa = view<const R>(c.kappa);
    F.chi = view<const R>(c.chi);
    F.D = view<const R>(c.D);
    return F;
}

// the cell records of a packed stage (c.rec: their first word and geometry)
template <int NS, class R>
Rec<NS, R> make_rec(const StageCall& c) {
    const Arr4<const Vec<R>> v = view<const Vec<R>>(c.rec);
    return Rec<NS, R>{c.pack ? v.p : nullptr, v.sy, v.sz, v.sn};
}

template <int NS, class R>
FieldsPack<NS, R> make_fields_pack(const StageCall& c) {
    FieldsPack<NS, R> F;
    F.q = make_rec<NS, R>(c);
    F.cons = view<const double>(c.cons_s);
    for (int d = 0; d < 3; ++d) {
        F.mom[d] = view<const double>(c.mom_s[d]);
        F.vel[d] = view<const double>(c.vel[d]);
    }
    F.pr = view<const double>(c.pr);
    F.pT = c.pT;
    F.zr = R(c.P.zeta_ratio);
    return F;
}

template <int MODE>
Noise<MODE> make_noise(const StageCall& c) {
    Noise<MODE> n;
    n.w = c.w;
    if constexpr (MODE == NZ_W || MODE == NZ_AB) for (int d = 0; d < 3; ++d) {
        n.a.fa[d] = view<const double>(c.nz.fa[d]);
        n.a.fb[d] = view<const double>(c.nz.fb[d]);
        n.a.foa[d] = c.nz.fa[d].ncomp - (c.P.ns + 1);
        n.a.fob[d] = c.nz.fb[d].ncomp - (c.P.ns + 1);
        n.a.ea[d] = view<const double>(c.nz.ea[d]);
        n.a.eb[d] = view<const double>(c.nz.eb[d]);
        n.a.ca[d] = view<const double>(c.nz.ca[d]);
        n.a.cb[d] = view<const double>(c.nz.cb[d]);
    }
    return n;
}

template <int NS, class R>
PrepArgs<NS, R> make_prep_args(const StageCall& c) {
    PrepArgs<NS, R> a;
    a.P = c.P;
    a.cons = view<const double>(c.cons_s);
    for (int d = 0; d < 3; ++d) {
        a.mom[d] = view<const double>(c.mom_s[d]);
        a.vel[d] = view<double>(c.vel[d]);
    }
    a.pr = view<double>(c.pr, c.pT);
    a.eta = view<R>(c.eta);
    a.zeta = view<R>(c.zeta);
    a.kappa = view<R>(c.kappa);
    a.chi = view<R>(c.chi);
    a.D = view<R>(c.D);
    const Rec<NS, R> q = make_rec<NS, R>(c);
    a.q = const_cast<Vec<R>*>(q.p);
    a.qsy = q.sy;
    a.qsz = q.sz;
    a.qsn = q.sn;
    a.prim = c.pack ? c.wprim : 2;
    a.coef = c.pack ? c.wcoef : 1;
    a.it = make_items(c.P.n[0] + 3, c.P.n[1] + 3, c.P.n[2] + 3);
    a.status = c.status;
    return a;
}

template <int NS, class R>
int launch_cellprep(const StageCall& c) {
    const PrepArgs<NS, R> a = make_prep_args<NS, R>(c);
    // (an occupancy-sized grid was measured slower here: blocks beyond the resident
    // set rebalance this kernel's uneven per-cell cost)
    k_cellprep<NS, R><<<grid_for(a.it.n, 128), 128, 0, c.stream>>>(a);
    return cuda_rc(cudaGetLastError());
}

// launch shapes available to the autotuner: block size of the stage kernels and
// the register cap of the face-flux kernel (minimum resident blocks per SM)
constexpr int kStageBlocks[] = {128, 256, 128, 128, 128};
constexpr int kFaceMinBlocks[] = {4, 2, 6, 10, 8};  // as instantiated in launch_stage_part_t
constexpr int kNumStageBlocks = 5;
// the fused stage kernel (k_stage_zm): tile of 16 x 8 cells; per fused tile the
// block size (128, 256 or 384 threads over the same tile) and the z-chunk depth
constexpr int kZmTX = 16, kZmTY = 8;
constexpr int kZmThreads[] = {128, 256, 256, 384};
constexpr int kZmChunks[] = {32, 32, 64, 32};
constexpr int kNumZmTiles = 4;
inline bool tile_is_fused(int t) { return t >= kNumStageBlocks && t < kNumStageBlocks + kNumZmTiles; }

template <class T>
int step_of(const Arr4<T>& a, int d) { return d == 0 ? 1 : (d == 1 ? a.sy : a.sz); }

// the face kernel's operands from the stage's views
template <int NS, class R, int NZ, bool PACK>
void make_face_args(StageArgs<NS, R, NZ, PACK>& a, const int n[3]) {
    const auto& F = a.F;
    auto& f = a.fi;
    // (a fab that the stage does not have has no views: its pointers stay null)
    auto comp = [](const auto& v, int c) { return v.p ? v.p + (int64_t)c * v.sn : nullptr; };
    f.T = comp(F.pr, F.pT);
    f.p = comp(F.pr, F.pT + 1);
    f.E = comp(F.cons, 4);
    for (int s = 0; s < NS; ++s) {
        f.Y[s] = comp(F.pr, F.pT + 2 + s);
        f.rY[s] = comp(F.cons, 5 + s);
    }
    f.psy = F.pr.sy;    f.psz = F.pr.sz;
    f.csy = F.cons.sy;  f.csz = F.cons.sz;
    f.tsy = a.S.ct.sy;  f.tsz = a.S.ct.sz;
    f.esy = a.S.et.sy;  f.esz = a.S.et.sz;
    if constexpr (!PACK) {
        f.kappa = F.kappa.p;
        for (int s = 0; s < NS; ++s) {
            f.X[s] = comp(F.pr, F.pT + 2 + NS + s);
            f.chi[s] = comp(F.chi, s);
        }
        for (int s = 0; s < NS * NS; ++s) f.D[s] = comp(F.D, s);
        f.ksy = F.kappa.sy; f.ksz = F.kappa.sz;
        f.hsy = F.chi.sy;   f.hsz = F.chi.sz;
        f.dsy = F.D.sy;     f.dsz = F.D.sz;
    }
    for (int d = 0; d < 3; ++d) {
        auto& x = a.fd[d];
        x.u = F.vel[d].p;  x.usy = F.vel[d].sy; x.usz = F.vel[d].sz;
        x.m = F.mom[d].p;  x.msy = F.mom[d].sy; x.msz = F.mom[d].sz;
        x.cs = comp(a.S.ct, d);
        x.cd = PACK ? nullptr : comp(a.S.ct, 3 + d);
        x.td = step_of(a.S.ct, d);
        x.pd = step_of(F.pr, d);
        x.cd_ = step_of(F.cons, d);
        x.kd = x.hd = x.dd = x.qd = 0;
        if constexpr (PACK) {
            x.qd = d == 0 ? 1 : (d == 1 ? F.q.sy : F.q.sz);
        } else {
            x.kd = step_of(F.kappa, d);
            x.hd = step_of(F.chi, d);
            x.dd = step_of(F.D, d);
        }
        // transverse directions and their edges: x (y on xy, z on xz), y (x on xy, z
        // on yz), z (x on xz, y on yz)
        const int t[2] = {d == 0 ? 1 : 0, d == 2 ? 1 : 2};
        for (int q = 0; q < 2; ++q) {
            const int e = d + t[q] == 1 ? 0 : (d + t[q] == 2 ? 1 : 2);
            auto& g = x.f[q];
            g.s = comp(a.S.et, PACK ? e : 2 * e);
            g.d = PACK ? nullptr : comp(a.S.et, 2 * e + 1);
            g.eq = step_of(a.S.et, t[q]);
            g.v = F.vel[t[q]].p;
            g.vsy = F.vel[t[q]].sy;
            g.vsz = F.vel[t[q]].sz;
            g.vq = step_of(F.vel[t[q]], t[q]);
            g.vd = step_of(F.vel[t[q]], d);
        }
        x.it = make_items(n[0] + (d == 0), n[1] + (d == 1), n[2] + (d == 2));
    }
}

template <int NS, class R, int NZ, bool PACK>
StageArgs<NS, R, NZ, PACK> make_stage_args(const StageCall& c) {
    StageArgs<NS, R, NZ, PACK> a;
    a.P = c.P;
    if constexpr (PACK) a.F = make_fields_pack<NS, R>(c);
    else a.F = make_fields<NS, R>(c);
    a.noise = make_noise<NZ>(c);
    a.mc = view<double>(c.smc);
    if constexpr (PACK) {
        // the same buffers with words of two (StageScratch): half the components
        a.S.ct = view<Pair<R>>(c.ct);
        a.S.et = view<Pair<R>>(c.et);
        a.S.me = view<double2>(c.sme);
        for (int d = 0; d < 3; ++d) {
            a.S.ff[d] = view<double2>(c.sff[d]);
            fhd_fab last = c.sff[d];
            last.data = static_cast<double*>(last.data) + (int64_t)2 * ((2 + NS) / 2) * a.S.ff[d].sn;
            a.S.fl[d] = view<double>(last);
        }
    } else {
        a.S.ct = view<R>(c.ct);
        a.S.et = view<R>(c.et);
        a.S.me = view<double>(c.sme);
        for (int d = 0; d < 3; ++d) a.S.ff[d] = view<double>(c.sff[d]);
    }
    for (int d = 0; d < 3; ++d) {
        a.mom0[d] = view<const double>(c.mom0[d]);
        a.mom_o[d] = view<double>(c.mom_o[d]);
    }
    a.cons0 = view<const double>(c.cons0);
    a.cons_o = view<double>(c.cons_o);
    a.src = view<const double>(c.src);
    a.stage = c.stage;
    a.img = c.img;
    const int* n = c.P.n;
    a.it_taus = make_items(n[0] + 2, n[1] + 2, n[2] + 2);
    a.it_upd = make_items(n[0] + 1, n[1] + 1, n[2] + 1);
    make_face_args(a, n);
    return a;
}

// The face kernel's launch shape when none was set (fhd_set_tile).  The kernel is
// bound by latency and issue, so resident warps count until spills cost more
// (us per step, all kernels, unless ms):
//   * faces that fit one wave of 128-register blocks (4 per SM; up to about 29^3) take
//     them: with no second wave, more residency buys nothing and spills cost (argon FP64
//     24^3 88.2 against 90.8 at 64 registers; 32^3 110.8 against 102.6);
//   * up to one wave of 80-register blocks (about 33^3): 32^3, faces alone, 44.6 against 47.5
//     at 64 registers; 40^3 138.5 against 135.9;
//   * above, 64 registers (argon FP64 48^3 191 against 213 at 128 registers, 128^3 2905
//     against 2933 at 80; mixed 128^3 1908 against 1975 at 80; four species FP64 64^3 803
//     against 841, mixed 405 against 418), with two exceptions: 48 for one species (96^3
//     FP64 703 against 732, mixed 632 against 644), and 80 for three and four species in
//     mixed precision beyond about 108^3 (100^3 1441 against 1408, 128^3 2940 against
//     3014).
template <int NS, class R>
int auto_face_tile(const int N[3]) {
    int64_t most = 0;
    for (int d = 0; d < 3; ++d) {
        const int64_t f = (int64_t)(N[0] + (d == 0)) * (N[1] + (d == 1)) * (N[2] + (d == 2));
        if (f > most) most = f;
    }
    const int64_t blocks = 3 * ((most + 127) / 128);
    if (blocks <= 4 * device_sms()) return 0;
    if (blocks <= 6 * device_sms()) return 2;
    if (NS == 1) return 3;
    return sizeof(R) == 4 && NS >= 3 && blocks > 200 * device_sms() ? 2 : 4;
}

inline int stage_block(const StageCall& c) {
    return (c.tile >= 0 && c.tile < kNumStageBlocks) ? kStageBlocks[c.tile] : 128;
}

// Up to 4 blocks of points per SM (about 42^3) the launch's time is one thread's chain of
// loads and FP64 operations: four threads per point cut it (argon FP64, per step: 16^3 30.6
// against 38.3 us with one, 32^3 32.4 against 38.6, 40^3 38.3 against 42.2; 44^3 44.3 against
// 43.2, 64^3 91 against 83, 128^3 512 against 393: there the kernel streams).  Four
// species and the mixed path alike (16^3 31.6 against 41.7 and 25.2 against 36.6 us, 40^3
// 44.0 against 46.1 and 37.6 against 37.4).  Not packed
// (walls, low dimensions, allocation-free) a small box takes one thread with all the
// registers it wants.
template <int NS, class R, int NZ, bool PACK>
void launch_update(const StageArgs<NS, R, NZ, PACK>& a, cudaStream_t s) {
    const int blocks = (a.it_upd.n + 127) / 128;
    constexpr int MB = !PACK ? 16 : (NS <= 2 ? 12 : 10);
    if (blocks > 4 * device_sms()) {
        k_update<NS, R, NZ, MB, PACK><<<resident_grid<k_update<NS, R, NZ, MB, PACK>>(a.it_upd.n, 128), 128, 0, s>>>(a);
    } else {
        if constexpr (PACK) k_update_split<NS, R, NZ><<<4 * blocks, 128, 0, s>>>(a);
        else k_update<NS, R, NZ, 4, PACK><<<blocks, 128, 0, s>>>(a);
    }
}

// part: 0 stresses, 1 face fluxes (all three directions), 2 update
template <int NS, class R, int NZ>
int launch_stage_part_t(const StageCall& c, int part) {
    const StageArgs<NS, R, NZ, true> a = make_stage_args<NS, R, NZ, true>(c);
    const int b = stage_block(c);
    if (part == 0) {
        // Staged up to five waves of its blocks (about 76^3): 16^3 argon FP64 26.1 against
        // 38.6 us per step, 64^3 75.0 against 87.5, 72^3 103.9 against 116.9; even at 80^3
        // (143); beyond, L1 holds more of the neighbours' operands than the columns leave
        // of it, 88^3 184 against 181, 128^3 535 against 511.  The same line for the other
        // species counts (16^3 25.7 against 38 us, 64^3 69 to 81 against 83 to 93) and in
        // mixed precision (24.7 to 25.8 against 35 to 36; 61 to 66 against 74 to 77).
        // Without noise there is less to overlap: mixed, 64^3 56 against 53 and 72^3 78
        // against 68, 3 % of those steps at most.
        constexpr auto S = k_taus_staged<NS, R, NZ>;
        constexpr int bytes = TausStage<NS, R>::bytes;
        const int wave = staged_blocks<S>(kStagedThreads, bytes);
        const int need = (a.it_taus.n + kStagedThreads - 1) / kStagedThreads;
        if (need <= 5 * wave)
            S<<<need < wave ? need : wave, kStagedThreads, bytes, c.stream>>>(a);
        else
            k_taus<NS, R, NZ, false, false, true><<<grid_for(a.it_taus.n, b), b, 0, c.stream>>>(a, StageAux<false>{});
    } else if (part == 1) {
        const int t = (c.tile >= 0 && c.tile < kNumStageBlocks) ? c.tile : auto_face_tile<NS, R>(c.P.n);
#define FHD_FACES(BS, MINB)                                                                             \
        {                                                                                               \
            constexpr auto K = k_faces<NS, R, NZ, BS, MINB, false, false, true>;                        \
            const int per = face_grid<K>(c.P.n, BS, 3);                                                 \
            K<<<3 * per, BS, 0, c.stream>>>(a, per, StageAux<false>{});                                 \
        }
        switch (t) {
            case 0: FHD_FACES(128, 4) break;
            case 1: FHD_FACES(256, 2) break;
            case 2: FHD_FACES(128, 6) break;
            case 3: FHD_FACES(128, 10) break;
            default: FHD_FACES(128, 8) break;
        }
#undef FHD_FACES
    } else {
        launch_update(a, c.stream);
    }
    return cuda_rc(cudaGetLastError());
}

// the same without packed operands, for the allocation-free step: its 16 MiB of static
// scratch hold the boxes that they were sized for only without the records.  FP64,
// small boxes.
template <int NS, int NZ>
int launch_stage_plain_t(const StageCall& c, int part) {
    const StageArgs<NS, double, NZ> a = make_stage_args<NS, double, NZ, false>(c);
    if (part == 0) {
        k_taus<NS, double, NZ><<<grid_for(a.it_taus.n, 128), 128, 0, c.stream>>>(a, StageAux<false>{});
    } else if (part == 1) {
        constexpr auto K = k_faces<NS, double, NZ, 128, 4>;
        const int per = face_grid<K>(c.P.n, 128, 3);
        K<<<3 * per, 128, 0, c.stream>>>(a, per, StageAux<false>{});
    } else {
        launch_update(a, c.stream);
    }
    return cuda_rc(cudaGetLastError());
}

// resident blocks per SM asked of the register allocator: the shared memory of a
// 16 x 8 tile (56-80 KB) holds 2-4 blocks per SM
template <int NS, class R>
constexpr int zm_min_blocks(int bt) {
    return bt == 128 ? (sizeof(R) == 8 ? (NS <= 2 ? 3 : 2) : (NS <= 2 ? 4 : 3)) : (bt == 256 ? (NS <= 2 ? 3 : 2) : 2);
}

template <int NS, class R, int NZ, int BT>
int launch_stage_zm_bt(const StageCall& c, int zc) {
    constexpr int TX = kZmTX, TY = kZmTY;
    constexpr size_t smem = ZmSmem<NS, R, TX, TY>::bytes;
    auto kern = k_stage_zm<NS, R, NZ, TX, TY, BT, zm_min_blocks<NS, R>(BT)>;
    // the dynamic shared memory above 48 KiB is opted into per device, once
    static bool set[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return FHD_ERR_CUDA; }
    if (dev < 0 || dev >= 64) return FHD_ERR_UNSUPPORTED;
    if (!set[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return FHD_ERR_CUDA;
        }
        set[dev] = true;
    }
    const StageArgs<NS, R, NZ> a = make_stage_args<NS, R, NZ, false>(c);
    const int* N = c.P.n;
    const dim3 grid((N[0] + TX - 1) / TX, (N[1] + TY - 1) / TY, (N[2] + zc - 1) / zc);
    kern<<<grid, BT, smem, c.stream>>>(a, zc);
    return cuda_rc(cudaGetLastError());
}

template <int NS, class R, int NZ>
int launch_stage_zm_t(const StageCall& c) {
    const int t = tile_is_fused(c.tile) ? c.tile - kNumStageBlocks : 0;
    switch (kZmThreads[t]) {
        case 256: return launch_stage_zm_bt<NS, R, NZ, 256>(c, kZmChunks[t]);
        case 384: return launch_stage_zm_bt<NS, R, NZ, 384>(c, kZmChunks[t]);
        default: return launch_stage_zm_bt<NS, R, NZ, 128>(c, kZmChunks[t]);
    }
}

// the stress (part 0) and face (part 1) launches of a stage whose fluxes the caller
// wants (StageAux), and of the flux operator, whose StageCall has no stage scratch but
// the stresses
template <int NS, int NZ, bool WL, bool PACK>
int launch_aux_stage_t(const StageCall& c, int part) {
    const StageArgs<NS, double, NZ, PACK> a = make_stage_args<NS, double, NZ, PACK>(c);
    StageAux<true> x;
    for (int d = 0; d < 3; ++d) {
        x.ff[d] = view<double>(c.ff[d]);
        x.cf[d] = view<double>(c.cf[d]);
    }
    for (int e = 0; e < 6; ++e) x.ef[e] = view<double>(c.ef[e]);
    if (part == 0) {
        k_taus<NS, double, NZ, WL, true, PACK><<<grid_for(a.it_taus.n, 128), 128, 0, c.stream>>>(a, x);
    } else {
        constexpr auto K = k_faces<NS, double, NZ, 128, (WL && NS > 2 ? 4 : 8), WL, true, PACK>;
        const int per = face_grid<K>(c.P.n, 128, c.P.dim);
        K<<<3 * per, 128, 0, c.stream>>>(a, per, x);
    }
    return cuda_rc(cudaGetLastError());
}

// the stage parts of a box with physical walls (FP64, one launch shape): the wall
// variants of the stresses and face fluxes, and the common update
template <int NS, int NZ>
int launch_walls_part_t(const StageCall& c, int part) {
    const StageArgs<NS, double, NZ> a = make_stage_args<NS, double, NZ, false>(c);
    if (part == 0) {
        k_taus<NS, double, NZ, true><<<grid_for(a.it_taus.n, 128), 128, 0, c.stream>>>(a, StageAux<false>{});
    } else if (part == 1) {
        // register cap: 64 up to two species (the periodic autotuner's choice at 256^3;
        // 128 was measured twice as slow for the wall variant), 128 above
        constexpr int MB = NS <= 2 ? 8 : 4;
        const int per = face_grid<k_faces<NS, double, NZ, 128, MB, true>>(c.P.n, 128, c.P.dim);
        k_faces<NS, double, NZ, 128, MB, true><<<3 * per, 128, 0, c.stream>>>(a, per, StageAux<false>{});
    } else {
        launch_update(a, c.stream);
    }
    return cuda_rc(cudaGetLastError());
}

template <int NS>
int launch_walls_part(const StageCall& c, int part) {
    switch (c.mode) {
        case NM_OFF: return launch_walls_part_t<NS, NZ_OFF>(c, part);
        case NM_AB: return launch_walls_part_t<NS, NZ_AB>(c, part);
        case NM_PHILOX: return launch_walls_part_t<NS, NZ_PHILOX>(c, part);
        default: return FHD_ERR_BAD_ARG;
    }
}

// BCMassTempPress + BCRhoRhoE on the ghost cells of the wall directions
template <int NS>
int launch_bc_prim(const DevParams& P, const WallParams& W, const fhd_fab& prim, const fhd_fab& cons,
                   const fhd_fab mom[3], cudaStream_t s) {
    BcPrimArgs<NS> a;
    a.P = P;
    a.W = W;
    a.prim = view<double>(prim);
    a.cons = view<double>(cons);
    for (int d = 0; d < 3; ++d) a.mom[d] = view<const double>(mom[d]);
    const int g = -prim.lo[0];
    int blo[3], bhi[3], clo[3], chi[3];
    for (int d = 0; d < 3; ++d) {
        blo[d] = -g;
        bhi[d] = P.n[d] - 1 + g;
        const bool w = P.walls && !P.periodic[d];
        clo[d] = w ? 0 : blo[d];
        chi[d] = w ? P.n[d] - 1 : bhi[d];
    }
    a.sh = make_shell(blo, bhi, clo, chi);
    if (a.sh.n == 0) return FHD_OK;
    k_bc_prim<NS><<<grid_for(a.sh.n, 128), 128, 0, s>>>(a);
    return cuda_rc(cudaGetLastError());
}

// The reference's boundary passes in its order, one launch each (k_bc_pass):
// for each direction d BCMassTempPress (lo, hi) and BCMomNormal (lo, hi) of
// mom[d] / vel[d] when d has walls, and BCMomTrans of mom[d] / vel[d] across the
// other directions' walls (x lo, x hi, y lo, ...); with rre, BCRhoRhoE of every
// wall side after them (setBCStag); without, the passes RK3stepStag makes before
// the conversion.
template <int NS>
int launch_bc_seq(const DevParams& P, const WallParams& W, const fhd_fab& prim, const fhd_fab& cons,
                  const fhd_fab* mom, const fhd_fab* vel, bool rre, cudaStream_t st) {
    BcPassArgs<NS> a;
    a.P = P;
    a.W = W;
    a.prim = view<double>(prim);
    a.cons = view<double>(cons);
    a.mx = view<const double>(mom[0]);
    a.my = view<const double>(mom[1]);
    a.mz = view<const double>(mom[2]);
    const int g = -prim.lo[0], gm = -mom[0].lo[0];
    auto wall = [&](int d) { return P.walls && !P.periodic[d]; };
    auto launch = [&](int fn, int side, int c) {
        a.fn = fn;
        a.side = side;
        a.c = c;
        const int d = side >> 1, hi = side & 1;
        for (int e = 0; e < 3; ++e) {
            const bool cell = fn == BC_MTP || fn == BC_RRE;
            const int gg = cell ? g : gm;
            const int nod = (!cell && e == c) ? 1 : 0;
            a.blo[e] = -gg;
            a.bhi[e] = P.n[e] - 1 + nod + gg;
            if (e == d) {
                if (fn == BC_MOMN) { a.blo[e] = hi ? P.n[e] : -gg; a.bhi[e] = hi ? P.n[e] + gg : 0; }
                else { a.blo[e] = hi ? P.n[e] : -gg; a.bhi[e] = hi ? P.n[e] + gg - 1 : -1; }
            }
        }
        if (fn == BC_MOMN || fn == BC_MOMT) {
            a.mom = view<double>(mom[c]);
            a.vel = view<double>(vel[c]);
        }
        const int64_t tot = (int64_t)(a.bhi[0] - a.blo[0] + 1) * (a.bhi[1] - a.blo[1] + 1) * (a.bhi[2] - a.blo[2] + 1);
        k_bc_pass<NS><<<grid_for(tot, 128), 128, 0, st>>>(a);
        return cuda_rc(cudaGetLastError());
    };
    int rc = FHD_OK;
    // every direction d: its own sides' passes when it has walls, and BCMomTrans of
    // mom[d] / vel[d] across the other directions' walls in any case
    for (int d = 0; d < 3 && !rc; ++d) {
        for (int h = 0; h < 2 && !rc && wall(d); ++h) rc = launch(BC_MTP, 2 * d + h, d);
        for (int h = 0; h < 2 && !rc && wall(d); ++h) rc = launch(BC_MOMN, 2 * d + h, d);
        for (int e = 0; e < 3 && !rc; ++e) {
            if (e == d || !wall(e)) continue;
            for (int h = 0; h < 2 && !rc; ++h) rc = launch(BC_MOMT, 2 * e + h, d);
        }
    }
    for (int side = 0; side < 6 && rre && !rc; ++side)
        if (wall(side >> 1)) rc = launch(BC_RRE, side, 0);
    return rc;
}

// the particle reservoir's fluxes and momenta (k_reservoir), the flux reset of one
// reservoir side (k_res_reset)
template <int NS>
int launch_reservoir(const ResArgs& a, cudaStream_t s) {
    if (a.face_pref[a.nsides] == 0) return FHD_OK;
    k_reservoir<NS><<<grid_for(a.face_pref[a.nsides], 128), 128, 0, s>>>(a);
    return cuda_rc(cudaGetLastError());
}

template <int NS>
int launch_res_reset(const ResResetArgs& a, cudaStream_t s) {
    const int d = a.side >> 1, e1 = d == 0 ? 1 : 0, e2 = d == 2 ? 1 : 2;
    const int64_t n = (int64_t)a.P.n[e1] * a.P.n[e2] + (int64_t)(a.P.n[e1] + 1) * a.P.n[e2] +
                      (int64_t)a.P.n[e1] * (a.P.n[e2] + 1);
    k_res_reset<NS><<<grid_for(n, 128), 128, 0, s>>>(a);
    return cuda_rc(cudaGetLastError());
}

// part: 0 stresses, 1 face fluxes, 2 update, 3 the fused kernel (all three)
template <int NS, class R>
int launch_stage_part(const StageCall& c, int part) {
    if (part == 3) {
        switch (c.mode) {
            case NM_OFF: return launch_stage_zm_t<NS, R, NZ_OFF>(c);
            case NM_AB: return launch_stage_zm_t<NS, R, NZ_AB>(c);
            case NM_PHILOX: return launch_stage_zm_t<NS, R, NZ_PHILOX>(c);
            default: return FHD_ERR_BAD_ARG;
        }
    }
    if (!c.pack) {
        if constexpr (sizeof(R) == 8) {
            if (c.mode == NM_OFF) return launch_stage_plain_t<NS, NZ_OFF>(c, part);
            if (c.mode == NM_PHILOX) return launch_stage_plain_t<NS, NZ_PHILOX>(c, part);
        }
        return FHD_ERR_BAD_ARG;
    }
    switch (c.mode) {
        case NM_OFF: return launch_stage_part_t<NS, R, NZ_OFF>(c, part);
        case NM_AB: return launch_stage_part_t<NS, R, NZ_AB>(c, part);
        case NM_PHILOX: return launch_stage_part_t<NS, R, NZ_PHILOX>(c, part);
        default: return FHD_ERR_BAD_ARG;
    }
}

// ---- batched launches ------------------------------------------------------------
// kinds: 0 cellprep, 1 stresses, 2-4 face fluxes x/y/z, 5 update, 6 conversion.
// For the conversion kind the StageCall carries prim in pr, cu in cons_o, mom in mom_o.
template <int NS>
ConvArgs<NS> make_conv_args(const StageCall& c) {
    ConvArgs<NS> a;
    a.P = c.P;
    a.prim = view<double>(c.pr);
    a.cons = view<double>(c.cons_o);
    for (int d = 0; d < 3; ++d) {
        a.vel[d] = view<double>(c.vel[d]);
        a.mom[d] = view<const double>(c.mom_o[d]);
    }
    a.it = make_items(c.P.n[0], c.P.n[1], c.P.n[2]);
    a.status = c.status;
    a.img = c.img;
    return a;
}

template <int NS, class R, int NZ>
size_t batch_args_size_t(int kind) {
    if (kind == 0) return sizeof(PrepArgs<NS, R>);
    if (kind == 6) return sizeof(ConvArgs<NS>);
    return sizeof(StageArgs<NS, R, NZ, true>);
}

template <int NS, class R, int NZ>
void batch_pack_t(int kind, const StageCall& c, void* dst) {
    if (kind == 0) {
        const PrepArgs<NS, R> a = make_prep_args<NS, R>(c);
        memcpy(dst, &a, sizeof(a));
    } else if (kind == 6) {
        const ConvArgs<NS> a = make_conv_args<NS>(c);
        memcpy(dst, &a, sizeof(a));
    } else {
        const StageArgs<NS, R, NZ, true> a = make_stage_args<NS, R, NZ, true>(c);
        memcpy(dst, &a, sizeof(a));
    }
}

// register caps of the batched face kernel (resident blocks of 128 per SM), the
// batch autotuner's choices; the default is the first for up to two species and
// the last above
constexpr int kBatchFaceMinBlocks[] = {8, 6, 4};
constexpr int kNumBatchFaceTiles = 3;

template <int NS, class R, int NZ, int MINB>
void batch_faces_t(int kind, const StageArgs<NS, R, NZ, true>* sa, const int* dbpref, int nmem, int nblocks, cudaStream_t s) {
    k_faces_b<NS, R, NZ, MINB><<<nblocks, 128, 0, s>>>(sa, dbpref, nmem, kind - 2);
}

template <int NS, class R, int NZ>
int batch_launch_t(int kind, int tile, const void* dargs, const int* dbpref, int nmem, int nblocks, cudaStream_t s) {
    if (nblocks <= 0 || nmem <= 0) return FHD_OK;
    using SA = StageArgs<NS, R, NZ, true>;
    const SA* sa = static_cast<const SA*>(dargs);
    switch (kind) {
        case 0: k_cellprep_b<NS, R><<<nblocks, 128, 0, s>>>(static_cast<const PrepArgs<NS, R>*>(dargs), dbpref, nmem); break;
        case 1: k_taus_b<NS, R, NZ><<<nblocks, 128, 0, s>>>(sa, dbpref, nmem); break;
        case 2:
        case 3:
        case 4:
            if (tile < 0 || tile >= kNumBatchFaceTiles) tile = NS <= 2 ? 0 : kNumBatchFaceTiles - 1;
            if (tile == 0) batch_faces_t<NS, R, NZ, kBatchFaceMinBlocks[0]>(kind, sa, dbpref, nmem, nblocks, s);
            else if (tile == 1) batch_faces_t<NS, R, NZ, kBatchFaceMinBlocks[1]>(kind, sa, dbpref, nmem, nblocks, s);
            else batch_faces_t<NS, R, NZ, kBatchFaceMinBlocks[2]>(kind, sa, dbpref, nmem, nblocks, s);
            break;
        case 5: k_update_b<NS, R, NZ><<<nblocks, 128, 0, s>>>(sa, dbpref, nmem); break;
        case 6: k_convert_b<NS><<<nblocks, 128, 0, s>>>(static_cast<const ConvArgs<NS>*>(dargs), dbpref, nmem); break;
        default: return FHD_ERR_BAD_ARG;
    }
    return cuda_rc(cudaGetLastError());
}

// the persistent batched step: grid = the blocks that fit on the GPU at once
template <int NS, class R, int NZ, int MINB>
int batch_persist_minb(const PersistArgs& a, cudaStream_t s) {
    const int grid = resident_blocks<k_batch_persist<NS, R, NZ, MINB>>(128);
    k_batch_persist<NS, R, NZ, MINB><<<grid, 128, 0, s>>>(a);
    return cuda_rc(cudaGetLastError());
}

// tile: the register cap of the batch face tiles (kBatchFaceMinBlocks: 64, 80 or
// 128 registers); -1 the default, 64 registers up to two species (measured on the
// 512-member ensemble: 156 / 170 / 223 ms per step FP64, 112 / 124 / 141 mixed)
// and 128 above
template <int NS, class R, int NZ>
int batch_persist_t(const PersistArgs& a, int tile, cudaStream_t s) {
    if (tile < 0 || tile >= kNumBatchFaceTiles) tile = NS <= 2 ? 0 : 2;
    if (tile == 0) return batch_persist_minb<NS, R, NZ, kBatchFaceMinBlocks[0]>(a, s);
    if (tile == 1) return batch_persist_minb<NS, R, NZ, kBatchFaceMinBlocks[1]>(a, s);
    return batch_persist_minb<NS, R, NZ, kBatchFaceMinBlocks[2]>(a, s);
}

#define FHD_NS_SWITCH(ns, CALL) \
    switch (ns) {                \
        case 1: return CALL(1);  \
        case 2: return CALL(2);  \
        case 3: return CALL(3);  \
        case 4: return CALL(4);  \
        default: return FHD_ERR_UNSUPPORTED; \
    }

}  // namespace fhd
