// fhd_sf.cu — static structure factor of cell-centred fields: the reference's
// StructFact (src_analysis/StructFact.cpp) for one periodic box.
//
// FortStructure (StructFact.cpp:231-311): for every variable that appears in a
// pair, a real-to-complex FFT over the box (cuFFT, D2Z; the reference uses
// amrex::FFT::R2C), the Hermitian half spectrum unpacked to the full grid and
// divided by sqrt(N) (ComputeFFT, :322-519), then for each pair (a, b)
//   cov_real += Re_a Re_b + Im_a Im_b,   cov_imag += -(Im_a Re_b) + Re_a Im_b.
// Here the unpacking is not materialised: the covariances are accumulated on the
// half spectrum (see SfArgs) in one kernel per sample and unfolded by the output
// kernels.
// CallFinalize / Finalize (:598-641) and ShiftFFT (:643-719): optional zeroing of
// k = 0, shift by N/2 in every direction, scaling by 1/nsamples and by
// 1/var_scaling, magnitude sqrt(re^2 + im^2).
//
// Stacks (the quasi-2-D runs' per-slice and the quasi-1-D runs' per-pencil
// StructFact vectors, main_driver.cpp:923-993): the members are independent
// structure factors of one shape; the dense copy of a variable holds them one
// after another, one batched cuFFT transforms them all, and the accumulators
// hold them one after another.  fhd_sf_stack_average fuses the reference's
// output loop (AddToExternal of every member, then the mult by 1/members).
//
// FP64 throughout; the accumulation and finalize arithmetic follow the
// reference's operation order (built with -fmad=false).  FFT values differ
// from another FFT library's at rounding level.
#include <cufft.h>

#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "fhd_launch.cuh"

using namespace fhd;

struct fhd_sf {
    int device = 0;
    int n[3] = {0, 0, 0};            // the box the variables fab covers
    int kind = FHD_SF_BOX;
    int m[3] = {0, 0, 0};            // one member's shape (the box itself unless a stack)
    int nmem = 1;                    // members
    int nvar = 0, ncov = 0;
    std::vector<int> pa, pb, varu;   // pairs (A, B) and the unique variables among them
    std::vector<double> scaling;     // 1 / var_scaling (StructFact.cpp:93-96)
    int64_t nsamples = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    double* cov = nullptr;           // [2][ncov][nmem][mz][my][mx/2+1]: real then imaginary accumulators
    double2* spec = nullptr;         // [nvaru][nmem][mz][my][mx/2+1] half spectra
    double* real = nullptr;          // [per_max][nmem][mz][my][mx] dense copy of the variables (FFT input)
    int* dpairs = nullptr;           // [2][ncov] pair -> unique-variable slot, then the variables' components
    double* dscale = nullptr;        // [ncov]
    cufftHandle plan = 0;
    // variables per execution of the plan: all of them, or one where their dense copy would
    // take more than the half grid saves (more variables than pairs) or that plan failed
    int per_max = 0, per_plan = 0;
    bool have_plan = false;
};

namespace {

// The covariances of real fields are Hermitian: at a mirrored point (i > nx/2, where the
// reference's unpacking takes the conjugate of entry (nx-i, -j, -k)) both spectra have
// negated imaginary parts, so the real covariance is the stored entry's and the
// imaginary one its negation, to the bit where it is not zero (a difference of equal
// products is +0.0 on both sides: the output subtracts from 0.0).  The accumulators are
// therefore kept on the half spectrum and unfolded at the output: half the traffic of a
// sample.
struct SfArgs {
    int nv, ncov;
    int64_t half;                    // half-spectrum entries of all members
    double sqrtnpts, rsqrtnpts;      // sqrt(N) of a member, and its reciprocal
    const double2* spec;
    const int* pairs;                // pa slots then pb slots
    double* cov;
    int reset;
};

// (re, im) of unique variable v at half-spectrum entry h, divided by sqrt(N)
// (ComputeFFT, StructFact.cpp:394-421); sqrt(N) is a run constant (fhd_div.h)
__device__ __forceinline__ double2 spec_at(const SfArgs& a, int v, int64_t h) {
    double2 s = a.spec[(int64_t)v * a.half + h];
    s.x = div_rcp(s.x, a.sqrtnpts, a.rsqrtnpts);
    s.y = div_rcp(s.y, a.sqrtnpts, a.rsqrtnpts);
    return s;
}

// A component of an output or input fab.  One component has fewer than 2^31 points
// (shape_fab_ok), all of them together may have more: 21 pairs at 512^3 are 2.8e9 values.
template <class T>
__device__ __forceinline__ T* sf_comp(const Arr4<T>& a, int n) { return a.p + (int64_t)n * a.sn; }

constexpr int kSfThreads = 256;
constexpr int kSfStaged = 12;        // variables whose values fit 48 KiB of shared memory per block

// One thread per half-spectrum entry.  STAGED (up to kSfStaged variables): the thread
// scales each variable's value once and keeps it in its own column of shared memory (a
// pair's two slots are known only at run time, which registers cannot be indexed by);
// else every pair reads and scales its two.  The accumulators of four pairs are
// loaded together before the first is stored.  Bound by HBM.  With a full-grid
// accumulator and four divisions per pair it took 153 us per sample at 144x112x96 (4
// variables, 10 pairs), more than half of the sample; two samples and the output of
// such a box went from 888 to 388 us with this, the batched transform and the output below.
template <bool STAGED>
__global__ void __launch_bounds__(kSfThreads) k_sf_accumulate(SfArgs a) {
    extern __shared__ double2 sv[];
    for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < a.half; h += (int64_t)gridDim.x * blockDim.x) {
        if (STAGED)
            for (int v = 0; v < a.nv; ++v) sv[v * kSfThreads + threadIdx.x] = spec_at(a, v, h);
        auto value = [&](int v) { return STAGED ? sv[v * kSfThreads + threadIdx.x] : spec_at(a, v, h); };
        constexpr int U = 4;
        for (int c0 = 0; c0 < a.ncov; c0 += U) {
            double re[U], im[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (c0 + u >= a.ncov || a.reset) continue;
                re[u] = a.cov[(int64_t)(c0 + u) * a.half + h];
                im[u] = a.cov[((int64_t)a.ncov + c0 + u) * a.half + h];
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int c = c0 + u;
                if (c >= a.ncov) continue;
                const double2 A = value(a.pairs[c]), B = value(a.pairs[a.ncov + c]);
                // cov_temp = 0 + Re_a Re_b; += Im_a Im_b   (StructFact.cpp:265-268)
                double tr = 0.0 + A.x * B.x;
                tr = tr + A.y * B.y;
                // cov_temp = 0 + Im_a Re_b; *= -1; += Re_a Im_b   (:276-280)
                double ti = 0.0 + A.y * B.x;
                ti = ti * -1.0;
                ti = ti + A.x * B.y;
                re[u] = a.reset ? tr : re[u] + tr;
                im[u] = a.reset ? ti : im[u] + ti;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (c0 + u >= a.ncov) continue;
                a.cov[(int64_t)(c0 + u) * a.half + h] = re[u];
                a.cov[((int64_t)a.ncov + c0 + u) * a.half + h] = im[u];
            }
        }
    }
}

// half-spectrum entry and sign of the imaginary part of full-grid point (i, j, k) of one member
__device__ __forceinline__ int64_t half_entry(int nx, int ny, int nz, int i, int j, int k, double& sign) {
    sign = 1.0;
    if (i > nx / 2) {
        sign = -1.0;
        i = nx - i;
        j = j == 0 ? 0 : ny - j;
        k = k == 0 ? 0 : nz - k;
    }
    return i + (int64_t)(nx / 2 + 1) * (j + (int64_t)ny * k);
}

struct SfFinArgs {
    int nx, ny, nz, nxh1, ncov, zero_avg;
    int64_t half;
    FastDiv dx, dxy;                 // by nxh1, nxh1 * ny
    double nsinv;
    const double* cov;
    const double* scale;
    Arr4<double> ore, oim, omag;
};

// Finalize (StructFact.cpp:598-620) with ShiftFFT (:643-719): destination point
// ((i + nx/2) % nx, ...) of source point (i, j, k).  One thread per half-spectrum entry
// writes its point and, where that is beyond nx/2, the mirrored one (equal but for the
// sign of the imaginary part), so that each entry is read, scaled and rooted once.
// Bound by its writes (30 components of 10 pairs).
__global__ void __launch_bounds__(256) k_sf_finalize(SfFinArgs a) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < a.half; q += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)a.dxy.div((uint32_t)q), r = (int)q - k * a.nxh1 * a.ny;
        const int j = (int)a.dx.div((uint32_t)r), i = r - j * a.nxh1;
        auto shift = [](int x, int n) { const int s = x + n / 2; return s >= n ? s - n : s; };
        const int ip = shift(i, a.nx), jp = shift(j, a.ny), kp = shift(k, a.nz);
        const bool mirror = a.nx - i > a.nx / 2 && i > 0;
        const int im = shift(a.nx - i, a.nx), jm = shift(j == 0 ? 0 : a.ny - j, a.ny),
                  km = shift(k == 0 ? 0 : a.nz - k, a.nz);
        const bool zero = a.zero_avg == 1 && q == 0;
        // (the three outputs have the box's cells and ghosts of their own)
        auto at = [](const Arr4<double>& v, int x, int y, int z) { return x + y * v.sy + z * v.sz; };
        const int ro = at(a.ore, ip, jp, kp), io = at(a.oim, ip, jp, kp), mo = at(a.omag, ip, jp, kp);
        const int rm = at(a.ore, im, jm, km), imm = at(a.oim, im, jm, km), mm = at(a.omag, im, jm, km);
#pragma unroll 2
        for (int c = 0; c < a.ncov; ++c) {
            double re = zero ? 0.0 : __ldg(a.cov + (int64_t)c * a.half + q);
            double im_ = zero ? 0.0 : __ldg(a.cov + ((int64_t)a.ncov + c) * a.half + q);
            re = re * a.nsinv;
            re = re * a.scale[c];
            im_ = im_ * a.nsinv;
            im_ = im_ * a.scale[c];
            double mag = 0.0 + re * re;
            mag = sqrt(mag + im_ * im_);
            double *const ore = sf_comp(a.ore, c), *const oim = sf_comp(a.oim, c), *const omag = sf_comp(a.omag, c);
            ore[ro] = re;
            oim[io] = im_;
            omag[mo] = mag;
            if (mirror) {
                ore[rm] = re;
                oim[imm] = 0.0 - im_;
                omag[mm] = mag;
            }
        }
    }
}

struct SfAvgArgs {
    int nx, ny, nz, ncov, zero_avg;
    int64_t Nm, nmem, half, halfm;
    double nsinv, meminv;
    const double* cov;
    const double* scale;
    Arr4<double> omag, ori;
};

// The reference's stack output loop (main_driver.cpp:1592-1618, 1683-1711): for
// every member in order, AddToExternal (StructFact.cpp:979-1009: Finalize of a
// copy, then x_mag += mag, x_realimag += (re, im), from zero), then both outputs
// times 1/members.  One thread per (pair, member point): it owns that pair's
// shifted destination and walks the members in order (a pencil stack has only
// n_cells[0] points, so the pairs multiply the independent chains).
__global__ void __launch_bounds__(256) k_sf_stack_avg(SfAvgArgs a) {
    const int64_t tot = a.Nm * a.ncov;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < tot; t += (int64_t)gridDim.x * blockDim.x) {
        const int c = int(t / a.Nm);
        const int64_t l = t - (int64_t)c * a.Nm;
        const int i = int(l % a.nx), j = int((l / a.nx) % a.ny), k = int(l / ((int64_t)a.nx * a.ny));
        const int ip = (i + a.nx / 2) % a.nx, jp = (j + a.ny / 2) % a.ny, kp = (k + a.nz / 2) % a.nz;
        const bool zero = a.zero_avg == 1 && i == 0 && j == 0 && k == 0;
        {
            double sm = 0.0, sr = 0.0, si = 0.0, sign;
            const int64_t h = half_entry(a.nx, a.ny, a.nz, i, j, k, sign);
            const double* cr = a.cov + (int64_t)c * a.half + h;
            const double* ci = a.cov + ((int64_t)a.ncov + c) * a.half + h;
            // the members' loads are independent of the sums: eight in flight per chain
#pragma unroll 8
            for (int64_t b = 0; b < a.nmem; ++b) {
                double re = zero ? 0.0 : __ldg(cr + b * a.halfm);
                double im = zero ? 0.0 : sign * __ldg(ci + b * a.halfm);
                re = re * a.nsinv;
                re = re * a.scale[c];
                im = im * a.nsinv;
                im = im * a.scale[c];
                double mag = 0.0 + re * re;
                mag = mag + im * im;
                sm = sm + sqrt(mag);
                sr = sr + re;
                si = si + im;
            }
            sf_comp(a.omag, c)[ip + jp * a.omag.sy + kp * a.omag.sz] = sm * a.meminv;
            sf_comp(a.ori, c)[ip + jp * a.ori.sy + kp * a.ori.sz] = sr * a.meminv;
            sf_comp(a.ori, a.ncov + c)[ip + jp * a.ori.sy + kp * a.ori.sz] = si * a.meminv;
        }
    }
}

}  // namespace

namespace {

int shape_fab_ok(const int n[3], const fhd_fab& f, int min_nc) {
    if (!f.data || f.dtype != FHD_F64 || f.ncomp < min_nc) return 0;
    const int g = -f.lo[0];
    if (g < 0) return 0;
    int64_t points = 1;
    for (int d = 0; d < 3; ++d) {
        if (f.nodal[d] != 0 || f.lo[d] != -g || f.hi[d] != n[d] - 1 + g) return 0;
        points *= n[d] + 2 * (int64_t)g;
        if (points > INT32_MAX) return 0;   // the kernels index a component with 32 bits
    }
    return 1;
}
int sf_fab_ok(const fhd_sf* s, const fhd_fab& f, int min_nc) { return shape_fab_ok(s->n, f, min_nc); }

int cufft_rc(cufftResult r) { return r == CUFFT_SUCCESS ? FHD_OK : FHD_ERR_CUDA; }

// D2Z plan of every variable and member at once (slowest dimension first: cuFFT is
// row-major): 3-D over the box, 2-D over a slice, 1-D over a pencil, transforms
// contiguous in the input and in the half spectra.  One execution per sample: 144x112x96
// with 4 variables took 12 kernels of about 10 us each with a plan per variable, 3 here.
int sf_plan(fhd_sf* s) {
    if (s->have_plan) return FHD_OK;
    int rc;
    const int rank = s->kind == FHD_SF_BOX ? 3 : (s->kind == FHD_SF_Z_SLICES ? 2 : 1);
    int dims[3], oemb[3];
    for (int r = 0; r < rank; ++r) dims[r] = oemb[r] = s->m[rank - 1 - r];
    oemb[rank - 1] = s->m[0] / 2 + 1;
    s->per_plan = (int64_t)s->nmem * s->per_max > INT32_MAX ? 1 : s->per_max;
    for (;;) {
        rc = cufft_rc(cufftPlanMany(&s->plan, rank, dims, dims, 1, s->m[0] * s->m[1] * s->m[2], oemb, 1,
                                    (s->m[0] / 2 + 1) * s->m[1] * s->m[2], CUFFT_D2Z, s->nmem * s->per_plan));
        if (!rc || s->per_plan == 1) break;
        cudaGetLastError();
        s->per_plan = 1;   // no room for the workspace of all variables: one at a time
    }
    if (rc) return rc;
    rc = cufft_rc(cufftSetStream(s->plan, s->stream));
    if (rc) {
        cufftDestroy(s->plan);
        return rc;
    }
    s->have_plan = true;
    return FHD_OK;
}

// dense copy of the variables (blockIdx.y); x pencils in the reference's member order
// (member p at y = p / ny, z = p % ny, ExtractXPencil's arguments in
// main_driver.cpp:1551), everything else in the box's own order
struct PackArgs {
    Arr4<const double> v;
    const int* comp;
    int nx, ny;
    int64_t N;
    FastDiv dx, dxy, dy;
    int pencils;
    double* out;
};
__global__ void __launch_bounds__(256) k_sf_pack(PackArgs a) {
    const double* const v = sf_comp(a.v, a.comp[blockIdx.y]);
    double* out = a.out + (int64_t)blockIdx.y * a.N;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < a.N; q += (int64_t)gridDim.x * blockDim.x) {
        if (a.pencils) {
            const int p = (int)a.dx.div((uint32_t)q), y = (int)a.dy.div((uint32_t)p);
            out[q] = v[(int)q - p * a.nx + y * a.v.sy + (p - y * a.ny) * a.v.sz];
        } else {
            const int k = (int)a.dxy.div((uint32_t)q), r = (int)q - k * a.nx * a.ny;
            const int j = (int)a.dx.div((uint32_t)r);
            out[q] = v[r - j * a.nx + j * a.v.sy + k * a.v.sz];
        }
    }
}

// Whether cuFFT can read the caller's fab itself: no ghosts, the used variables
// consecutive components (then the transforms follow each other as in the dense copy),
// members in the box's order, and a first element on the 16-byte boundary that cuFFT
// asks of its input.  The out-of-place transform leaves its input unchanged.
bool direct_input(const fhd_sf* s, const fhd_fab& f) {
    if (s->kind == FHD_SF_X_PENCILS || f.lo[0] != 0) return false;
    for (size_t u = 1; u < s->varu.size(); ++u)
        if (s->varu[u] != s->varu[0] + (int)u) return false;
    const int64_t N = (int64_t)s->n[0] * s->n[1] * s->n[2];
    return ((uintptr_t)(static_cast<const double*>(f.data) + N * s->varu[0]) & 15) == 0;
}

}  // namespace

extern "C" {

int fhd_sf_create(fhd_sf** out, const int n_cells[3], int nvar, int ncov, const int* pairA, const int* pairB,
                  const double* var_scaling, int device) {
    return fhd_sf_create_stack(out, n_cells, FHD_SF_BOX, nvar, ncov, pairA, pairB, var_scaling, device);
}

int fhd_sf_create_stack(fhd_sf** out, const int n_cells[3], int kind, int nvar, int ncov, const int* pairA,
                        const int* pairB, const double* var_scaling, int device) {
    if (!out || !n_cells || nvar < 1 || !var_scaling) return FHD_ERR_BAD_ARG;
    if (kind != FHD_SF_BOX && kind != FHD_SF_Z_SLICES && kind != FHD_SF_X_PENCILS) return FHD_ERR_BAD_ARG;
    for (int d = 0; d < 3; ++d)
        if (n_cells[d] < (kind == FHD_SF_BOX || d == 0 ? 2 : 1)) return FHD_ERR_BAD_ARG;
    if (kind == FHD_SF_Z_SLICES && n_cells[1] < 2) return FHD_ERR_BAD_ARG;
    int64_t cells = 1;
    for (int d = 0; d < 3; ++d) {
        cells *= n_cells[d];
        if (cells > INT32_MAX) return FHD_ERR_UNSUPPORTED;
    }
    if (kind == FHD_SF_X_PENCILS && n_cells[1] != n_cells[2]) return FHD_ERR_UNSUPPORTED;
    fhd_sf* s = new (std::nothrow) fhd_sf;
    if (!s) return FHD_ERR_OOM;
    s->device = device;
    s->kind = kind;
    for (int d = 0; d < 3; ++d) s->n[d] = s->m[d] = n_cells[d];
    if (kind == FHD_SF_Z_SLICES) {
        s->m[2] = 1;
        s->nmem = n_cells[2];
    } else if (kind == FHD_SF_X_PENCILS) {
        s->m[1] = s->m[2] = 1;
        s->nmem = n_cells[1] * n_cells[2];
    }
    s->nvar = nvar;
    if (!pairA || !pairB) {
        // all NVAR (NVAR + 1) / 2 pairs: A = j, B = i for i <= j (StructFact.cpp:45-69)
        for (int i = 0; i < nvar; ++i)
            for (int j = i; j < nvar; ++j) {
                s->pa.push_back(j);
                s->pb.push_back(i);
            }
    } else {
        for (int c = 0; c < ncov; ++c) {
            if (pairA[c] < 0 || pairA[c] >= nvar || pairB[c] < 0 || pairB[c] >= nvar) {
                delete s;
                return FHD_ERR_BAD_ARG;  // StructFact.cpp:186-190
            }
            s->pa.push_back(pairA[c]);
            s->pb.push_back(pairB[c]);
        }
    }
    s->ncov = (int)s->pa.size();
    if (s->ncov < 1) {
        delete s;
        return FHD_ERR_BAD_ARG;
    }
    for (int c = 0; c < s->ncov; ++c) s->scaling.push_back(1.0 / var_scaling[c]);
    // unique variables, ascending (StructFact.cpp:100-152)
    std::vector<int> used(nvar, 0);
    for (int c = 0; c < s->ncov; ++c) used[s->pa[c]] = used[s->pb[c]] = 1;
    std::vector<int> slot(nvar, -1);
    for (int v = 0; v < nvar; ++v)
        if (used[v]) {
            slot[v] = (int)s->varu.size();
            s->varu.push_back(v);
        }
    std::vector<int> hp(2 * s->ncov);
    for (int c = 0; c < s->ncov; ++c) {
        hp[c] = slot[s->pa[c]];
        hp[s->ncov + c] = slot[s->pb[c]];
    }
    hp.insert(hp.end(), s->varu.begin(), s->varu.end());
    // full-grid accumulators and one variable's copy took 2 ncov + 1 grids beside the
    // spectra, the half-grid ones and per_max copies take ncov + per_max
    s->per_max = (int)s->varu.size() <= s->ncov + 1 ? (int)s->varu.size() : 1;
    const int64_t N = (int64_t)s->n[0] * s->n[1] * s->n[2];
    const int64_t half = (int64_t)(s->m[0] / 2 + 1) * s->m[1] * s->m[2] * s->nmem;
    int rc = FHD_OK;
    if (cudaSetDevice(device) != cudaSuccess) rc = FHD_ERR_CUDA;
    if (!rc && cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) rc = FHD_ERR_CUDA;
    if (!rc) s->own_stream = true;
    if (!rc && (cudaMalloc(&s->cov, sizeof(double) * 2 * s->ncov * half) != cudaSuccess ||
                cudaMalloc(&s->spec, sizeof(double2) * s->varu.size() * half) != cudaSuccess ||
                cudaMalloc(&s->real, sizeof(double) * s->per_max * N) != cudaSuccess ||
                cudaMalloc(&s->dpairs, sizeof(int) * hp.size()) != cudaSuccess ||
                cudaMalloc(&s->dscale, sizeof(double) * s->ncov) != cudaSuccess))
        rc = FHD_ERR_OOM;
    if (!rc && (cudaMemcpy(s->dpairs, hp.data(), sizeof(int) * hp.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
                cudaMemcpy(s->dscale, s->scaling.data(), sizeof(double) * s->ncov, cudaMemcpyHostToDevice) != cudaSuccess ||
                cudaMemset(s->cov, 0, sizeof(double) * 2 * s->ncov * half) != cudaSuccess))
        rc = FHD_ERR_CUDA;
    if (rc) {
        cudaGetLastError();
        fhd_sf_destroy(s);
        return rc;
    }
    *out = s;
    return FHD_OK;
}

int fhd_sf_destroy(fhd_sf* s) {
    if (!s) return FHD_ERR_BAD_ARG;
    cudaSetDevice(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    if (s->have_plan) cufftDestroy(s->plan);
    cudaFree(s->cov);
    cudaFree(s->spec);
    cudaFree(s->real);
    cudaFree(s->dpairs);
    cudaFree(s->dscale);
    if (s->own_stream) cudaStreamDestroy(s->stream);
    delete s;
    return FHD_OK;
}

int fhd_sf_set_stream(fhd_sf* s, void* stream) {
    if (!s) return FHD_ERR_BAD_ARG;
    if (s->own_stream) {
        cudaStreamSynchronize(s->stream);
        cudaStreamDestroy(s->stream);
        s->own_stream = false;
    }
    s->stream = static_cast<cudaStream_t>(stream);
    if (s->have_plan) return cufft_rc(cufftSetStream(s->plan, s->stream));
    return FHD_OK;
}

int fhd_sf_ncov(const fhd_sf* s) { return s ? s->ncov : -1; }
int64_t fhd_sf_nsamples(const fhd_sf* s) { return s ? s->nsamples : -1; }

int fhd_sf_fort_structure(fhd_sf* s, fhd_fab variables, int reset) {
    if (!s || !sf_fab_ok(s, variables, s->nvar)) return FHD_ERR_BAD_ARG;
    cudaSetDevice(s->device);
    int rc = sf_plan(s);
    if (rc) return rc;
    const int64_t N = (int64_t)s->n[0] * s->n[1] * s->n[2];
    const int64_t half = (int64_t)(s->m[0] / 2 + 1) * s->m[1] * s->m[2] * s->nmem;
    const int nv = (int)s->varu.size();
    auto exec = [&](double* in, int u) {
        return cufft_rc(cufftExecD2Z(s->plan, in, reinterpret_cast<cufftDoubleComplex*>(s->spec + u * half)));
    };
    if (s->per_plan == nv && direct_input(s, variables)) {
        rc = exec(static_cast<double*>(variables.data) + N * s->varu[0], 0);
    } else {
        PackArgs p;
        p.v = view<const double>(variables);
        p.nx = s->n[0];
        p.ny = s->n[1];
        p.N = N;
        p.dx = fast_div((uint32_t)s->n[0]);
        p.dxy = fast_div((uint32_t)(s->n[0] * s->n[1]));
        p.dy = fast_div((uint32_t)s->n[1]);
        p.pencils = s->kind == FHD_SF_X_PENCILS ? 1 : 0;
        p.out = s->real;   // one variable at a time: each at the buffer's aligned start
        for (int u = 0; u < nv && !rc; u += s->per_plan) {
            p.comp = s->dpairs + 2 * s->ncov + u;
            k_sf_pack<<<dim3(grid_for(N, 256, 148 * 8), s->per_plan), 256, 0, s->stream>>>(p);
            rc = cuda_rc(cudaGetLastError());
            if (!rc) rc = exec(s->real, u);
        }
    }
    if (rc) return rc;
    SfArgs a;
    a.nv = nv;
    a.ncov = s->ncov;
    a.half = half;
    a.sqrtnpts = std::sqrt((double)((int64_t)s->m[0] * s->m[1] * s->m[2]));  // StructFact.cpp:348-350, one member's box
    a.rsqrtnpts = 1.0 / a.sqrtnpts;
    a.spec = s->spec;
    a.pairs = s->dpairs;
    a.cov = s->cov;
    a.reset = (reset == 1 || s->nsamples == 0) ? 1 : 0;
    const int grid = grid_for(half, kSfThreads);
    if (nv <= kSfStaged) k_sf_accumulate<true><<<grid, kSfThreads, sizeof(double2) * kSfThreads * nv, s->stream>>>(a);
    else k_sf_accumulate<false><<<grid, kSfThreads, 0, s->stream>>>(a);
    rc = cuda_rc(cudaGetLastError());
    if (rc) return rc;
    s->nsamples = (reset == 1) ? 1 : s->nsamples + 1;  // :307-311
    return FHD_OK;
}

int fhd_sf_finalize(fhd_sf* s, fhd_fab cov_real, fhd_fab cov_imag, fhd_fab cov_mag, int zero_avg) {
    if (!s || s->nsamples < 1 || s->kind != FHD_SF_BOX) return FHD_ERR_BAD_ARG;
    if (!sf_fab_ok(s, cov_real, s->ncov) || !sf_fab_ok(s, cov_imag, s->ncov) || !sf_fab_ok(s, cov_mag, s->ncov))
        return FHD_ERR_BAD_ARG;
    cudaSetDevice(s->device);
    SfFinArgs a;
    a.nx = s->n[0];
    a.ny = s->n[1];
    a.nz = s->n[2];
    a.ncov = s->ncov;
    a.zero_avg = zero_avg;
    a.nxh1 = s->n[0] / 2 + 1;
    a.half = (int64_t)a.nxh1 * s->n[1] * s->n[2];
    a.dx = fast_div((uint32_t)a.nxh1);
    a.dxy = fast_div((uint32_t)(a.nxh1 * s->n[1]));
    a.nsinv = 1.0 / (double)s->nsamples;  // StructFact.cpp:603
    a.cov = s->cov;
    a.scale = s->dscale;
    a.ore = view<double>(cov_real);
    a.oim = view<double>(cov_imag);
    a.omag = view<double>(cov_mag);
    k_sf_finalize<<<grid_for(a.half, 256), 256, 0, s->stream>>>(a);
    return cuda_rc(cudaGetLastError());
}

int fhd_sf_stack_average(fhd_sf* s, fhd_fab mag, fhd_fab realimag, int zero_avg) {
    if (!s || s->nsamples < 1 || s->kind == FHD_SF_BOX) return FHD_ERR_BAD_ARG;
    if (!shape_fab_ok(s->m, mag, s->ncov) || !shape_fab_ok(s->m, realimag, 2 * s->ncov)) return FHD_ERR_BAD_ARG;
    cudaSetDevice(s->device);
    SfAvgArgs a;
    a.nx = s->m[0];
    a.ny = s->m[1];
    a.nz = s->m[2];
    a.ncov = s->ncov;
    a.zero_avg = zero_avg;
    a.Nm = (int64_t)s->m[0] * s->m[1] * s->m[2];
    a.nmem = s->nmem;
    a.halfm = (int64_t)(s->m[0] / 2 + 1) * s->m[1] * s->m[2];
    a.half = a.halfm * a.nmem;
    a.nsinv = 1.0 / (double)s->nsamples;  // StructFact.cpp:603
    a.meminv = 1.0 / (double)s->nmem;     // ncellsinv (main_driver.cpp:1610, 1702)
    a.cov = s->cov;
    a.scale = s->dscale;
    a.omag = view<double>(mag);
    a.ori = view<double>(realimag);
    k_sf_stack_avg<<<grid_for(a.Nm * a.ncov, 256), 256, 0, s->stream>>>(a);
    return cuda_rc(cudaGetLastError());
}

int fhd_sf_synchronize(fhd_sf* s) {
    if (!s) return FHD_ERR_BAD_ARG;
    return cuda_rc(cudaStreamSynchronize(s->stream));
}

}  // extern "C"
