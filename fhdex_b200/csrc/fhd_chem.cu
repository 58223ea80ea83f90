// fhd_chem.cu — the chemistry source kernel (compute_compressible_chemistry_source_CLE,
// chemistry_functions.cpp:128-193) and its launcher.  Built with -fmad=false: every
// product and sum is rounded on its own, as the host C++ evaluates it.
//
// One thread per valid cell, grid-stride.  Per cell it reads p, T and the NS mole
// fractions, draws (or reads) the nreaction noises and writes the NS species
// components of the source: (2 + NS) + NS doubles of HBM traffic, plus 2 x
// nreaction noise doubles when the A/B fields are injected.
#include "fhd_chem.cuh"
#include "fhd_launch.cuh"

namespace fhd {

struct ChemArgs {
    RunParams P;
    ChemParams C;
    Arr4<const double> pr;   // prim: T comp 4, p comp 5, X comps 6+NS..
    Items it;                // valid cells
    Arr4<double> src;        // species n -> comp 5+n
    Arr4<const double> na, nb;
    int mode;
    double w;                // stage weight of the B field
};

template <int NS>
static __global__ void __launch_bounds__(128) k_chem(ChemArgs a) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < a.it.n; q += gridDim.x * blockDim.x) {
        int i, j, k;
        a.it.point(q, i, j, k);
        double W[MAXR];
#pragma unroll
        for (int m = 0; m < MAXR; ++m) W[m] = 0.0;
        if (a.mode == CN_AB) {
            for (int m = 0; m < a.C.nr; ++m) W[m] = 1.0 * a.na(i, j, k, m) + a.w * a.nb(i, j, k, m);
        } else if (a.mode == CN_W) {
            for (int m = 0; m < a.C.nr; ++m) W[m] = a.na(i, j, k, m);
        } else if (a.mode == CN_PHILOX) {
            // the values fhd_fill_step_noise writes: A = 0.0 + 1.0 * z_A, B = 0.0 + 1.0 * z_B
            const uint32_t pidx = canon(a.P, i, j, k);
            const uint64_t step = noise_step(a.P);
            for (int m = 0; m < a.C.nr; m += 2) {
                float z[4];
                normal_quad(a.P.key0, a.P.key1, pidx, fid_chem(m) >> 1, step, z);
                W[m] = 1.0 * (0.0 + 1.0 * (double)z[0]) + a.w * (0.0 + 1.0 * (double)z[1]);
                if (m + 1 < a.C.nr) W[m + 1] = 1.0 * (0.0 + 1.0 * (double)z[2]) + a.w * (0.0 + 1.0 * (double)z[3]);
            }
        }
        double X[NS], S[NS];
#pragma unroll
        for (int n = 0; n < NS; ++n) X[n] = a.pr(i, j, k, 6 + NS + n);
        chem_point<NS>(a.P, a.C, a.pr(i, j, k, 5), a.pr(i, j, k, 4), X, W, S);
#pragma unroll
        for (int n = 0; n < NS; ++n) a.src(i, j, k, 5 + n) = S[n];
    }
}

template <int NS>
static int chem_launch_t(const ChemArgs& a, cudaStream_t s) {
    k_chem<NS><<<grid_for(a.it.n, 128), 128, 0, s>>>(a);
    return cuda_rc(cudaGetLastError());
}

int chem_launch(const DevParams& P, const ChemParams& C, const fhd_fab& prim, const fhd_fab& source,
                const fhd_fab* na, const fhd_fab* nb, int mode, double w, cudaStream_t s) {
    ChemArgs a;
    std::memset(&a, 0, sizeof(a));
    a.P = P;
    a.C = C;
    a.pr = view<const double>(prim);
    a.src = view<double>(source);
    if (na) a.na = view<const double>(*na);
    if (nb) a.nb = view<const double>(*nb);
    a.mode = mode;
    a.it = make_items(P.n[0], P.n[1], P.n[2]);
    a.w = w;
    switch (P.ns) {
        case 1: return chem_launch_t<1>(a, s);
        case 2: return chem_launch_t<2>(a, s);
        case 3: return chem_launch_t<3>(a, s);
        case 4: return chem_launch_t<4>(a, s);
        default: return FHD_ERR_UNSUPPORTED;
    }
}

}  // namespace fhd
