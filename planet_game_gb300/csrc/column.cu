// K12: per-cell grey column radiation for sm_103a.
//
// For every cell, N equal-mass sigma layers (N <= 16; the reference caps N at 8,
// sim/planet/atmosphere/atmosphere.hpp:85, the same formulas hold for any N):
//   emissivity   eps_k = -expm1(-(tau_d dp/p0 + kappa_v q_k dp/g))   (atmosphere_column.hpp:85-104)
//   cloud optics f_k, tau_k, R_k, kappa_l LWP_k, transmission, column fraction
//                                                                     (atmosphere_column.hpp:599-623)
//   cloud LW     eps_k' = -expm1(log1p(-eps_k) - kappa_l LWP_k)       (atmosphere_column.hpp:627-634)
//   two-stream   absorbed_k, downward surface LW, OLR                 (atmosphere_column.hpp:125-143)
// with layer emission eps_k sigma T_k^4 (atmosphere_column.hpp:918) and a black surface
// sigma Ts^4 below. FP64 throughout.
//
// What bounds it is the FP64 pipe (two results a cycle and SM), so the formulas are rearranged to
// spend less of it, each within a rounding or two of the reference's:
//   eps_k' = -expm1(-(tau_d dp/p0 + kappa_v q_k dp/g + kappa_l LWP_k)): the logarithm of 1 - eps_k
//     is the clear depth itself, so one expm1 takes the place of two and a log1p;
//   the layer's mass dp/g is divided out once a column, not once a layer;
//   a broken cloud (LWP_k < W_c, f_k < 1) has the in-cloud path W_c, so its tau_k and R_k / f_k are
//     constants of the launch, and an overcast layer alone divides;
//   the two-stream sums use fused multiply-adds.
// 40,962 columns of 10 layers, the whole call: 152 us before, 45 after; error against 64-bit
// formulas 1.5e-16 either way.
//
// Layout: layer-major [N][cells] arrays, one thread per cell, the column in registers.
#include "column.hpp"
#include "common.cuh"
#include "profile.hpp"

#include <stdexcept>

namespace psgb {
namespace {

// Constants of a launch, formed on the host.
struct ColumnTerms {
    double dry_per_pa;      // tau_d / p0
    double tau_per_path;    // 3 / (2 rho_w r_e)
    double asymmetry;       // 1 - g
    double per_cloud_path;  // 1 / W_c
    double broken_tau;      // tau of the in-cloud path W_c
    double broken_share;    // its R / f
};

constexpr int kColumnThreads = 32;

template <int L>
__global__ void __launch_bounds__(kColumnThreads) k_column(std::uint32_t cells, ColumnConstants k, ColumnTerms terms,
                                                           const double* __restrict__ temp, const double* __restrict__ hum,
                                                           const double* __restrict__ cloud, const double* __restrict__ ts,
                                                           const double* __restrict__ ps, double* __restrict__ emissivity,
                                                           double* __restrict__ absorbed, double* __restrict__ fraction,
                                                           double* __restrict__ reflectance, double* __restrict__ scalars) {
    const std::uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cells) return;
    const double p_s = ps[c];
    const double dry = terms.dry_per_pa * (p_s / static_cast<double>(L));
    const double mass = p_s / (k.gravity * static_cast<double>(L));
    double eps[L], emis[L];
    double clear = 1.0, transmission = 1.0, col_tau = 0.0;
#pragma unroll
    for (int l = 0; l < L; ++l) {
        const std::size_t i = static_cast<std::size_t>(l) * cells + c;
        const double q = hum[i];
        double depth = __fma_rn(k.vapour_absorption, (q > 0.0 ? q : 0.0) * mass, dry);
        const double ql = cloud[i];
        const double path = (ql > 0.0 ? ql : 0.0) * mass;
        double f = 0.0, r = 0.0;
        if (path > 0.0) {
            const double ratio = path * terms.per_cloud_path;
            double tau = terms.broken_tau;
            f = ratio;
            r = ratio * terms.broken_share;
            if (!(ratio < 1.0)) {
                f = 1.0;
                tau = path * terms.tau_per_path;
                r = terms.asymmetry * tau / __fma_rn(terms.asymmetry, tau, 2.0);
            }
            clear *= 1.0 - f;
            transmission *= 1.0 - r;
            col_tau = __fma_rn(f, tau, col_tau);
            const double lw = k.cloud_longwave_absorption * path;
            if (lw > 0.0) depth += lw;
        }
        const double e = -expm1(-depth);
        fraction[i] = f;
        reflectance[i] = r;
        eps[l] = e;
        emissivity[i] = e;
        const double t = temp[i];
        const double t2 = t * t;
        emis[l] = e * k.stefan_boltzmann * (t2 * t2);
    }
    double above[L];
    double down = 0.0;
#pragma unroll
    for (int l = L - 1; l >= 0; --l) {
        above[l] = down;
        down = __fma_rn(1.0 - eps[l], down, emis[l]);
    }
    const double tsc = ts[c];
    const double ts2 = tsc * tsc;
    double up = k.stefan_boltzmann * (ts2 * ts2);
#pragma unroll
    for (int l = 0; l < L; ++l) {
        absorbed[static_cast<std::size_t>(l) * cells + c] = eps[l] * (up + above[l]);
        up = __fma_rn(1.0 - eps[l], up, emis[l]);
    }
    scalars[c] = down;
    scalars[cells + c] = up;
    scalars[2 * static_cast<std::size_t>(cells) + c] = transmission;
    scalars[3 * static_cast<std::size_t>(cells) + c] = 1.0 - clear;
    scalars[4 * static_cast<std::size_t>(cells) + c] = col_tau;
}

}  // namespace

void launch_column_radiation(std::uint32_t cells, std::uint32_t layers, const ColumnConstants& k,
                             const double* temp, const double* hum, const double* cloud, const double* ts,
                             const double* ps, double* emissivity, double* absorbed, double* fraction,
                             double* reflectance, double* scalars, cudaStream_t st) {
    ColumnTerms terms{};
    terms.dry_per_pa = k.dry_optical_depth / k.reference_pressure;
    terms.tau_per_path = 3.0 / (2.0 * 1000.0 * k.effective_radius);
    terms.asymmetry = 1.0 - k.cloud_asymmetry;
    terms.per_cloud_path = 1.0 / k.in_cloud_water_path;
    terms.broken_tau = 3.0 * k.in_cloud_water_path / (2.0 * 1000.0 * k.effective_radius);
    terms.broken_share = terms.asymmetry * terms.broken_tau / (2.0 + terms.asymmetry * terms.broken_tau);
    // one-warp blocks: the FP64 pipe needs few warps, and finer blocks even out the SMs' shares
    // (40,962 columns are 2.1 blocks of 128 an SM, three on some)
    const dim3 grid((cells + kColumnThreads - 1) / kColumnThreads), block(kColumnThreads);
#define PSGB_COLUMN_CASE(N) \
    case N: PSGB_LAUNCH(kFamColumn, st, (k_column<N><<<grid, block, 0, st>>>(cells, k, terms, temp, hum, cloud, ts, ps, emissivity, absorbed, fraction, reflectance, scalars))); break;
    switch (layers) {
        PSGB_COLUMN_CASE(1) PSGB_COLUMN_CASE(2) PSGB_COLUMN_CASE(3) PSGB_COLUMN_CASE(4)
        PSGB_COLUMN_CASE(5) PSGB_COLUMN_CASE(6) PSGB_COLUMN_CASE(7) PSGB_COLUMN_CASE(8)
        PSGB_COLUMN_CASE(9) PSGB_COLUMN_CASE(10) PSGB_COLUMN_CASE(11) PSGB_COLUMN_CASE(12)
        PSGB_COLUMN_CASE(13) PSGB_COLUMN_CASE(14) PSGB_COLUMN_CASE(15) PSGB_COLUMN_CASE(16)
        default: throw std::invalid_argument("column radiation supports 1 to 16 layers");
    }
#undef PSGB_COLUMN_CASE
}

}  // namespace psgb
