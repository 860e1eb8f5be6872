// Finite-volume operators and the implicit heat step's flux form, for sm_103a.
//
// K1 laplacian / diffusion_source  (sim/planet/operators/finite_volume.cpp:91-111,
//                                   sim/planet/surface/heat_transport.cpp:28-36,579-593)
// K2 gradient                       (finite_volume.cpp:55-89)
// K3 divergence                     (finite_volume.cpp:34-53)
// K13 transport step flux form      (heat_transport.cpp:734-770)
//
// One thread per cell over ELL slot-major neighbour arrays (coalesced per slot); the
// neighbour values are gathered through L2, where the reference's space-filling cell
// order keeps them close. Accumulation is FP64 in the reference's order without
// fused multiply-adds, so diffusion_source and gradient are bit-identical to the
// reference and the Laplacian differs only by using the precomputed l/d weight.
//
// What bounds K1-K3 is the FP64 unit (a warp instruction every 19 cycles an SM, conversions
// included), not memory: so the divisions by mesh lengths, areas and determinants take stored
// reciprocals (for 64-bit fields divide_by, the same bits in half the instructions); 32-bit fields,
// whose results are rounded to 32 bits, fuse their products and sums and divide in three operations;
// what is 32 bits wide is widened from its bits; and a block is two warps, so that the SMs' shares
// differ little (at 40,962 cells blocks of eight gave some SMs 16 warps and most 8).
// Cold, before and after, in us:      gradient     divergence   Laplacian
//   40,962 cells, 64 bits            19.2 -> 12.8   7.6 -> 6.0   7.0 -> 5.3
//   655,362 cells, 32 bits            149 -> 85      45 -> 33      46 -> 32
#include "common.cuh"
#include "profile.hpp"
#include "operators.hpp"
#include "phases.cuh"

namespace psgb {
namespace {

constexpr unsigned kOperatorThreads = 64;

// The arithmetic of a field's type: 64 bits in the reference's roundings, 32 bits with fused
// products and a quotient from one correction, both in 64 bits and no further from the exact value.
template <typename T>
__device__ __forceinline__ double add_product(double sum, double a, double b) {
    if constexpr (sizeof(T) == 8) return dadd(sum, dmul(a, b));
    else return __fma_rn(a, b, sum);
}
template <typename T>
__device__ __forceinline__ double product_difference(double a, double b, double c, double d) {   // a b - c d
    if constexpr (sizeof(T) == 8) return dsub(dmul(a, b), dmul(c, d));
    else return __fma_rn(a, b, -dmul(c, d));
}
template <typename T>
__device__ __forceinline__ double quotient(double s, double d, double r) {
    if constexpr (sizeof(T) == 8) return divide_by(s, d, r);
    // zeros, infinities and NaN are divided; of the others nothing leaves the range of 64 bits
    const std::uint32_t high = static_cast<std::uint32_t>(__double2hiint(s)) & 0x7fffffffu;
    if (__double2hiint(r) == 0 || high - 1u >= 0x7ff00000u - 1u) return __ddiv_rn(s, d);
    const double q = dmul(s, r);
    return __fma_rn(__fma_rn(-d, q, s), r, q);
}

__global__ void k_reciprocal(std::size_t n, const double* __restrict__ d, double* __restrict__ r) {
    const std::size_t i = std::size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) r[i] = reciprocal_of(d[i]);
}

template <typename T>
__global__ void __launch_bounds__(kOperatorThreads) k_laplacian(std::uint32_t n, std::uint32_t P, const std::int32_t* __restrict__ nbr,
                            const double* __restrict__ w, const double* __restrict__ area,
                            const double* __restrict__ rarea, const T* __restrict__ in, T* __restrict__ out) {
    const std::uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double own = widen(in[c]);
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const double wj = w[j * P + c];
        const double v = widen(in[nbr[j * P + c]]);
        sum = add_product<T>(sum, dsub(v, own), wj);
    }
    out[c] = static_cast<T>(quotient<T>(sum, area[c], rarea[c]));
}

// H = K * (sum_k w_k (T_k - T_c)) / A, the reference's diffusion_source.
__global__ void k_diffusion_source(std::uint32_t n, std::uint32_t P, const std::int32_t* __restrict__ nbr,
                                   const double* __restrict__ w, const double* __restrict__ area,
                                   double conductance, const double* __restrict__ t,
                                   double* __restrict__ out) {
    const std::uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double own = t[c];
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) sum = dadd(sum, dmul(dsub(t[nbr[j * P + c]], own), w[j * P + c]));
    out[c] = __ddiv_rn(dmul(conductance, sum), area[c]);
}

// A node's area-weighted mean of its fine cells' values, summed over the members in cell
// order and divided by the node's area (surface_energy.cpp:1285-1296); two fields at once
// (mean and slope of a response), the second optional.
__global__ void k_group_mean(std::uint32_t n, const std::uint32_t* __restrict__ member_offset,
                             const std::uint32_t* __restrict__ member, const double* __restrict__ fine_area,
                             const double* __restrict__ graph_area, const double* __restrict__ a,
                             const double* __restrict__ b, double* __restrict__ mean_a, double* __restrict__ mean_b) {
    const std::uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    double sa = 0.0, sb = 0.0;
    for (std::uint32_t k = member_offset[g]; k < member_offset[g + 1]; ++k) {
        const std::uint32_t c = member[k];
        const double area = fine_area[c];
        sa = dadd(sa, dmul(area, a[c]));
        if (b != nullptr) sb = dadd(sb, dmul(area, b[c]));
    }
    mean_a[g] = __ddiv_rn(sa, graph_area[g]);
    if (b != nullptr) mean_b[g] = __ddiv_rn(sb, graph_area[g]);
}

// Every fine cell takes its node's value (surface_energy.cpp:1583, 1595).
__global__ void k_group_scatter(std::uint32_t fine_cells, const std::uint32_t* __restrict__ group_of_cell,
                                const double* __restrict__ node_value, double* __restrict__ out) {
    const std::uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < fine_cells) out[c] = node_value[group_of_cell[c]];
}

template <typename T>
__global__ void __launch_bounds__(kOperatorThreads) k_gradient(std::uint32_t n, std::uint32_t P, const std::int32_t* __restrict__ nbr,
                           const std::uint8_t* __restrict__ degree, const double* __restrict__ dist,
                           const double* __restrict__ rdist, const float* __restrict__ ne,
                           const float* __restrict__ nn, const double* __restrict__ gm,
                           const double* __restrict__ rdet, const T* __restrict__ in,
                           T* __restrict__ east, T* __restrict__ north) {
    const std::uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double own = widen(in[c]);
    const int deg = degree[c];
    double re = 0.0, rn = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        if (j < deg) {
            const double a = widen(ne[j * P + c]);
            const double b = widen(nn[j * P + c]);
            const double slope = quotient<T>(dsub(widen(in[nbr[j * P + c]]), own), dist[j * P + c], rdist[j * P + c]);
            re = add_product<T>(re, slope, a);
            rn = add_product<T>(rn, slope, b);
        }
    }
    const double mee = gm[c], men = gm[P + c], mnn = gm[2 * P + c], det = gm[3 * P + c], r = rdet[c];
    east[c] = static_cast<T>(quotient<T>(product_difference<T>(mnn, re, men, rn), det, r));
    north[c] = static_cast<T>(quotient<T>(product_difference<T>(mee, rn, men, re), det, r));
}

template <typename T>
__global__ void __launch_bounds__(kOperatorThreads) k_divergence(std::uint32_t n, std::uint32_t P, const std::int32_t* __restrict__ edge,
                             const std::uint8_t* __restrict__ first, const std::uint8_t* __restrict__ degree,
                             const double* __restrict__ length, const double* __restrict__ area,
                             const double* __restrict__ rarea, const T* __restrict__ flux, T* __restrict__ out) {
    const std::uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const int deg = degree[c];
    const unsigned mask = first[c];
    double net = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        if (j < deg) {
            const int e = edge[j * P + c];
            const double f = widen(flux[e]);
            const double signed_flux = ((mask >> j) & 1u) ? f : -f;
            net = add_product<T>(net, signed_flux, length[e]);
        }
    }
    out[c] = static_cast<T>(quotient<T>(net, area[c], rarea[c]));
}

// ---- transport step -------------------------------------------------------------

// Right-hand side of (A/s) x + K L x = (A/s) T0 + A S, and the constant slope s = dt/C.
__global__ void k_step_rhs(std::uint32_t rows, const std::int32_t* __restrict__ tile_inst,
                           const std::int32_t* __restrict__ tile_rows, const double* __restrict__ area,
                           const double* __restrict__ slope_of, const double* __restrict__ t0,
                           const double* __restrict__ src, double* __restrict__ rhs,
                           double* __restrict__ slope, double* __restrict__ x0, unsigned long long* bytes) {
    const int tile = blockIdx.x;
    const int row = tile * kTile + threadIdx.x;
    // area, T0, S in; rhs, slope, x0 out
    if (bytes != nullptr && threadIdx.x == 0) atomicAdd(bytes, 48ull * static_cast<unsigned>(tile_rows[tile]));
    if (threadIdx.x >= tile_rows[tile]) {
        rhs[row] = 0.0;
        slope[row] = 1.0;
        x0[row] = 0.0;
        return;
    }
    const double s = slope_of[tile_inst[tile]];
    slope[row] = s;
    const double a = area[row];
    rhs[row] = dadd(dmul(__ddiv_rn(a, s), t0[row]), dmul(a, src[row]));
    x0[row] = t0[row];
}

// Flux form of the solved temperature: H = (1/A) sum_k G_k w_k (T_k - T_c), with G
// the planet's K or the per-entry conductance; T_new = T0 + s (S + H). Per-tile
// partial sums, then per-planet sums in k_sum_tiles' tree: sum A H, sum A |H|, sum A H T,
// sum A S, sum A |S|, sum A (T_new - T0) / s.
__global__ void k_step_finish(std::uint32_t P, const std::int32_t* __restrict__ tile_inst,
                              const std::int32_t* __restrict__ tile_rows,
                              const std::int32_t* __restrict__ nbr, const double* __restrict__ w,
                              const double* __restrict__ area, const double* __restrict__ conductance,
                              const double* __restrict__ edge_conductance,
                              const double* __restrict__ slope_of, const double* __restrict__ t,
                              const double* __restrict__ t0, const double* __restrict__ src,
                              double* __restrict__ h_out, double* __restrict__ t_new,
                              double* __restrict__ partial, unsigned long long* bytes) {
    const int tile = blockIdx.x;
    const int row = tile * kTile + threadIdx.x;
    const int inst = tile_inst[tile];
    // columns, weights (and per-entry conductances), area, T, T0, S in; H, T_new out
    if (bytes != nullptr && threadIdx.x == 0)
        atomicAdd(bytes, (edge_conductance != nullptr ? 168ull : 120ull) * static_cast<unsigned>(tile_rows[tile]));
    double v[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};   // six, and two zeros that fill up the tree
    if (threadIdx.x < tile_rows[tile]) {
        const double own = t[row];
        double sum = 0.0;
        double h;
        if (edge_conductance == nullptr) {
#pragma unroll
            for (int j = 0; j < 6; ++j) sum = dadd(sum, dmul(dsub(t[nbr[j * P + row]], own), w[j * P + row]));
            h = __ddiv_rn(dmul(conductance[inst], sum), area[row]);
        } else {
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const double g = dmul(edge_conductance[j * P + row], w[j * P + row]);
                sum = dadd(sum, dmul(g, dsub(t[nbr[j * P + row]], own)));
            }
            h = __ddiv_rn(sum, area[row]);
        }
        const double s = slope_of[inst];
        const double tn = dadd(t0[row], dmul(s, dadd(src[row], h)));
        h_out[row] = h;
        t_new[row] = tn;
        const double a = area[row];
        const double flux = dmul(a, h);
        v[0] = flux;
        v[1] = fabs(flux);
        v[2] = dmul(flux, own);
        v[3] = dmul(a, src[row]);
        v[4] = fabs(v[3]);
        v[5] = dmul(a, __ddiv_rn(dsub(tn, t0[row]), s));
    }
    ph::group_sum<double, 8>(v, 0, threadIdx.x);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < 6; ++q) partial[tile * 8 + q] = v[q];
    }
}

// Per-planet sums of the tile partials in a fixed tree: warp q sums quantity q, lane l tiles
// l, l + 32, ... in order (eight loads in flight), then the butterfly. One thread a quantity in
// tile order, a load and an addition after the other, took 273 us on a level-8 planet's 2,561
// tiles; this takes 8.
constexpr int kSumWarps = 6;
__global__ void __launch_bounds__(32 * kSumWarps) k_sum_tiles(std::uint32_t instances,
                                                              const std::uint32_t* __restrict__ tile_begin,
                                                              const double* __restrict__ partial,
                                                              double* __restrict__ out) {
    const std::uint32_t inst = blockIdx.x;
    if (inst >= instances) return;
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const std::uint32_t begin = tile_begin[inst], end = tile_begin[inst + 1];
    double s = 0.0;
    for (std::uint32_t t0 = begin + lane; t0 < end; t0 += 8 * 32) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = t0 + 32u * u < end ? partial[(t0 + 32u * u) * 8 + q] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (t0 + 32u * u < end) s += v[u];
        }
    }
    s = warp_sum(s);
    if (lane == 0) out[inst * 8 + q] = s;
}

__global__ void k_mask_rhs(std::size_t n, const double* __restrict__ slope, double* __restrict__ rhs) {
    const std::size_t i = blockIdx.x * std::size_t(blockDim.x) + threadIdx.x;
    if (i < n && !(slope[i] > 0.0)) rhs[i] = 0.0;
}

}  // namespace

void launch_mask_rhs(std::size_t n, const double* slope, double* rhs, cudaStream_t st) {
    PSGB_LAUNCH(kFamStep, st, k_mask_rhs<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(n, slope, rhs));
}

void fill_reciprocals(const DevMesh& m) {
    const auto fill = [](std::size_t n, const double* d, double* r) {
        k_reciprocal<<<static_cast<unsigned>((n + 255) / 256), 256>>>(n, d, r);
        PSGB_CUDA(cudaGetLastError());
    };
    fill(std::size_t(6) * m.p, m.dist, m.rdist);
    fill(m.p, m.area, m.rarea);
    fill(m.p, m.gm + std::size_t(3) * m.p, m.rdet);
    PSGB_CUDA(cudaStreamSynchronize(nullptr));
}

template <typename T>
void launch_laplacian(const DevMesh& m, const T* in, T* out, cudaStream_t st) {
    const unsigned g = (m.n + kOperatorThreads - 1) / kOperatorThreads;
    PSGB_LAUNCH(kFamOperator, st, k_laplacian<T><<<g, kOperatorThreads, 0, st>>>(m.n, m.p, m.nbr, m.w, m.area, m.rarea, in, out));
}
template <typename T>
void launch_gradient(const DevMesh& m, const T* in, T* east, T* north, cudaStream_t st) {
    const unsigned g = (m.n + kOperatorThreads - 1) / kOperatorThreads;
    PSGB_LAUNCH(kFamOperator, st, k_gradient<T><<<g, kOperatorThreads, 0, st>>>(m.n, m.p, m.nbr, m.degree, m.dist, m.rdist, m.ne, m.nn,
                                                                              m.gm, m.rdet, in, east, north));
}
template <typename T>
void launch_divergence(const DevMesh& m, const T* flux, T* out, cudaStream_t st) {
    const unsigned g = (m.n + kOperatorThreads - 1) / kOperatorThreads;
    PSGB_LAUNCH(kFamOperator, st, k_divergence<T><<<g, kOperatorThreads, 0, st>>>(m.n, m.p, m.edge, m.first, m.degree, m.edge_length,
                                                                                m.area, m.rarea, flux, out));
}
void launch_diffusion_source(const DevMesh& m, double conductance, const double* t, double* out,
                             cudaStream_t st) {
    PSGB_LAUNCH(kFamOperator, st, k_diffusion_source<<<(m.n + 255) / 256, 256, 0, st>>>(m.n, m.p, m.nbr, m.w, m.graph_area, conductance, t, out));
}

void launch_group_mean(const DevMesh& m, const double* a, const double* b, double* mean_a, double* mean_b,
                       cudaStream_t st) {
    PSGB_LAUNCH(kFamOperator, st, k_group_mean<<<(m.n + 255) / 256, 256, 0, st>>>(m.n, m.member_offset, m.member, m.fine_area,
                                                                               m.graph_area, a, b, mean_a, mean_b));
}
void launch_group_scatter(const DevMesh& m, const double* node_value, double* out, cudaStream_t st) {
    PSGB_LAUNCH(kFamOperator, st, k_group_scatter<<<(m.fine_cells + 255) / 256, 256, 0, st>>>(m.fine_cells, m.group_of_cell,
                                                                                           node_value, out));
}

template void launch_laplacian<float>(const DevMesh&, const float*, float*, cudaStream_t);
template void launch_laplacian<double>(const DevMesh&, const double*, double*, cudaStream_t);
template void launch_gradient<float>(const DevMesh&, const float*, float*, float*, cudaStream_t);
template void launch_gradient<double>(const DevMesh&, const double*, double*, double*, cudaStream_t);
template void launch_divergence<float>(const DevMesh&, const float*, float*, cudaStream_t);
template void launch_divergence<double>(const DevMesh&, const double*, double*, cudaStream_t);

void launch_step_rhs(const StepView& v, const double* t0, const double* src, double* rhs, double* slope,
                     double* x0, cudaStream_t st) {
    PSGB_LAUNCH(kFamStep, st, k_step_rhs<<<v.tiles, kTile, 0, st>>>(v.rows, v.tile_inst, v.tile_rows, v.area, v.slope_of, t0, src,
                                          rhs, slope, x0, v.bytes));
}

void launch_step_finish(const StepView& v, const double* t, const double* t0, const double* src,
                        double* h, double* t_new, double* partial, double* sums, cudaStream_t st) {
    PSGB_LAUNCH(kFamStep, st, k_step_finish<<<v.tiles, kTile, 0, st>>>(v.rows, v.tile_inst, v.tile_rows, v.nbr, v.w, v.area,
                                             v.conductance, v.edge_conductance, v.slope_of, t, t0, src, h,
                                             t_new, partial, v.bytes));
    PSGB_LAUNCH(kFamStep, st, k_sum_tiles<<<v.instances, 32 * kSumWarps, 0, st>>>(v.instances, v.tile_begin, partial, sums));
}

}  // namespace psgb
