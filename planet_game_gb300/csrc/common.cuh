// Shared device-side helpers for the GB300 heat-transport kernels.
//
// Layout conventions used by every kernel:
//  * rows of a level are padded to a multiple of kTile (256) so that a tile -
//    the reference's deterministic 256-cell block (planet_mesh.hpp:76) - never
//    straddles two planets of a batch;
//  * neighbour data is ELL, slot-major: entry (slot j, row r) sits at j * P + r for a
//    level with padded row count P, so a warp reads 32 consecutive rows of one slot
//    (fully coalesced); rows with fewer neighbours pad with (column = row, value = 0);
//  * every reduction is deterministic: a fixed warp-shuffle tree inside a tile,
//    per-tile partials in global memory, and the last tile of a planet to finish
//    (integer ticket) sums that planet's partials in tile order.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <stdexcept>
#include <string>
#include <utility>

namespace psgb {

constexpr int kTile = 256;

// The device of the calling thread (-1: none).
inline int current_device() {
    int device = -1;
    if (cudaGetDevice(&device) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return device;
}

// Programmatic dependent launch. Solve kernels run back to back on one stream, each
// short; launched with launch_pdl, a kernel's blocks may be scheduled while its
// predecessor drains. Every such kernel starts with pdl_begin(): it waits until the
// predecessor grid has completed and its writes are visible (so nothing is read early),
// then allows the successor to be scheduled. Measured on GB300 in CUDA graphs, early
// scheduling saves ~0.2 us per launch for grids of up to a few hundred blocks and costs
// up to 4 us for grids of thousands (their waiting blocks hold the SMs' block slots), so
// only grids of at most kPdlMaxBlocks blocks take it; pdl_begin() is free for the others.
__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

constexpr unsigned kPdlMaxBlocks = 1024;

template <typename... P, typename... A>
inline void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A&&... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = grid.x * grid.y * grid.z <= kPdlMaxBlocks ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
    if (e != cudaSuccess) throw std::runtime_error(std::string("kernel launch: ") + cudaGetErrorString(e));
}

// Warp-level sum in a fixed butterfly order (result valid in every lane).
template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Double precision add/multiply that the compiler may not fuse into an FMA, for
// sums whose rounding must match the reference's sequential CPU loops.
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }

// An SM starts an FP64 instruction of a warp every 19 cycles; a comparison or a conversion of a
// double counts as one, whole-number work beside them is free.

// The reciprocal that divide_by() takes: RN(1/d) of a d of ordinary size, else 0.
__device__ __forceinline__ double reciprocal_of(double d) {
    return fabs(d) > 0x1p-100 && fabs(d) < 0x1p100 ? __ddiv_rn(1.0, d) : 0.0;
}

// s / d, correctly rounded, in five operations on r = reciprocal_of(d) (Markstein, IBM J. Res.
// Dev. 34, 1990: with r = RN(1/d) and a quotient q within one unit in the last place,
// RN(q + r (s - d q)) is RN(s/d); one such step from q = RN(s r) gives that quotient, the next
// rounds it). A dividend so large or small that a remainder could leave the range is divided.
__device__ __forceinline__ double divide_by(double s, double d, double r) {
    const std::uint32_t high = static_cast<std::uint32_t>(__double2hiint(s)) & 0x7fffffffu;
    constexpr std::uint32_t low = (1023u - 800u) << 20, span = 1600u << 20;   // 2^-800 <= |s| < 2^800
    if (__double2hiint(r) != 0 && high - low < span) {
        double q = __dmul_rn(s, r);
        q = __fma_rn(__fma_rn(-d, q, s), r, q);
        return __fma_rn(__fma_rn(-d, q, s), r, q);
    }
    if (__double2hiint(r) != 0 && (high | static_cast<std::uint32_t>(__double2loint(s))) == 0u) return __dmul_rn(s, r);
    return __ddiv_rn(s, d);
}

// A float as a double, put together from its bits; zero, subnormals, infinities and NaN are converted.
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double widen(float v) {
    const std::uint32_t u = __float_as_uint(v), exponent = u & 0x7f800000u;
    if (exponent - 0x00800000u < 0x7f000000u)
        return __hiloint2double(static_cast<int>((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))),
                                static_cast<int>(u << 29));
    return static_cast<double>(v);
}

}  // namespace psgb
