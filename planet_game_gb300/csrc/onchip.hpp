// Solves held on chip: one planet per thread-block cluster, its matrix hierarchy and every
// vector of the solve spread over the shared memory and registers of the cluster's blocks.
//
// k_onchip_solve (onchip_kernel.cuh) runs a whole refined BiCGSTAB solve in one launch.
// Arguments are plain device pointers, sizes and shared-memory offsets, filled by the host
// driver (onchip.cpp).
#pragma once

#include "kernels.hpp"
#include "persistent.hpp"

#include <cuda_runtime.h>

#include <cstdint>

namespace psgb {

// A row's place in the cluster in 16 bits: block rank in bits 12-15, row of the block below.
constexpr unsigned kOnchipRankShift = 12;
constexpr unsigned kOnchipMaxSpan = 1u << kOnchipRankShift;
constexpr unsigned kOnchipMaxCluster = 16;
constexpr unsigned kOnchipMaxTiles = 256;   // fine-level tiles of a planet (a reduction sums eight sets of 32, a lane a tile)

template <typename T>
struct OnchipLevel {
    const std::int32_t* col;   // [width][pitch], batch rows
    const T* vd;               // [width + 1][pitch]
    const T* inv;              // [pitch]
    const std::int32_t* agg;   // [pitch]: row on the next level (absent on the coarsest)
    const std::uint32_t* moff; // next level's member lists
    const std::uint32_t* member;
    std::uint32_t pitch;
    std::uint32_t width;       // ELL width: 6 or 8
    std::uint32_t n;           // rows of each planet of the launch
    std::uint32_t span;        // rows a block holds
    // byte offsets in the block's shared memory
    std::uint32_t o_m, o_col, o_agg, o_moff, o_mem, o_x, o_y, o_b, o_r;
    int pre, post, inner;
    int starts_in_x;
    T correction;
};

template <typename T>
struct OnchipArgs {
    OnchipLevel<T> level[kMaxLevels];
    int coarsest;                       // the last level
    int cluster;                        // blocks per planet
    std::uint32_t planets;              // planets of the launch
    std::uint32_t instances;            // planets of the batch
    const std::uint32_t* list;          // [planets] their indices in the batch (null: 0, 1, ...)
    const std::uint32_t* tile_range;    // [levels][instances][2]
    const std::uint64_t* dense_offset;  // per planet, into dense_inv
    const T* dense_inv;
    std::uint32_t o_dense, o_phat, o_shat, o_part, o_list;
    std::uint32_t o_part2;              // reductions' partials alternate between o_part and here
    T omega;
    InstanceScalars* sc;
    const std::int32_t* fine_col;
    const double* fine_vd64;
    const double* rhs64;
    double* x64;
    const std::uint8_t* active;
    double tolerance, inner_tolerance;
    int max_iterations, max_refinements;
};

constexpr unsigned kOnchipThreads = 384;   // a block's at most

// One translation unit per precision. R: fine rows per thread (1, 2, 4 or, in FP32, 7).
template <typename T>
bool onchip_has(int rows_per_thread);
// Whether the solve kernel keeps its fine rows in registers (else in shared memory).
template <typename T>
constexpr bool onchip_held(int rows_per_thread) { return sizeof(T) * rows_per_thread <= 16; }
// The most phases a V-cycle's list may hold, and one's bytes.
constexpr int kOnchipMaxPhases = 256;
constexpr unsigned kOnchipPhaseBytes = 48;
template <typename T>
int onchip_active_clusters(int rows_per_thread, unsigned cluster, unsigned threads, std::size_t shared_bytes);
template <typename T>
void onchip_launch(const OnchipArgs<T>& args, int rows_per_thread, unsigned threads, std::size_t shared_bytes,
                   cudaStream_t st);

}  // namespace psgb
