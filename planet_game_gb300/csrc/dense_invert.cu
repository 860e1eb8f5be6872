// The inverse of every planet's coarsest level (the reference's factor_dense,
// sim/planet/surface/heat_transport.cpp:202-226, solved for every unit vector): symmetric
// positive definite, at most 400 rows, Gauss-Jordan in place without pivoting.
//
// n pivots in turn, each n^2 FP64 multiply-adds: in one block with the matrix in global memory a
// pivot took 8 us (162 rows: 1.25 ms, 222 rows: 3.5 ms, most of a matrix's assembly), the FP64
// pipe of one SM (two results a cycle) and the trips to L2 about equally. Here a planet takes a
// cluster, its rows shared out over the blocks' shared memory, so a pivot costs n^2 / C
// multiply-adds a block. The block that holds the next pivot's row updates that row first,
// scales it and stores it into every block while the other rows are still being updated, so one
// cluster barrier a pivot is all the blocks wait for. Every element goes through the same
// operations in the same order as in one block: the same bits. A new L4 planet's first step went
// from 2.9 to 2.1 ms with it (162 rows), a solve that assembles for every Newton step from 6.24 to
// 6.18 (42 rows, 65 us an inverse before).
#include "common.cuh"
#include "host/per_device.hpp"
#include "kernels.hpp"
#include "phases.cuh"
#include "profile.hpp"

#include <array>
#include <stdexcept>
#include <string>

namespace psgb {
namespace {

constexpr int kInvertThreads = 256;
constexpr int kInvertWarps = kInvertThreads / 32;

__device__ __forceinline__ void store_in_block(std::uint32_t address, unsigned rank, double v) {
    std::uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(address), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__device__ __forceinline__ void meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(kInvertThreads) k_dense_invert(DenseView dense, int level, LevelView<double> lv, int cluster,
                                                                double* __restrict__ inv64, float* __restrict__ inv32) {
    pdl_begin();
    const int inst = static_cast<int>(blockIdx.x) / cluster, rank = static_cast<int>(blockIdx.x) % cluster;
    if (dense.level[inst] != level) return;   // the whole cluster
    const int n = static_cast<int>(dense.size[inst]);
    const std::int64_t base = dense.row_base[inst];
    const int span = (n + cluster - 1) / cluster;   // row i: block i % cluster, its row i / cluster
    extern __shared__ double invert_smem[];
    double* a = invert_smem;                        // [span][n]
    double* pivot = a + static_cast<std::size_t>(span) * n;   // [2][n]: the scaled pivot rows, alternating
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const std::uint32_t P = lv.rows, W = lv.width;
    for (int idx = threadIdx.x; idx < span * n; idx += kInvertThreads) a[idx] = 0.0;
    __syncthreads();
    for (int s = threadIdx.x; s < span; s += kInvertThreads) {
        const int i = s * cluster + rank;
        if (i >= n) break;
        const std::int64_t row = base + i;
        a[s * n + i] = lv.vd[W * P + row];
        for (std::uint32_t j = 0; j < W; ++j) {
            const std::int64_t c = lv.col[j * P + row];
            if (c == row) continue;
            a[s * n + (c - base)] += lv.vd[j * P + row];
        }
    }
    // One warp: row k of this block scaled by its pivot, kept and stored into every block.
    const auto scale = [&](int k, int s) {
        double* row = a + static_cast<std::size_t>(s) * n;
        const double inverse = 1.0 / row[k];
        __syncwarp();
        const std::uint32_t to = static_cast<std::uint32_t>(__cvta_generic_to_shared(pivot + (k & 1) * n));
        for (int j = lane; j < n; j += 32) {
            const double v = (j == k ? 1.0 : row[j]) * inverse;
            row[j] = v;
            for (int r = 0; r < cluster; ++r) store_in_block(to + static_cast<std::uint32_t>(j) * 8u, static_cast<unsigned>(r), v);
        }
        __syncwarp();
    };
    meet();   // every block has started, and its rows stand
    if (rank == 0 && warp == 0) scale(0, 0);
    meet();
    for (int k = 0; k < n; ++k) {
        const double* p = pivot + (k & 1) * n;
        const int next = k + 1;
        const int mine = next < n && next % cluster == rank ? next / cluster : -1;   // the next pivot's row, if here
        const auto update = [&](int s) {
            double* row = a + static_cast<std::size_t>(s) * n;
            const double f = row[k];
            __syncwarp();
            for (int j = lane; j < n; j += 32) row[j] = __fma_rn(-f, p[j], j == k ? 0.0 : row[j]);
            __syncwarp();
        };
        if (mine >= 0 && warp == mine % kInvertWarps) {
            update(mine);
            scale(next, mine);
        }
        for (int s = warp; s < span; s += kInvertWarps) {
            const int i = s * cluster + rank;
            if (i >= n || i == k || s == mine) continue;
            update(s);
        }
        meet();
    }
    for (int idx = threadIdx.x; idx < span * n; idx += kInvertThreads) {
        const int i = (idx / n) * cluster + rank;
        if (i >= n) break;
        const std::size_t at = dense.offset[inst] + static_cast<std::size_t>(i) * n + idx % n;
        inv64[at] = a[idx];
        inv32[at] = static_cast<float>(a[idx]);
    }
}

std::size_t invert_bytes(int n, int cluster) {
    return (static_cast<std::size_t>((n + cluster - 1) / cluster) * n + 2 * static_cast<std::size_t>(n)) * sizeof(double);
}

}  // namespace

void launch_dense_invert(const DenseView& dense, int level, const LevelView<double>& lv, std::uint32_t max_rows,
                         std::uint32_t planets, double* inv64, float* inv32, cudaStream_t st) {
    static PerDevice<bool> ready;
    ready.of(current_device(), [] {
        if (cudaFuncSetAttribute(k_dense_invert, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
            cudaFuncSetAttribute(k_dense_invert, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            throw std::runtime_error("dense inverse: the device cannot launch its clusters");
        return true;
    });
    // As many blocks a planet as let every planet run at once (clusters of 16, 8, 4 and 2 with
    // full shared memory that are resident on 152 SMs: 7, 15, 36, 76), and as its rows need.
    const int n = static_cast<int>(max_rows);
    int cluster = planets <= 7 ? 16 : planets <= 15 ? 8 : planets <= 36 ? 4 : 2;
    while (cluster > 1 && cluster * 4 > n) cluster /= 2;   // at least four rows a block
    while (cluster < 16 && invert_bytes(n, cluster) > 227 * 1024) cluster *= 2;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(dense.instances * static_cast<unsigned>(cluster));
    cfg.blockDim = dim3(kInvertThreads);
    cfg.dynamicSmemBytes = invert_bytes(n, cluster);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    PSGB_LAUNCH(kFamSetup, st, {
        const cudaError_t e = cudaLaunchKernelEx(&cfg, k_dense_invert, dense, level, lv, cluster, inv64, inv32);
        if (e != cudaSuccess) throw std::runtime_error(std::string("dense inverse launch: ") + cudaGetErrorString(e));
    });
}

}  // namespace psgb
