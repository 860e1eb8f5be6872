// Device side of the on-chip solves (onchip.hpp); included by one translation unit per
// precision (onchip_f32.cu, onchip_f64.cu).
//
// What bounds a small planet's solve is not bandwidth but the chain of its phases: a level-5
// V-cycle is a dozen dependent phases of a few hundred nanoseconds of work, and as a kernel
// each costs a launch plus three dependent trips to L2 (tile word, column, neighbour), 2.5
// to 4 us. Here a thread-block cluster keeps the planet's matrix, columns, aggregates and
// vectors in its blocks' shared memory from the first refinement to the last: a phase is one
// gather through distributed shared memory and one cluster barrier, 0.36 us in FP32 with 192
// rows a block and 0.48 us with 672 (a probe of six remote gathers, their multiply-adds, a
// store and the barrier; the barrier alone is 0.19 us), where a grid barrier alone costs 1.3.
//
// Rows are shared out in 32-row warps (256-row tiles on a level with block-local sweeps), so
// that the blocks differ by at most one warp and every reduction keeps the tile tree of
// phases.cuh: a warp's partial, the eight warps of a tile in order, the tiles as sum_partials
// adds them. Every row's arithmetic is phases.cuh's, spelled out as the fused multiply-adds
// the compiler forms there, so the results are the kernel schedule's bit for bit.
#pragma once

#define PSGB_PHASE_RESTRICT
#include "host/per_device.hpp"
#include "onchip.hpp"
#include "phases.cuh"

#include <array>
#include <stdexcept>
#include <string>
#include <type_traits>

namespace psgb {
namespace oc {

using ph::fnma;

__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
using ph::prod;

// All writes of this block before it are visible to the cluster's blocks after it.
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The same in two halves: what other blocks do not write may be read in between.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// The address in block `rank`'s shared memory that `a` is in this block's. Not volatile: the
// addresses of many gathers are formed side by side, ahead of the loads (in program order with
// its load each took about 25 cycles of its own).
__device__ __forceinline__ std::uint32_t in_block(std::uint32_t a, std::uint32_t rank) {
    std::uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

// The address of a row's entry in the vector at the start of shared memory; that of the vector
// at offset o is o more.
template <typename T>
__device__ __forceinline__ std::uint32_t entry_of(std::uint32_t base, std::uint32_t code) {
    return in_block(base + (code & (kOnchipMaxSpan - 1)) * static_cast<std::uint32_t>(sizeof(T)), code >> kOnchipRankShift);
}

// The entries at `at[N]` of the vector at offset `vec`.
template <int N>
__device__ __forceinline__ void gather(std::uint32_t vec, const std::uint32_t (&at)[N], float (&v)[N]) {
#pragma unroll
    for (int j = 0; j < N; ++j) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[j]) : "r"(at[j] + vec) : "memory");
}
template <int N>
__device__ __forceinline__ void gather(std::uint32_t vec, const std::uint32_t (&at)[N], double (&v)[N]) {
#pragma unroll
    for (int j = 0; j < N; ++j) asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v[j]) : "r"(at[j] + vec) : "memory");
}

// v to entry `at` of the vector at shared-memory address `vec` in block `rank`.
__device__ __forceinline__ void scatter(std::uint32_t vec, std::uint32_t rank, std::uint32_t at, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(in_block(vec + at * 4u, rank)), "f"(v) : "memory");
}
__device__ __forceinline__ void scatter(std::uint32_t vec, std::uint32_t rank, std::uint32_t at, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(in_block(vec + at * 8u, rank)), "d"(v) : "memory");
}

struct Block {
    unsigned char* smem;
    std::uint32_t base;    // shared-memory address of smem
    std::uint32_t rank;    // in the cluster
    int tid, lane, warp, threads, warps;
    template <typename V>
    __device__ __forceinline__ V* at(std::uint32_t offset) const { return reinterpret_cast<V*>(smem + offset); }
};

__device__ __forceinline__ Block block_of(unsigned char* smem) {
    Block k;
    k.smem = smem;
    k.base = static_cast<std::uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(k.rank));
    k.tid = static_cast<int>(threadIdx.x);
    k.lane = k.tid & 31;
    k.warp = k.tid >> 5;
    k.threads = static_cast<int>(blockDim.x);
    k.warps = k.threads >> 5;
    return k;
}

// Rows of a level this block holds.
__device__ __forceinline__ int own_rows(std::uint32_t n, std::uint32_t span, std::uint32_t rank) {
    const std::uint32_t first = rank * span;
    return first >= n ? 0 : static_cast<int>(n - first < span ? n - first : span);
}
__device__ __forceinline__ std::uint16_t place_of(std::uint32_t row, std::uint32_t span) {
    const std::uint32_t rank = row / span;
    return static_cast<std::uint16_t>((rank << kOnchipRankShift) | (row - rank * span));
}

// A row in shared memory: its W off-diagonals, diagonal and 1 / diagonal as 16-byte words,
// word-major (word q of the block's row i at m[q * span + i]), so that a warp reads each word
// in one conflict-free 128-bit access and a row needs 2 (FP32, W = 6) to 5 (FP64, W = 8) of
// them, where slot-major values and 16-bit columns took 15 to 19 accesses and as many
// addresses in registers (the whole solve then spilled). W is 6 on the fine level and 8 on
// every coarse one; narrower rows pad with zero couplings to themselves. The columns' places
// fill one more 16-byte word; the fine level's seventh entry is the row's aggregate.
template <typename T, int W>
struct RowWords {
    static constexpr int per = 16 / static_cast<int>(sizeof(T));
    static constexpr int count = (W + 2 + per - 1) / per;
};

template <typename T, int W>
struct MatrixRow {
    T v[RowWords<T, W>::count * RowWords<T, W>::per];   // off-diagonals, then diagonal, 1 / diagonal
    __device__ __forceinline__ T diagonal() const { return v[W]; }
    __device__ __forceinline__ T inverse() const { return v[W + 1]; }
};

template <int W>
__device__ __forceinline__ MatrixRow<float, W> matrix_row(const float4* m, std::uint32_t span, int row, float) {
    MatrixRow<float, W> r;
#pragma unroll
    for (int q = 0; q < RowWords<float, W>::count; ++q) {
        const float4 w = m[q * span + row];
        r.v[4 * q] = w.x; r.v[4 * q + 1] = w.y; r.v[4 * q + 2] = w.z; r.v[4 * q + 3] = w.w;
    }
    return r;
}
template <int W>
__device__ __forceinline__ MatrixRow<double, W> matrix_row(const float4* m, std::uint32_t span, int row, double) {
    MatrixRow<double, W> r;
    const double2* d = reinterpret_cast<const double2*>(m);
#pragma unroll
    for (int q = 0; q < RowWords<double, W>::count; ++q) {
        const double2 w = d[q * span + row];
        r.v[2 * q] = w.x; r.v[2 * q + 1] = w.y;
    }
    return r;
}

// Entry j of a row's eight 16-bit places.
__device__ __forceinline__ std::uint32_t place(const uint4& c, int j) {
    const std::uint32_t w = j < 2 ? c.x : j < 4 ? c.y : j < 6 ? c.z : c.w;
    return (j & 1) != 0 ? w >> 16 : w & 0xFFFFu;
}

constexpr int kCoarseWidth = 8;

// A fine row's matrix entries and places, as the level's arrays have them; `self` where the
// planet's row is missing (a thread without a row).
template <typename T>
struct FineRow {
    MatrixRow<T, 6> m;
    std::uint32_t code[7];   // the neighbours' places, the aggregate's
};
template <typename T>
__device__ __forceinline__ FineRow<T> fetch_fine(const OnchipLevel<T>& L, const OnchipLevel<T>& C, std::uint32_t g,
                                                 std::uint32_t row0, std::uint32_t next0) {
    FineRow<T> r;
#pragma unroll
    for (int j = 0; j < 7; ++j) r.m.v[j] = __ldcg(&L.vd[std::size_t(j) * L.pitch + g]);
    r.m.v[7] = __ldcg(&L.inv[g]);
#pragma unroll
    for (int j = 0; j < 6; ++j) r.code[j] = place_of(static_cast<std::uint32_t>(L.col[std::size_t(j) * L.pitch + g]) - row0, L.span);
    r.code[6] = place_of(static_cast<std::uint32_t>(L.agg[g]) - next0, C.span);
    return r;
}

// The fine level into shared memory (solves whose threads hold too many rows for registers).
template <typename T>
__device__ void load_fine(const Block& k, const OnchipLevel<T>& L, const OnchipLevel<T>& C, std::uint32_t row0,
                          std::uint32_t next0) {
    const int rows = own_rows(L.n, L.span, k.rank);
    constexpr int per = RowWords<T, 6>::per;
    T* m = k.at<T>(L.o_m);
    uint4* col = k.at<uint4>(L.o_col);
    for (int i = k.tid; i < rows; i += k.threads) {
        const FineRow<T> r = fetch_fine(L, C, row0 + k.rank * L.span + i, row0, next0);
#pragma unroll
        for (int j = 0; j < 8; ++j) m[(static_cast<std::size_t>(j / per) * L.span + i) * per + j % per] = r.m.v[j];
        col[i] = make_uint4(r.code[0] | r.code[1] << 16, r.code[2] | r.code[3] << 16, r.code[4] | r.code[5] << 16, r.code[6]);
    }
    // threads without a row run through the block's row 0: its places stay in the cluster
    const std::uint32_t self = k.rank << kOnchipRankShift;
    if (rows == 0 && k.tid == 0) col[0] = make_uint4(self | self << 16, self | self << 16, self | self << 16, self);
}

// A coarse level into shared memory: matrix words, the neighbours' addresses (two words of
// four, word-major), the aggregate's address.
template <typename T>
__device__ void load_coarse(const Block& k, const OnchipLevel<T>& L, const OnchipLevel<T>& C, std::uint32_t row0,
                            std::uint32_t next0) {
    constexpr int W = kCoarseWidth, per = RowWords<T, W>::per;
    const int rows = own_rows(L.n, L.span, k.rank);
    const std::uint32_t g0 = row0 + k.rank * L.span;
    T* m = k.at<T>(L.o_m);
    std::uint32_t* col = k.at<std::uint32_t>(L.o_col);
    for (int i = k.tid; i < rows; i += k.threads) {
        const std::uint32_t self = (k.rank << kOnchipRankShift) | static_cast<std::uint32_t>(i);
        const auto word = [&](int j) -> T& { return m[(static_cast<std::size_t>(j / per) * L.span + i) * per + j % per]; };
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const bool real = static_cast<std::uint32_t>(j) < L.width;
            word(j) = real ? __ldcg(&L.vd[std::size_t(j) * L.pitch + g0 + i]) : T(0);
            const std::uint32_t code =
                real ? place_of(static_cast<std::uint32_t>(L.col[std::size_t(j) * L.pitch + g0 + i]) - row0, L.span) : self;
            col[(static_cast<std::size_t>(j / 4) * L.span + i) * 4 + j % 4] = entry_of<T>(k.base, code);
        }
        word(W) = __ldcg(&L.vd[std::size_t(L.width) * L.pitch + g0 + i]);
        word(W + 1) = __ldcg(&L.inv[g0 + i]);
        k.at<std::uint32_t>(L.o_agg)[i] = entry_of<T>(k.base, place_of(static_cast<std::uint32_t>(L.agg[g0 + i]) - next0, C.span));
    }
}

// The members of each own row of the next level: in `count` their number, and above bit 16 where
// their addresses start, in words of four; a row's are padded with its first to whole pairs of
// words. All threads of the block call it.
template <typename T>
__device__ void load_members(const Block& k, const OnchipLevel<T>& L, const OnchipLevel<T>& C, std::uint32_t row0,
                             std::uint32_t next0) {
    const int crows = own_rows(C.n, C.span, k.rank);
    const std::uint32_t c0 = next0 + k.rank * C.span;
    std::uint32_t* count = k.at<std::uint32_t>(L.o_moff);
    for (int i = k.tid; i < crows; i += k.threads) count[i] = L.moff[c0 + i + 1] - L.moff[c0 + i];
    __syncthreads();
    std::uint32_t* mem = k.at<std::uint32_t>(L.o_mem);
    for (int i = k.tid; i < crows; i += k.threads) {
        std::uint32_t start = 0;
        for (int j = 0; j < i; ++j) start += ((count[j] & 0xFFFFu) + 7u) / 8u * 2u;
        const std::uint32_t n = count[i] & 0xFFFFu, m0 = L.moff[c0 + i], end = (n + 7u) / 8u * 8u;
        for (std::uint32_t m = 0; m < end; ++m)
            mem[start * 4u + m] = entry_of<T>(k.base, place_of(L.member[m0 + (m < n ? m : 0u)] - row0, L.span));
        // other threads still read the number below bit 16
        count[i] = n | start << 16;
    }
}

// The coarsest inverse's rows this block solves.
template <typename T>
__device__ void load_dense(const Block& k, const OnchipArgs<T>& a, int inst) {
    const OnchipLevel<T>& L = a.level[a.coarsest];
    const int rows = own_rows(L.n, L.span, k.rank), n = static_cast<int>(L.n);
    const T* src = a.dense_inv + a.dense_offset[inst] + std::size_t(k.rank) * L.span * n;
    T* dst = k.at<T>(a.o_dense);
    for (int i = k.tid; i < rows * n; i += k.threads) dst[i] = __ldcg(&src[i]);
}

// ---- the V-cycle as a list of phases ------------------------------------------------------------
//
// The code of a phase stands once and the cycle walks a list of phases, one cluster barrier
// each. What a phase reads that no block writes (its entry in the list, matrix words,
// addresses) is loaded between the arrival at the barrier before it and the wait. A phase is a
// few warps' worth of work, so its time is that of its longest chain of instructions: addresses
// are held ready made (a shift, a mask, a `mapa` and an addition a gather otherwise, 150 of a
// row's 250 instructions), and a row's words come in 128-bit loads.

enum Op : std::uint32_t { kSweep, kBlockSweep, kResidual, kRestrict, kDense, kProlong };

struct __align__(16) Phase {
    std::uint32_t kind;     // Op, bit 8: a phase of the fine level
    std::uint32_t rows;     // this block's rows of the level it writes
    std::uint32_t span;     // rows a block holds of that level (word-major arrays' stride)
    std::uint32_t m;        // matrix words (dense: the inverse's rows; restriction: member words)
    std::uint32_t col;      // addresses (restriction: member counts; prolongation: aggregates)
    std::uint32_t src;      // vectors: read at the gathered entries ...
    std::uint32_t dst;      // ... written
    std::uint32_t b;        // right-hand side (restriction: written)
    std::uint32_t aux;      // dense: rows; restriction: where 1 / diagonal lies, 16 bytes a row (0: coarsest level)
    std::uint32_t inner;    // block-local sweeps
    double correction;      // prolongation
};
static_assert(sizeof(Phase) == kOnchipPhaseBytes, "the host lays the list out");
constexpr std::uint32_t kFinePhase = 256u;
constexpr std::uint32_t kHat = 0xFFFFFFFFu;   // the vector the cycle is solving for (fine level)

template <typename T>
__device__ int build_cycle(const Block& k, const OnchipArgs<T>& a, Phase* out) {
    int n = 0;
    const auto x_of = [&](int l) { return l == 0 ? kHat : a.level[l].o_x; };
    const auto add = [&](std::uint32_t kind, int l, bool in_x) {
        const OnchipLevel<T>& L = a.level[l];
        Phase p{};
        p.kind = kind | (l == 0 ? kFinePhase : 0u);
        p.rows = static_cast<std::uint32_t>(own_rows(L.n, L.span, k.rank));
        p.span = L.span;
        p.m = L.o_m;
        p.col = L.o_col;
        p.src = in_x ? x_of(l) : L.o_y;
        p.dst = kind == kResidual ? L.o_r : (in_x ? L.o_y : x_of(l));
        p.b = L.o_b;
        p.inner = static_cast<std::uint32_t>(L.inner);
        if (kind == kProlong) {
            p.col = L.o_agg;
            p.dst = p.src;
            p.src = a.level[l + 1].o_x;
            p.correction = static_cast<double>(L.correction);
        } else if (kind == kRestrict) {
            const OnchipLevel<T>& C = a.level[l + 1];
            constexpr std::uint32_t at = kCoarseWidth + 1, per = RowWords<T, kCoarseWidth>::per;
            p.kind = kind;
            p.rows = static_cast<std::uint32_t>(own_rows(C.n, C.span, k.rank));
            p.span = C.span;
            p.m = L.o_mem;
            p.col = L.o_moff;
            p.src = L.o_r;
            p.dst = C.starts_in_x ? C.o_x : C.o_y;
            p.b = C.o_b;
            p.aux = l + 1 == a.coarsest ? 0u : C.o_m + (at / per) * C.span * 16u + (at % per) * static_cast<std::uint32_t>(sizeof(T));
            p.inner = k.rank * C.span;
        } else if (kind == kDense) {
            p.m = a.o_dense;
            p.dst = L.o_x;
            p.aux = L.n;
        }
        out[n++] = p;
    };
    for (int l = 0; l < a.coarsest; ++l) {
        const OnchipLevel<T>& L = a.level[l];
        bool in_x = L.starts_in_x != 0;
        for (int s = 1; s < L.pre; ++s, in_x = !in_x) add(L.inner > 1 ? kBlockSweep : kSweep, l, in_x);
        add(kResidual, l, in_x);
        add(kRestrict, l, in_x);
    }
    add(kDense, a.coarsest, true);
    for (int l = a.coarsest - 1; l >= 0; --l) {
        const OnchipLevel<T>& L = a.level[l];
        bool in_x = (L.starts_in_x != 0) == (((L.pre - 1) & 1) == 0);   // where the sweeps down ended
        add(kProlong, l, in_x);
        // the first post-sweep is fused with the prolongation elsewhere: a plain one
        for (int s = 0; s < L.post; ++s, in_x = !in_x) add(L.inner > 1 && s > 0 ? kBlockSweep : kSweep, l, in_x);
    }
    return n;
}

// What a phase of a coarse level reads that no block writes, this thread's (first) row.
template <typename T>
struct Ahead {
    MatrixRow<T, kCoarseWidth> m;
    std::uint32_t at[8];   // neighbours, the first eight members, or (at[0]) the aggregate
    std::uint32_t count;   // members, and where they start
};

__device__ __forceinline__ void words(const uint4& lo, const uint4& hi, std::uint32_t (&at)[8]) {
    at[0] = lo.x; at[1] = lo.y; at[2] = lo.z; at[3] = lo.w;
    at[4] = hi.x; at[5] = hi.y; at[6] = hi.z; at[7] = hi.w;
}

template <typename T>
__device__ __forceinline__ void load_ahead(const Block& k, const Phase& p, std::uint32_t kind, int i, Ahead<T>& h) {
    if (static_cast<std::uint32_t>(i) >= p.rows) return;
    const int span = static_cast<int>(p.span);
    if (kind == kProlong) {
        h.at[0] = k.at<std::uint32_t>(p.col)[i];
    } else if (kind == kRestrict) {
        h.count = k.at<std::uint32_t>(p.col)[i];
        const uint4* w = k.at<uint4>(p.m) + (h.count >> 16);
        words(w[0], w[1], h.at);
    } else if (kind != kDense) {
        h.m = matrix_row<kCoarseWidth>(k.at<float4>(p.m), p.span, i, T(0));
        const uint4* w = k.at<uint4>(p.col);
        words(w[i], w[span + i], h.at);
    }
}

// Block-local sweeps (phases.cuh `smooth_block`): the tile's own rows iterate in `dst`, its
// neighbours in other tiles held at `src`. Whole tiles belong to one block here and the
// block's threads are a multiple of 256 (or hold every row at once).
template <typename T>
__device__ __forceinline__ void sweep_block(const Block& k, const Phase& p, Ahead<T>& h, T omega) {
    constexpr int W = kCoarseWidth;
    const int rows = static_cast<int>(p.rows);
    T* y = k.at<T>(p.dst);
    for (int i0 = 0; i0 < rows; i0 += k.threads) {
        const int i = i0 + k.tid;
        const bool live = i < rows;
        const int row = live ? i : 0;
        if (i0 > 0 || !live) load_ahead(k, p, kBlockSweep, row, h);
        T held[W];
        gather(p.src, h.at, held);
        // a neighbour of the same tile: the same block's memory, the same 256 rows
        const std::uint32_t home = entry_of<T>(k.base, (k.rank << kOnchipRankShift) | (static_cast<std::uint32_t>(row) & ~255u));
        std::uint32_t local[W];
#pragma unroll
        for (int j = 0; j < W; ++j) local[j] = (h.at[j] - home) / static_cast<std::uint32_t>(sizeof(T));
        const int tile = row & ~255;
        const T bv = k.at<T>(p.b)[row];
        T xo = k.at<T>(p.src)[row];
        if (live) y[i] = xo;
        __syncthreads();
        for (std::uint32_t sweep = 0; sweep < p.inner; ++sweep) {
            T s = bv;
#pragma unroll
            for (int j = 0; j < W; ++j) s = fnma(h.m.v[j], local[j] < 256u ? y[tile + static_cast<int>(local[j])] : held[j], s);
            const T out = ph::jacobi_update(xo, omega, h.m.inverse(), s);
            __syncthreads();
            if (live) y[i] = out;
            xo = out;
            __syncthreads();
        }
    }
}

// A phase of the coarse levels, the restriction from the fine one among them (its barrier is
// the caller's).
template <typename T>
__device__ __forceinline__ void coarse_phase(const Block& k, const Phase& p, std::uint32_t kind, Ahead<T>& h, int cluster,
                                             T omega) {
    const int rows = static_cast<int>(p.rows);
    if (kind == kDense) {
        // x = A^-1 b, one warp a row, two rows at a time
        const int n = static_cast<int>(p.aux);
        const T* inv = k.at<T>(p.m);
        const T* b = k.at<T>(p.b);
        for (int row = k.warp; row < rows; row += 2 * k.warps) {
            const int other = row + k.warps < rows ? row + k.warps : row;
            T s0 = T(0), s1 = T(0);
#pragma unroll 2
            for (int j = k.lane; j < n; j += 32) {
                const T g = b[j];
                s0 = fma_(inv[row * n + j], g, s0);
                s1 = fma_(inv[other * n + j], g, s1);
            }
            const T both[2] = {s0, s1};
            T mine;
            int which;
            bool owner;
            ph::warp_sum_halving<T, 2>(both, k.lane, mine, which, owner);
            if (owner) k.at<T>(p.dst)[which == 0 ? row : other] = mine;
        }
        return;
    }
    if (kind == kBlockSweep) {
        sweep_block(k, p, h, omega);
        return;
    }
    for (int i = k.tid; i < rows; i += k.threads) {
        if (i != k.tid) load_ahead(k, p, kind, i, h);
        if (kind == kProlong) {   // x += correction * e[agg]
            const std::uint32_t at[1] = {h.at[0]};
            T e[1];
            gather(p.src, at, e);
            k.at<T>(p.dst)[i] = add_(k.at<T>(p.dst)[i], prod(static_cast<T>(p.correction), e[0]));
            continue;
        }
        T g[8];
        gather(p.src, h.at, g);
        if (kind == kRestrict) {
            // the members' residuals in ascending order, up to 24 gathers in flight (an aggregate
            // has 7 to 25 rows, 15 to 17 in the median); then the zero-start sweep. A coarsest
            // level's right-hand side is written to every block of the cluster, for the dense
            // rows to read at home.
            const int count = static_cast<int>(h.count & 0xFFFFu);
            const uint4* w = k.at<uint4>(p.m) + (h.count >> 16);
            T g1[8], g2[8];
            std::uint32_t at[8];
            if (count > 8) {
                words(w[2], w[3], at);
                gather(p.src, at, g1);
            }
            if (count > 16) {
                words(w[4], w[5], at);
                gather(p.src, at, g2);
            }
            T s = T(0);
#pragma unroll
            for (int j = 0; j < 8; ++j) s = j < count ? add_(s, g[j]) : s;
            if (count > 8) {
#pragma unroll
                for (int j = 0; j < 8; ++j) s = 8 + j < count ? add_(s, g1[j]) : s;
            }
            if (count > 16) {
#pragma unroll
                for (int j = 0; j < 8; ++j) s = 16 + j < count ? add_(s, g2[j]) : s;
            }
#pragma unroll 1
            for (int m = 24; m < count; m += 8) {
                words(w[m / 4], w[m / 4 + 1], at);
                gather(p.src, at, g);
                for (int j = 0; j < 8; ++j) s = m + j < count ? add_(s, g[j]) : s;
            }
            if (p.aux == 0u) {
                for (int r = 0; r < cluster; ++r)
                    scatter(k.base + p.b, static_cast<std::uint32_t>(r), p.inner + static_cast<std::uint32_t>(i), s);
            } else {
                k.at<T>(p.b)[i] = s;
                k.at<T>(p.dst)[i] = prod(prod(omega, *k.at<T>(p.aux + 16u * static_cast<std::uint32_t>(i))), s);
            }
            continue;
        }
        const T xo = k.at<T>(p.src)[i];
        T s = k.at<T>(p.b)[i];
        if (kind == kResidual) s = fnma(h.m.diagonal(), xo, s);
#pragma unroll
        for (int j = 0; j < kCoarseWidth; ++j) s = fnma(h.m.v[j], g[j], s);
        if (kind != kResidual) s = ph::sweep_update(xo, omega, h.m.inverse(), s);
        k.at<T>(p.dst)[i] = s;
    }
}

// ---- reductions ---------------------------------------------------------------------------------

struct Reduce {
    double tiles[2][8];            // sums of 32 tiles each
    InstanceScalars s;
    double tolerance, inner_tolerance;
    int max_iterations, max_refinements;
    std::uint32_t n;               // fine rows of the planet
    int phases;                    // of the cycle
};

// The scalar step of a reduction (phases.cuh) on its sums, thread 0.
__device__ __forceinline__ void scalar_step(Reduce& red, int kind, const double* sum) {
    InstanceScalars& s = red.s;
    switch (kind) {
        case ph::kFinOuterInit: ph::finish_outer_init(s, sum, red.tolerance); break;
        case ph::kFinOuterResidual: ph::finish_outer_residual(s, sum, red.max_refinements); break;
        case ph::kFinBicgInit: ph::finish_bicg_init(s, sum, red.inner_tolerance, red.max_iterations); break;
        case ph::kFinBicgV: ph::finish_bicg_v(s, sum); break;
        case ph::kFinBicgS: ph::finish_bicg_s(s, sum); break;
        case ph::kFinBicgT: ph::finish_bicg_t(s, sum); break;
        default: ph::finish_bicg_x(s, sum); break;
    }
}

// Completes a reduction: one or two quantities from the 32-row partials every block has at
// `part` (quantity-major, whole tiles of eight), a tile's eight partials in order, the tiles in
// sum_partials' tree, then the scalar step. Every block sums on its own, so that no result has
// to be sent back. A warp's FP64 instruction holds its scheduler's FP64 unit for 64 cycles (two
// results a cycle and SM), so the quantities and the sets of 32 tiles go to warps of their own,
// spread over the four schedulers: for a level-5 planet 3,100 cycles in one warp, its chains side
// by side.
template <typename A>
__device__ __noinline__ void finish(Block k, Reduce* red_p, std::uint32_t part, int kind, bool two) {
    Reduce& red = *red_p;
    cluster_barrier();
    const std::uint32_t chunks = (red.n + 31) / 32, tiles = (red.n + 255) / 256;
    const std::uint32_t sets = (tiles + 31) / 32;
    const std::uint32_t jobs = two ? 2 * sets : sets;
#pragma unroll 1
    for (std::uint32_t job = static_cast<std::uint32_t>(k.warp); job < jobs; job += static_cast<std::uint32_t>(k.warps)) {
        const std::uint32_t q = two ? job & 1u : 0u, set = two ? job >> 1 : job;
        const std::uint32_t t = 32u * set + static_cast<std::uint32_t>(k.lane);
        const A* at = k.at<A>(part) + 8u * (q * tiles + ::min(t, tiles - 1u));
        A v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = at[u];
        A s = v[0];
#pragma unroll
        for (int u = 1; u < 8; ++u) s = 8u * t + u < chunks ? add_(s, v[u]) : s;
        const double total = warp_sum(t < tiles ? static_cast<double>(s) : 0.0);
        if (k.lane == 0) red.tiles[q][set] = total;
    }
    __syncthreads();
    if (k.warp == 0) {
        // lane q: quantity q
        const int q = two ? k.lane & 1 : 0;
        double s = red.tiles[q][0];
#pragma unroll 1
        for (std::uint32_t w = 1; w < sets; ++w) s = __dadd_rn(s, red.tiles[q][w]);
        const double sum[2] = {s, __shfl_sync(0xffffffffu, s, 1)};
        if (k.lane == 0) scalar_step(red, kind, sum);
    }
    __syncthreads();
}

// This thread's rows of the fine level: chunk warp + r * warps, lane; a place past the block's
// rows is off and runs through row 0, storing nothing.
template <int R>
struct Rows {
    int row[R];
    bool on[R];
};

// 32-row partials of q[NQ][R] into every block's slots at shared-memory address `part`. Sent so, a reduction reads its partials at home; gathered by each block, a
// warp's load would reach a dozen blocks and be split as often.
template <typename T, int NQ, int R>
__device__ __forceinline__ void write_partials(const Block& k, std::uint32_t part, std::uint32_t stride, std::uint32_t chunk0,
                                               int cluster, const T (&q)[NQ][R], int rows) {
    // the chains by recursive halving (phases.cuh): every lane ends with one value's total, each
    // value in 32 / N lanes
    constexpr int N = NQ * R <= 1 ? 1 : NQ * R <= 2 ? 2 : NQ * R <= 4 ? 4 : NQ * R <= 8 ? 8 : 16;
    T v[N];
#pragma unroll
    for (int u = 0; u < N; ++u) v[u] = u < NQ * R ? q[u / R][u % R] : T(0);
    T mine;
    int which;
    bool owner;
    ph::warp_sum_halving<T, N>(v, k.lane, mine, which, owner);
    const int i = which / R, r = which % R;
    const int chunk = k.warp + r * k.warps;
    if (i >= NQ || chunk * 32 >= rows) return;
    // the lanes that hold a value differ in the low bits: one block each, or several
#pragma unroll 1
    for (int rank = k.lane & (32 / N - 1); rank < cluster; rank += 32 / N)
        scatter(part, static_cast<std::uint32_t>(rank), static_cast<std::uint32_t>(i) * stride + chunk0 + static_cast<std::uint32_t>(chunk), mine);
}

template <typename T>
__device__ __forceinline__ int planet_of(const OnchipArgs<T>& a) {
    const unsigned i = blockIdx.x / static_cast<unsigned>(a.cluster);
    return static_cast<int>(a.list != nullptr ? a.list[i] : i);
}

// ---- the whole solve ------------------------------------------------------------------------------

// Rows of the fine level a thread keeps in registers: matrix, addresses, aggregate.
template <typename T, int R>
constexpr bool kHeld = sizeof(T) * R <= 16;

template <typename T, int R>
struct Solve {
    const OnchipArgs<T>& a;
    const Block& k;
    Reduce& red;
    const Phase* list;
    int rows;               // own fine rows
    std::uint32_t chunk0;   // the block's first 32-row chunk
    std::uint32_t stride;   // partials of one quantity: whole tiles of eight chunks
    std::uint32_t slot;     // reductions so far: partial slots alternate
    Rows<R> my;
    static constexpr int kIn = kHeld<T, R> ? R : 1;
    MatrixRow<T, 6> held[kIn];
    std::uint32_t at[kIn][7];

    __device__ std::uint32_t part() const { return (slot & 1u) != 0 ? a.o_part2 : a.o_part; }
    template <typename A, int NQ>
    __device__ __forceinline__ void reduce(const A (&q)[NQ][R], int kind) {
        write_partials<A, NQ, R>(k, k.base + part(), stride, chunk0, a.cluster, q, rows);
        finish<A>(k, &red, part(), kind, NQ == 2);
        ++slot;
    }

    __device__ __forceinline__ void load(std::uint32_t row0, std::uint32_t next0) {
        if constexpr (kHeld<T, R>) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const FineRow<T> f = fetch_fine(a.level[0], a.level[1],
                                                my.on[r] ? row0 + k.rank * a.level[0].span + my.row[r] : row0, row0, next0);
                held[r] = f.m;
#pragma unroll
                for (int j = 0; j < 7; ++j) at[r][j] = entry_of<T>(k.base, f.code[j]);
            }
        } else {
            load_fine(k, a.level[0], a.level[1], row0, next0);
        }
    }
    __device__ __forceinline__ MatrixRow<T, 6> fine_row(int r) const {
        if constexpr (kHeld<T, R>) return held[r];
        else return matrix_row<6>(k.at<float4>(a.level[0].o_m), a.level[0].span, my.row[r], T(0));
    }
    // addresses of the neighbours (and, last, of the aggregate) of this thread's row r
    __device__ __forceinline__ void addresses(int r, std::uint32_t (&to)[7]) const {
        if constexpr (kHeld<T, R>) {
#pragma unroll
            for (int j = 0; j < 7; ++j) to[j] = at[r][j];
        } else {
            const uint4 c = k.at<uint4>(a.level[0].o_col)[my.row[r]];
#pragma unroll
            for (int j = 0; j < 7; ++j) to[j] = entry_of<T>(k.base, place(c, j));
        }
    }

    // f(r, matrix row, its neighbours' entries of the vector at o_x) for this thread's rows, up to
    // kTogether of them with their gathers in flight at once.
    template <typename F>
    __device__ __forceinline__ void stencil(std::uint32_t o_x, F&& f) const {
        constexpr int kTogether = sizeof(T) == 4 ? (R < 3 ? R : 3) : (R < 2 ? R : 2);
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += kTogether) {
            T g[kTogether][6];
#pragma unroll
            for (int u = 0; u < kTogether; ++u) {
                if (r0 + u >= R) break;
                std::uint32_t to[7], first[6];
                addresses(r0 + u, to);
#pragma unroll
                for (int j = 0; j < 6; ++j) first[j] = to[j];
                gather(o_x, first, g[u]);
            }
#pragma unroll
            for (int u = 0; u < kTogether; ++u) {
                if (r0 + u >= R) break;
                f(r0 + u, fine_row(r0 + u), g[u]);
            }
        }
    }

    // M b from the zero-start iterate already written (and the barrier after it passed); b in
    // registers, the result at o_x.
    __device__ __forceinline__ void vcycle(const T (&b)[R], std::uint32_t o_x) {
        const T omega = a.omega;
        const int phases = red.phases;
        Ahead<T> ahead;
        Phase p = list[0];
        std::uint32_t kind = p.kind;
        if ((kind & kFinePhase) == 0) load_ahead(k, p, kind, k.tid, ahead);
#pragma unroll 1
        for (int i = 0;;) {
            if ((kind & kFinePhase) == 0) {
                coarse_phase(k, p, kind, ahead, a.cluster, omega);
            } else {
                const std::uint32_t src = p.src == kHat ? o_x : p.src, dst = p.dst == kHat ? o_x : p.dst;
                if (kind == (kFinePhase | kProlong)) {
                    T e[R];
                    std::uint32_t from[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        std::uint32_t to[7];
                        addresses(r, to);
                        from[r] = to[6];
                    }
                    gather(src, from, e);
                    const T c = a.level[0].correction;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if (my.on[r]) k.at<T>(dst)[my.row[r]] = add_(k.at<T>(dst)[my.row[r]], prod(c, e[r]));
                    }
                } else {
                    const bool residual = kind == (kFinePhase | kResidual);
                    stencil(src, [&](int r, const MatrixRow<T, 6>& m, const T (&g)[6]) {
                        const T xo = k.at<T>(src)[my.row[r]];
                        T s = residual ? fnma(m.diagonal(), xo, b[r]) : b[r];
#pragma unroll
                        for (int j = 0; j < 6; ++j) s = fnma(m.v[j], g[j], s);
                        if (!residual) s = ph::sweep_update(xo, omega, m.inverse(), s);
                        if (my.on[r]) k.at<T>(dst)[my.row[r]] = s;
                    });
                }
            }
            cluster_arrive();
            if (++i < phases) {
                p = list[i];
                kind = p.kind;
                if ((kind & kFinePhase) == 0) load_ahead(k, p, kind, k.tid, ahead);
            }
            cluster_wait();
            if (i >= phases) break;
        }
    }

    // y = A x at this thread's rows (0 where off).
    __device__ __forceinline__ void product(std::uint32_t o_x, T (&y)[R]) const {
        stencil(o_x, [&](int r, const MatrixRow<T, 6>& m, const T (&g)[6]) {
            // the first two products: the compiler fuses the diagonal's into the sum in phases.cuh
            T s = fma_(m.diagonal(), k.at<T>(o_x)[my.row[r]], prod(m.v[0], g[0]));
#pragma unroll
            for (int j = 1; j < 6; ++j) s = fma_(m.v[j], g[j], s);
            y[r] = my.on[r] ? s : T(0);
        });
    }

    // BiCGSTAB on the residual in `b` from zero; the solution's rows in `x`.
    __device__ __forceinline__ void bicgstab(const T (&b)[R], T (&x)[R]) {
        const OnchipLevel<T>& L = a.level[0];
        T rr[R], shadow[R], p[R], v[R], q1[1][R], q2[2][R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            rr[r] = shadow[r] = b[r];
            x[r] = p[r] = v[r] = T(0);
            q1[0][r] = prod(b[r], b[r]);
        }
        reduce(q1, ph::kFinBicgInit);
        bool open = red.s.status == kRunning;
        // the two halves of an iteration share one copy of the V-cycle: M p, then M s
#pragma unroll 1
        for (int half = 0; open; half ^= 1) {
            const std::uint32_t o_hat = half == 0 ? a.o_phat : a.o_shat;
            const std::uint32_t first = L.starts_in_x ? o_hat : L.o_y;
            T m[R];
            if (half == 0) {
                const T beta = ph::beta_of<T>(red.s), om = ph::omega_of<T>(red.s);
#pragma unroll
                for (int r = 0; r < R; ++r) m[r] = p[r] = fma_(beta, fnma(om, v[r], p[r]), rr[r]);
            } else {
                const T alpha = ph::alpha_of<T>(red.s);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    m[r] = rr[r] = fnma(alpha, v[r], rr[r]);   // s
                    q1[0][r] = prod(rr[r], rr[r]);
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const T z = prod(prod(a.omega, fine_row(r).inverse()), m[r]);
                if (my.on[r]) k.at<T>(first)[my.row[r]] = z;
            }
            if (half == 0) {
                cluster_barrier();
            } else {
                reduce(q1, ph::kFinBicgS);
                if (red.s.status != kRunning) break;
                if (red.s.half_done) {
                    // converged at s: x += alpha p_hat closes the iteration
                    const T alpha = ph::alpha_of<T>(red.s);
#pragma unroll
                    for (int r = 0; r < R; ++r) x[r] = fma_(alpha, k.at<T>(a.o_phat)[my.row[r]], x[r]);
                    __syncthreads();
                    if (k.tid == 0) {
                        const double none[2] = {0.0, 0.0};
                        ph::finish_bicg_x(red.s, none);
                    }
                    __syncthreads();
                    break;
                }
            }
            vcycle(m, o_hat);
            product(o_hat, m);
            if (half == 0) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    v[r] = m[r];
                    q1[0][r] = prod(shadow[r], v[r]);
                }
                reduce(q1, ph::kFinBicgV);
                open = red.s.status == kRunning;
                continue;
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                q2[0][r] = prod(m[r], m[r]);
                q2[1][r] = prod(m[r], rr[r]);
            }
            reduce(q2, ph::kFinBicgT);
            if (red.s.status != kRunning) break;
            const T alpha = ph::alpha_of<T>(red.s), w = ph::omega_of<T>(red.s);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                x[r] = add_(x[r], fma_(alpha, k.at<T>(a.o_phat)[my.row[r]], prod(w, k.at<T>(a.o_shat)[my.row[r]])));
                rr[r] = fnma(w, m[r], rr[r]);
                q2[0][r] = my.on[r] ? prod(rr[r], rr[r]) : T(0);
                q2[1][r] = prod(shadow[r], rr[r]);
            }
            reduce(q2, ph::kFinBicgX);
            open = red.s.status == kRunning;
        }
    }
};

// At most kOnchipThreads threads a block. Few threads with several rows each: the cluster
// barrier is cheaper (0.19 us with 256 threads, 0.29 with 1024), and a thread has 168 registers
// for the solve, its rows' matrix and addresses with it, where 1024 threads have 64 and spill
// most of it to an L1 that the shared memory leaves no room in. FP32 with one or two rows a thread
// stays in registers whole; the others spill a little (bytes of stores and loads a thread: FP32
// four rows 168 and 188, seven 12 and 24; FP64 one row 44 and 64, two 388 and 420, four 172 and
// 216).
template <typename T, int R>
__global__ void __launch_bounds__(kOnchipThreads, 1) k_onchip_solve(const __grid_constant__ OnchipArgs<T> a) {
    extern __shared__ __align__(16) unsigned char onchip_smem[];
    __shared__ Reduce red;
    const Block k = block_of(onchip_smem);
    Phase* const list = k.at<Phase>(a.o_list);
    const int inst = planet_of(a);
    if (a.active != nullptr && a.active[inst] == 0) {   // the whole cluster
        if (k.rank == 0 && k.tid == 0) {
            InstanceScalars& s = a.sc[inst];
            s.outer_status = kConverged;
            s.status = kConverged;
            s.refinements = 0;
            s.inner_total = 0;
            s.outer_r_norm = 0.0;
            s.outer_b_norm = 0.0;
        }
        return;
    }
    const auto first_row = [&](int l) { return a.tile_range[(l * a.instances + inst) * 2] * static_cast<std::uint32_t>(kTile); };
    const OnchipLevel<T>& L = a.level[0];
    Solve<T, R> sv{a, k, red, list, own_rows(L.n, L.span, k.rank), k.rank * (L.span / 32u), (L.n + 255u) / 256u * 8u, 0u};
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int row = (k.warp + r * k.warps) * 32 + k.lane;
        sv.my.on[r] = row < sv.rows;
        sv.my.row[r] = sv.my.on[r] ? row : 0;
    }
    const std::uint32_t row0 = first_row(0);
    const std::size_t g0 = row0 + std::size_t(k.rank) * L.span;
    // ||b|| first: its loads overlap the hierarchy's
    double d[1][R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const double bv = sv.my.on[r] ? a.rhs64[g0 + sv.my.row[r]] : 0.0;
        d[0][r] = __dmul_rn(bv, bv);
    }
    if (k.tid == 0) {
        red.s = a.sc[inst];
        red.tolerance = a.tolerance;
        red.inner_tolerance = a.inner_tolerance;
        red.max_iterations = a.max_iterations;
        red.max_refinements = a.max_refinements;
        red.n = L.n;
        red.phases = build_cycle(k, a, list);
    }
    sv.load(row0, first_row(1));
    load_members(k, a.level[0], a.level[1], row0, first_row(1));
#pragma unroll 1
    for (int l = 1; l < a.coarsest; ++l) {
        load_coarse(k, a.level[l], a.level[l + 1], first_row(l), first_row(l + 1));
        load_members(k, a.level[l], a.level[l + 1], first_row(l), first_row(l + 1));
    }
    load_dense(k, a, inst);
    cluster_barrier();   // every block of the cluster has started before the first remote store
    sv.reduce(d, ph::kFinOuterInit);
    const std::size_t P = L.pitch;
#pragma unroll 1
    for (int round = 0; round <= a.max_refinements; ++round) {
        // r = b - A x in FP64 (FP64 matrix, x through L2: the cluster's blocks write its rows)
        T b[R];
        constexpr int kTogether = R < 2 ? R : 2;
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += kTogether) {
            int col[kTogether][6];
            double g[kTogether][6], v[kTogether][7], own[kTogether], rhs[kTogether];
#pragma unroll
            for (int u = 0; u < kTogether; ++u) {
                if (r0 + u >= R) break;
                const std::size_t at = sv.my.on[r0 + u] ? g0 + sv.my.row[r0 + u] : row0;   // off: a row that is there
#pragma unroll
                for (int j = 0; j < 6; ++j) col[u][j] = a.fine_col[j * P + at];
#pragma unroll
                for (int j = 0; j < 7; ++j) v[u][j] = a.fine_vd64[j * P + at];
                own[u] = __ldcg(&a.x64[at]);
                rhs[u] = a.rhs64[at];
            }
#pragma unroll
            for (int u = 0; u < kTogether; ++u) {
                if (r0 + u >= R) break;
#pragma unroll
                for (int j = 0; j < 6; ++j) g[u][j] = __ldcg(&a.x64[col[u][j]]);
            }
#pragma unroll
            for (int u = 0; u < kTogether; ++u) {
                if (r0 + u >= R) break;
                double s = fnma(v[u][6], own[u], rhs[u]);
#pragma unroll
                for (int j = 0; j < 6; ++j) s = fnma(v[u][j], g[u][j], s);
                b[r0 + u] = sv.my.on[r0 + u] ? static_cast<T>(s) : T(0);
                d[0][r0 + u] = sv.my.on[r0 + u] ? prod(s, s) : 0.0;
            }
        }
        sv.reduce(d, ph::kFinOuterResidual);
        if (red.s.outer_status != kRunning) break;
        T x[R];
        sv.bicgstab(b, x);
        __syncthreads();
        if (k.tid == 0) ph::outer_account(red.s);
        __syncthreads();
        if (red.s.outer_status == kRunning) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (sv.my.on[r]) a.x64[g0 + sv.my.row[r]] = __ldcg(&a.x64[g0 + sv.my.row[r]]) + static_cast<double>(x[r]);
            }
        }
        cluster_barrier();
    }
    if (k.rank == 0 && k.tid == 0) a.sc[inst] = red.s;
    cluster_barrier();   // no block leaves while another may still read its shared memory
}

// ---- host side of one precision -------------------------------------------------------------------

template <typename T>
using KernelOf = void (*)(OnchipArgs<T>);

template <typename T>
KernelOf<T> kernel_of(int rows_per_thread) {
    switch (rows_per_thread) {
        case 1: return k_onchip_solve<T, 1>;
        case 2: return k_onchip_solve<T, 2>;
        case 4: return k_onchip_solve<T, 4>;
        case 7:
            if constexpr (sizeof(T) == 4) return k_onchip_solve<T, 7>;
            return nullptr;
        default: return nullptr;
    }
}

// Dynamic shared memory a block of the kernel may take, with the kernel's attributes set
// (0: the current device cannot launch it).
template <typename T>
unsigned shared_limit(int rows_per_thread) {
    static PerDevice<std::array<unsigned, 8>> limits;
    return limits.of(current_device(), [] {
        std::array<unsigned, 8> out{};
        int device = 0, optin = 0, cluster = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&cluster, cudaDevAttrClusterLaunch, device) != cudaSuccess || cluster == 0 ||
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) {
            cudaGetLastError();
            return out;
        }
        for (int r = 0; r < 8; ++r) {
            if (kernel_of<T>(r) == nullptr) continue;
            cudaFuncAttributes fa{};
            const void* f = reinterpret_cast<const void*>(kernel_of<T>(r));
            if (cudaFuncGetAttributes(&fa, f) != cudaSuccess) { cudaGetLastError(); continue; }
            const long room = static_cast<long>(optin) - static_cast<long>(fa.sharedSizeBytes);
            if (room <= 0 ||
                cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(room)) != cudaSuccess ||
                cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            out[r] = static_cast<unsigned>(room);
        }
        return out;
    })[static_cast<std::size_t>(rows_per_thread)];
}

struct Config {
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg{};
    Config(unsigned cluster, unsigned blocks, unsigned threads, std::size_t bytes, cudaStream_t st) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cluster;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = bytes;
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
};

}  // namespace oc

template <typename T>
bool onchip_has(int rows_per_thread) {
    return oc::kernel_of<T>(rows_per_thread) != nullptr;
}

template <typename T>
int onchip_active_clusters(int rows_per_thread, unsigned cluster, unsigned threads, std::size_t shared_bytes) {
    if (shared_bytes > oc::shared_limit<T>(rows_per_thread)) return 0;
    oc::Config c(cluster, cluster, threads, shared_bytes, nullptr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, oc::kernel_of<T>(rows_per_thread), &c.cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return clusters;
}

template <typename T>
void onchip_launch(const OnchipArgs<T>& args, int rows_per_thread, unsigned threads, std::size_t shared_bytes,
                   cudaStream_t st) {
    if (shared_bytes > oc::shared_limit<T>(rows_per_thread)) throw std::logic_error("on-chip solve: the planet does not fit");
    const unsigned cluster = static_cast<unsigned>(args.cluster);
    oc::Config c(cluster, args.planets * cluster, threads, shared_bytes, st);
    PSGB_LAUNCH(kFamOnchip, st, {
        const cudaError_t e = cudaLaunchKernelEx(&c.cfg, oc::kernel_of<T>(rows_per_thread), args);
        if (e != cudaSuccess) throw std::runtime_error(std::string("on-chip solve launch: ") + cudaGetErrorString(e));
    });
}

}  // namespace psgb
