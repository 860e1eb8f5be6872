// The non-symmetric transport solves on a planet's transport graph, on the GPU:
//
//  - block ILU(0) (sim/core/math/incomplete_lu.cpp): factorisation and triangular solves
//    level-scheduled inside each block (one CTA per block, the rows of a dependency
//    level in parallel), the same operations in the same order as the reference's, so
//    the factor and its solves are bit-identical;
//  - right-preconditioned BiCGSTAB as the reference's (heat_transport.cpp:823-897), x0 = 0,
//    shadow = r0, its breakdown tests; dots are fixed-order device reductions;
//  - advection_diffusion_source (heat_transport.cpp:774-815), bit-identical;
//  - solve_implicit_tracer (heat_transport.cpp:901-1081): the stacked layers' implicit
//    upwind/eddy/vertical system, BiCGSTAB with the stacked block ILU(0), the flux form
//    of the solution accumulated per row in the reference's order;
//  - solve_implicit_advection_diffusion (heat_transport.cpp:1083-1318): Newton on h with
//    the Jacobian on the graph's pattern, BiCGSTAB preconditioned by the V-cycle of the
//    eddies' symmetric part followed by the block ILU(0) of the full Jacobian on what is
//    left, and the line search of the implicit transport solve.
//
// Compiled without FMA contraction: every expression rounds as the reference's does.
#include "../../include/planetsim_gb300.h"
#include "capi_internal.hpp"
#include "common.cuh"
#include "host/ilu_pattern.hpp"
#include "host/per_device.hpp"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <functional>
#include <limits>
#include <map>
#include <memory>
#include <stdexcept>
#include <utility>
#include <vector>

namespace psgb {

namespace {

constexpr int kThreads = 256;
constexpr int kIluThreads = 128;

unsigned blocks_of(std::size_t n) { return static_cast<unsigned>((n + kThreads - 1) / kThreads); }

// std::max(a, b): b if a < b, else a (NaN in `a` kept, as the reference's).
__device__ __forceinline__ double std_max(double a, double b) { return a < b ? b : a; }

void require(bool ok, const char* what) {
    if (!ok) throw std::invalid_argument(what);
}

#define PSGB_CHECK_LAUNCH() PSGB_CUDA(cudaGetLastError())

// ---- block ILU(0) -------------------------------------------------------------------

struct IluView {
    const std::uint32_t *start, *column, *diagonal, *update_start, *update_t, *update_at;
    const std::int32_t* source;
    const std::uint32_t *lo_block, *lo_level, *lo_order, *up_block, *up_level, *up_order;
    double* value;
    int* flag;
    std::uint32_t rows;
};

// value = the matrix on the pattern: diagonal * scale, off-diagonals from their CSR entries.
__global__ void k_ilu_load(IluView v, const double* __restrict__ diag, const double* __restrict__ off, double scale) {
    const std::uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= v.rows) return;
    for (std::uint32_t q = v.start[i]; q < v.start[i + 1]; ++q) {
        const std::int32_t k = v.source[q];
        v.value[q] = k < 0 ? diag[i] * scale : off[k];
    }
}

// IKJ elimination restricted to the pattern (incomplete_lu.cpp:108-135), a level at a time.
__global__ void __launch_bounds__(kIluThreads) k_ilu_factor(IluView v) {
    const std::uint32_t b = blockIdx.x;
    for (std::uint32_t lv = v.lo_block[b]; lv < v.lo_block[b + 1]; ++lv) {
        for (std::uint32_t idx = v.lo_level[lv] + threadIdx.x; idx < v.lo_level[lv + 1]; idx += kIluThreads) {
            const std::uint32_t i = v.lo_order[idx];
            for (std::uint32_t q = v.start[i]; q < v.diagonal[i]; ++q) {
                const double pivot = v.value[v.diagonal[v.column[q]]];
                if (pivot == 0.0) atomicExch(v.flag, 1);   // the reference throws here
                const double lq = v.value[q] / pivot;
                v.value[q] = lq;
                for (std::uint32_t u = v.update_start[q]; u < v.update_start[q + 1]; ++u)
                    v.value[v.update_at[u]] -= lq * v.value[v.update_t[u]];
            }
        }
        __syncthreads();
    }
}

// x <- (LU)^-1 x (incomplete_lu.cpp:137-152): forward, then backward, level by level.
__global__ void __launch_bounds__(kIluThreads) k_ilu_solve(IluView v, double* __restrict__ x, const int* skip) {
    if (skip != nullptr && *skip != 0) return;
    const std::uint32_t b = blockIdx.x;
    for (std::uint32_t lv = v.lo_block[b]; lv < v.lo_block[b + 1]; ++lv) {
        for (std::uint32_t idx = v.lo_level[lv] + threadIdx.x; idx < v.lo_level[lv + 1]; idx += kIluThreads) {
            const std::uint32_t i = v.lo_order[idx];
            double sum = x[i];
            for (std::uint32_t q = v.start[i]; q < v.diagonal[i]; ++q) sum -= v.value[q] * x[v.column[q]];
            x[i] = sum;
        }
        __syncthreads();
    }
    for (std::uint32_t lv = v.up_block[b]; lv < v.up_block[b + 1]; ++lv) {
        for (std::uint32_t idx = v.up_level[lv] + threadIdx.x; idx < v.up_level[lv + 1]; idx += kIluThreads) {
            const std::uint32_t i = v.up_order[idx];
            double sum = x[i];
            for (std::uint32_t q = v.diagonal[i] + 1; q < v.start[i + 1]; ++q) sum -= v.value[q] * x[v.column[q]];
            x[i] = sum / v.value[v.diagonal[i]];
        }
        __syncthreads();
    }
}

// The triangular solves with the block's x in shared memory and per-level records (the
// row, its couplings' block-local columns and their factor values packed next to them):
// a thread owns one row of a level and loads the next level's record before the current
// level computes. Same terms in the same order as k_ilu_solve: same bits.
//
//
// A level is a few dozen to a few hundred rows of up to eight products and differences each, and
// on the way back a division. An SM starts an FP64 instruction of a warp every 19 cycles, the
// same warp's next one after 66, and one lane costs what 32 do: the levels are bound by these
// instructions. So a warp's rows have the same number of couplings and the terms that none of them
// has are not issued (as selections, every row paid for eight); the division by the diagonal takes
// its stored reciprocal; and a level's records are
// loaded, one value a plane, while the level before computes. A pair of SMs a block, half of each level's rows on either, was slower: its barrier and
// the store to the partner take 400 to 900 cycles a level, as much as the halves save.
// Ten layers on 10,242 nodes, 41 blocks of 2,560 rows in 23 levels each way: 51 us a
// solve, 86 before.
struct IluRecords {
    const std::uint32_t* head;     // the row and, from bit 16, its couplings
    const uint4* cols;             // eight 16-bit columns
    double* val;                   // [8][rows]: packed after each factorisation
    double2* diag;                 // upper: the diagonal and its reciprocal (0: divide)
    const std::uint32_t* q;        // [rows][8]: value positions
    const std::uint32_t* dq;       // upper: the row's diagonal position
    const std::uint32_t* block;    // [blocks + 1] levels
    const std::uint32_t* level;    // [levels + 1]
};

struct IluShared {
    IluRecords lo, up;
    const std::uint32_t* block_start;   // [blocks + 1] rows
    std::uint32_t rows;
};

__global__ void k_ilu_pack(std::uint32_t rows, IluShared s, const double* __restrict__ value) {
    const std::uint32_t idx = blockIdx.x * kThreads + threadIdx.x;
    if (idx >= rows) return;
#pragma unroll
    for (std::uint32_t k = 0; k < 8; ++k) {
        s.lo.val[k * rows + idx] = k < s.lo.head[idx] >> 16 ? value[s.lo.q[idx * 8 + k]] : 0.0;
        s.up.val[k * rows + idx] = k < s.up.head[idx] >> 16 ? value[s.up.q[idx * 8 + k]] : 0.0;
    }
    const double d = value[s.up.dq[idx]];
    s.up.diag[idx] = make_double2(d, reciprocal_of(d));
}

// A row's record as it is loaded; nothing here is looked at before its level.
struct Rec {
    std::uint32_t head;
    uint4 cols;
    double val[8];
    double2 diag;
};

// The row's differences, for a warp whose rows have at most N couplings; a lane with fewer takes
// off +0, which changes nothing.
template <int N>
__device__ __forceinline__ double subtract_terms(const Rec& c, const double* xs, double sum) {
    const std::uint32_t count = c.head >> 16;
    double p[N];
#pragma unroll
    for (std::uint32_t k = 0; k < N; ++k) {
        const std::uint32_t w = k < 2 ? c.cols.x : k < 4 ? c.cols.y : k < 6 ? c.cols.z : c.cols.w;
        p[k] = k < count ? xs[k & 1 ? w >> 16 : w & 0xffffu] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < N; ++k) p[k] = c.val[k] * p[k];
#pragma unroll
    for (int k = 0; k < N; ++k) sum -= p[k];
    return sum;
}

constexpr unsigned kIluSharedThreads = 512;   // the widest level the shared-memory solve takes

// out <- (LU)^-1 in, the same vector or another; a thread block a block of the matrix, a thread a
// row of each level. `skip`: a device word that, where set, makes the solve needless (null: always
// run). `deepest`: most levels of one triangle.
__global__ void __launch_bounds__(kIluSharedThreads, 1) k_ilu_solve_shared(IluShared s, const double* in, double* out,
                                                                          const int* skip, std::uint32_t deepest) {
    if (skip != nullptr && *skip != 0) return;
    extern __shared__ double ilu_smem[];
    double* xs = ilu_smem;
    const std::uint32_t b = blockIdx.x;
    const std::uint32_t first = s.block_start[b], n = s.block_start[b + 1] - first;
    std::uint32_t* starts = reinterpret_cast<std::uint32_t*>(xs + n);   // level starts of both triangles
    const std::uint32_t lo0 = s.lo.block[b], lo_levels = s.lo.block[b + 1] - lo0;
    const std::uint32_t up0 = s.up.block[b], levels = lo_levels + s.up.block[b + 1] - up0;
    for (std::uint32_t l = threadIdx.x; l <= lo_levels; l += blockDim.x) starts[l] = s.lo.level[lo0 + l];
    for (std::uint32_t l = threadIdx.x; l <= levels - lo_levels; l += blockDim.x) starts[deepest + 1 + l] = s.up.level[up0 + l];
    for (std::uint32_t r = threadIdx.x; r < n; r += blockDim.x) xs[r] = in[first + r];
    __syncthreads();
    // levels 0 .. lo_levels there, the others back
    const auto level = [&](std::uint32_t lv) {
        return starts + (lv < lo_levels ? lv : deepest + 1 + lv - lo_levels);
    };
    const auto load = [&](std::uint32_t lv) {
        const bool upper = lv >= lo_levels;
        const IluRecords& R = upper ? s.up : s.lo;
        const std::uint32_t* st = level(lv);
        const std::uint32_t idx = lv < levels ? st[0] + threadIdx.x : 0u;
        Rec c{0xffffu, make_uint4(0u, 0u, 0u, 0u), {}, make_double2(1.0, 0.0)};
        if (lv < levels && idx < st[1]) {
            c.head = R.head[idx];
            c.cols = R.cols[idx];
#pragma unroll
            for (std::uint32_t k = 0; k < 8; ++k) c.val[k] = R.val[std::size_t(k) * s.rows + idx];
            if (upper) c.diag = R.diag[idx];
        }
        return c;
    };
    Rec c = load(0);
    for (std::uint32_t lv = 0; lv < levels; ++lv) {
        const Rec next = load(lv + 1);
        const std::uint32_t row = c.head & 0xffffu;
        const bool on = row != 0xffffu;   // at most 4096 rows
        double sum = on ? xs[row] : 0.0;
        switch (__shfl_sync(0xffffffffu, c.head >> 16, 0)) {   // the most of the warp: a level's rows are in falling order
            case 0: break;
            case 1: sum = subtract_terms<1>(c, xs, sum); break;
            case 2: sum = subtract_terms<2>(c, xs, sum); break;
            case 3: sum = subtract_terms<3>(c, xs, sum); break;
            case 4: sum = subtract_terms<4>(c, xs, sum); break;
            case 5: sum = subtract_terms<5>(c, xs, sum); break;
            case 6: sum = subtract_terms<6>(c, xs, sum); break;
            case 7: sum = subtract_terms<7>(c, xs, sum); break;
            default: sum = subtract_terms<8>(c, xs, sum); break;
        }
        if (on) {
            if (lv >= lo_levels) sum = divide_by(sum, c.diag.x, c.diag.y);
            xs[row] = sum;
        }
        __syncthreads();
        c = next;
    }
    for (std::uint32_t r = threadIdx.x; r < n; r += blockDim.x) out[first + r] = xs[r];
}

// Its shared memory: the block's vector and both triangles' level starts.
constexpr std::size_t ilu_shared_bytes(std::uint32_t rows, std::uint32_t deepest) {
    return std::size_t(rows) * sizeof(double) + 2 * (std::size_t(deepest) + 1) * sizeof(std::uint32_t);
}

// Whether the device gives k_ilu_solve_shared the most that any factor needs: kIluSharedRows rows,
// a level each (64 KB). Asked for once a device, and never less: the limit belongs to the kernel,
// not to a factor.
bool ilu_shared_opted_in() {
    static PerDevice<bool> ready;
    return ready.of(current_device(), [] {
        const bool ok = cudaFuncSetAttribute(k_ilu_solve_shared, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(ilu_shared_bytes(kIluSharedRows, kIluSharedRows))) == cudaSuccess;
        if (!ok) cudaGetLastError();
        return ok;
    });
}

}  // namespace

// A block ILU(0) structure on the device, its values refactored per matrix.
class DeviceIlu {
  public:
    explicit DeviceIlu(const IluPattern& p) : rows_(p.rows), blocks_(p.blocks) {
        v_.start = store_.upload(p.start);
        v_.column = store_.upload(p.column);
        v_.diagonal = store_.upload(p.diagonal);
        v_.update_start = store_.upload(p.update_start);
        v_.update_t = store_.upload(p.update_t);
        v_.update_at = store_.upload(p.update_at);
        v_.source = store_.upload(p.source);
        v_.lo_block = store_.upload(p.lower.block_level);
        v_.lo_level = store_.upload(p.lower.level_start);
        v_.lo_order = store_.upload(p.lower.order);
        v_.up_block = store_.upload(p.upper.block_level);
        v_.up_level = store_.upload(p.upper.level_start);
        v_.up_order = store_.upload(p.upper.order);
        v_.value = store_.alloc<double>(p.column.size());
        v_.flag = store_.alloc<int>(1);
        v_.rows = p.rows;
        // the shared-memory solve, when the pattern has its records and a level fits a block
        const std::uint32_t widest = std::max(p.lower.widest, p.upper.widest);
        if (!p.lower.rec_row.empty() && widest <= kIluSharedThreads) {
            auto records = [&](const LevelSchedule& sch, bool upper) {
                IluRecords r{};
                std::vector<std::uint32_t> head(p.rows);
                for (std::uint32_t idx = 0; idx < p.rows; ++idx)
                    head[idx] = sch.rec_row[idx] | static_cast<std::uint32_t>(sch.rec_count[idx]) << 16;
                r.head = store_.upload(head);
                r.cols = reinterpret_cast<const uint4*>(store_.upload(sch.rec_col));
                r.val = store_.alloc<double>(sch.rec_q.size());
                r.q = store_.upload(sch.rec_q);
                r.block = upper ? v_.up_block : v_.lo_block;
                r.level = upper ? v_.up_level : v_.lo_level;
                if (upper) {
                    std::vector<std::uint32_t> dq(p.rows);
                    for (std::uint32_t idx = 0; idx < p.rows; ++idx) dq[idx] = p.diagonal[sch.order[idx]];
                    r.dq = store_.upload(dq);
                    r.diag = store_.alloc<double2>(p.rows);
                }
                return r;
            };
            shared_.lo = records(p.lower, false);
            shared_.up = records(p.upper, true);
            std::uint32_t most = 0;
            std::vector<std::uint32_t> starts(p.blocks + 1, 0);
            for (std::uint32_t b = 0; b < p.blocks; ++b) {
                // block b's rows: the lower schedule lists them level by level
                const std::uint32_t lv0 = p.lower.block_level[b], lv1 = p.lower.block_level[b + 1];
                const std::uint32_t count = lv1 > lv0 ? p.lower.level_start[lv1] - p.lower.level_start[lv0] : 0;
                starts[b + 1] = starts[b] + count;
                most = std::max(most, count);
            }
            shared_.block_start = store_.upload(starts);
            deepest_ = std::max(p.lower.deepest, p.upper.deepest);
            shared_threads_ = std::max(1u, (widest + 31) / 32) * 32;
            shared_.rows = p.rows;
            shared_bytes_ = ilu_shared_bytes(most, deepest_);
            use_shared_ = shared_bytes_ <= 48 * 1024 || ilu_shared_opted_in();
        }
    }

    // Factors diag * scale + off (CSR entries as the pattern's source); throws Breakdown
    // on a zero pivot, where the reference throws std::runtime_error.
    void factor(const double* diag, const double* off, double scale, cudaStream_t st) {
        PSGB_CUDA(cudaMemsetAsync(v_.flag, 0, sizeof(int), st));
        k_ilu_load<<<blocks_of(rows_), kThreads, 0, st>>>(v_, diag, off, scale);
        PSGB_CHECK_LAUNCH();
        k_ilu_factor<<<blocks_, kIluThreads, 0, st>>>(v_);
        PSGB_CHECK_LAUNCH();
        if (use_shared_) {
            k_ilu_pack<<<blocks_of(rows_), kThreads, 0, st>>>(rows_, shared_, v_.value);
            PSGB_CHECK_LAUNCH();
        }
        int flag = 0;
        PSGB_CUDA(cudaMemcpyAsync(&flag, v_.flag, sizeof(int), cudaMemcpyDeviceToHost, st));
        PSGB_CUDA(cudaStreamSynchronize(st));
        if (flag != 0) throw Breakdown("incomplete LU: zero pivot");
    }

    // out <- (LU)^-1 in (the same vector, or another). `skip`: a device word; the solve is left
    // out where it is set.
    void solve(const double* in, double* out, cudaStream_t st, const int* skip = nullptr) const {
        if (use_shared_) {
            k_ilu_solve_shared<<<blocks_, shared_threads_, shared_bytes_, st>>>(shared_, in, out, skip, deepest_);
        } else {
            if (in != out) PSGB_CUDA(cudaMemcpyAsync(out, in, std::size_t(rows_) * 8, cudaMemcpyDeviceToDevice, st));
            k_ilu_solve<<<blocks_, kIluThreads, 0, st>>>(v_, out, skip);
        }
        PSGB_CHECK_LAUNCH();
    }

    std::uint32_t rows() const { return rows_; }
    std::size_t device_bytes() const { return store_.bytes(); }

  private:
    DeviceStore store_;
    IluView v_{};
    std::uint32_t rows_, blocks_;
    IluShared shared_{};
    bool use_shared_ = false;
    std::uint32_t deepest_ = 0;
    unsigned shared_threads_ = 0;
    std::size_t shared_bytes_ = 0;
};

namespace {

// ---- reductions and BiCGSTAB -------------------------------------------------------

// Fixed-order block sum (256 threads): a butterfly in each warp, then one over the eight
// warp sums; the same bits on every run.
__device__ double tree_sum(double v, double* sh) {
    const int t = threadIdx.x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((t & 31) == 0) sh[t >> 5] = v;
    __syncthreads();
    double r = (t & 31) < kThreads / 32 ? sh[t & 31] : 0.0;
    if (t < 32) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if (t == 0) sh[32] = r;
    }
    __syncthreads();
    r = sh[32];
    __syncthreads();
    return r;
}
__device__ double tree_max(double v, double* sh) {
    const int t = threadIdx.x;
    sh[t] = v;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (t < s) sh[t] = fmax(sh[t], sh[t + s]);
        __syncthreads();
    }
    const double r = sh[0];
    __syncthreads();
    return r;
}

constexpr int kQ = 4;   // quantities per block partial

// One block: the partials of `quantities` values in fixed order; bit q of max_mask: a max.
__global__ void __launch_bounds__(kThreads) k_finish(unsigned blocks, int quantities, unsigned max_mask,
                                                     const double* __restrict__ partial, double* __restrict__ out) {
    __shared__ double sh[kThreads];
    for (int q = 0; q < quantities; ++q) {
        const bool is_max = (max_mask >> q) & 1u;
        double v = 0.0;
        for (unsigned b = threadIdx.x; b < blocks; b += kThreads) {
            const double x = partial[b * kQ + q];
            v = is_max ? fmax(v, x) : v + x;
        }
        const double r = is_max ? tree_max(v, sh) : tree_sum(v, sh);
        if (threadIdx.x == 0) out[q] = r;
    }
}

// BiCGSTAB's scalars on the device: each step of the iteration is decided where its sums are
// finished, by the last block of the kernel that forms them, so that the host only looks in from
// time to time and the GPU never waits for it. 102,420 rows: an iteration's vectors, products and
// sums 55 us beside its two solves; with kernels for the sums alone, read back and decided by the
// host, 130 us.
struct BicgState {
    int done;         // nothing runs any more
    int half;         // converged at s: x += alpha p_hat closes the solve
    int skip_second;  // done or half
    int iteration, max_iterations;
    unsigned arrived;   // blocks of the kernel under way
    double rho, alpha, omega, beta, b_norm, tolerance;
};

enum BicgSum : int { kSumStart, kSumV, kSumS, kSumT, kSumX };

__device__ void bicg_step(BicgState& s, int kind, double a, double b) {
    const auto next = [&](double rho_next) {   // the head of an iteration
        if (s.iteration >= s.max_iterations || rho_next == 0.0 || s.omega == 0.0) {
            s.done = 1;
        } else {
            s.beta = rho_next / s.rho * (s.alpha / s.omega);
            s.rho = rho_next;
        }
    };
    if (kind == kSumStart) {          // b . b (and shadow . r, the same sum)
        s.b_norm = sqrt(a);
        s.rho = s.alpha = s.omega = 1.0;
        if (!(s.b_norm > 0.0)) s.done = 1;
        else next(a);
    } else if (kind == kSumV) {       // shadow . v
        if (a == 0.0) s.done = 1;
        else s.alpha = s.rho / a;
    } else if (kind == kSumS) {       // s . s
        ++s.iteration;
        if (sqrt(a) <= s.tolerance * s.b_norm) s.half = 1;
    } else if (kind == kSumT) {       // t . t, t . s
        s.omega = a > 0.0 ? b / a : 0.0;
    } else if (s.half != 0 || sqrt(a) <= s.tolerance * s.b_norm) {   // r . r, shadow . r
        s.done = 1;
    } else {
        next(b);
    }
    s.skip_second = s.done | s.half;
}

// A block's sums of one or two quantities; the last block to arrive sums all blocks' in fixed order
// (k_finish's) and takes the step. Every block has read the state by then.
__device__ __forceinline__ void sum_and_step(int kind, double a, double b, double* sh, double* partial, BicgState* state) {
    __shared__ bool last;
    const bool two = kind == kSumT || kind == kSumX;
    const double s1 = tree_sum(a, sh);
    const double s2 = two ? tree_sum(b, sh) : 0.0;
    if (threadIdx.x == 0) {
        partial[blockIdx.x * kQ + 0] = s1;
        partial[blockIdx.x * kQ + 1] = s2;
        __threadfence();
        last = atomicAdd(&state->arrived, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double v[2] = {0.0, 0.0};
    for (unsigned k = threadIdx.x; k < gridDim.x; k += kThreads) {
        v[0] = v[0] + __ldcg(&partial[k * kQ]);
        if (two) v[1] = v[1] + __ldcg(&partial[k * kQ + 1]);
    }
    const double sum = tree_sum(v[0], sh);
    const double other = two ? tree_sum(v[1], sh) : 0.0;
    if (threadIdx.x == 0) {
        state->arrived = 0;
        bicg_step(*state, kind, sum, other);
    }
}

__global__ void __launch_bounds__(kThreads) k_bicg_start(std::uint32_t n, const double* __restrict__ b,
                                                         double* __restrict__ x, double* __restrict__ r,
                                                         double* __restrict__ shadow, double* __restrict__ p,
                                                         double* __restrict__ v, BicgState* state, double* partial) {
    __shared__ double sh[kThreads];
    const std::uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    const double bv = i < n ? b[i] : 0.0;
    if (i < n) {
        x[i] = 0.0;
        r[i] = bv;
        shadow[i] = bv;
        p[i] = 0.0;
        v[i] = 0.0;
    }
    sum_and_step(kSumStart, i < n ? bv * bv : 0.0, 0.0, sh, partial, state);
}
__global__ void k_bicg_p(std::uint32_t n, const double* __restrict__ r, double* __restrict__ p,
                         const double* __restrict__ v, const BicgState* state) {
    if (state->done != 0) return;
    const double beta = state->beta, omega = state->omega;
    const std::uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i < n) p[i] = r[i] + beta * (p[i] - omega * v[i]);
}
__global__ void __launch_bounds__(kThreads) k_bicg_s(std::uint32_t n, const double* __restrict__ r,
                                                     const double* __restrict__ v, double* __restrict__ s,
                                                     BicgState* state, double* partial) {
    __shared__ double sh[kThreads];
    if (state->done != 0) return;
    const double alpha = state->alpha;
    const std::uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    double sv = 0.0;
    if (i < n) {
        sv = r[i] - alpha * v[i];
        s[i] = sv;
    }
    sum_and_step(kSumS, i < n ? sv * sv : 0.0, 0.0, sh, partial, state);
}
__global__ void __launch_bounds__(kThreads) k_bicg_x(std::uint32_t n, double* __restrict__ x, double* __restrict__ r,
                                                     const double* __restrict__ p_hat, const double* __restrict__ s_hat,
                                                     const double* __restrict__ s, const double* __restrict__ t,
                                                     const double* __restrict__ shadow, BicgState* state,
                                                     double* partial) {
    __shared__ double sh[kThreads];
    if (state->done != 0) return;
    const double alpha = state->alpha, omega = state->omega;
    const std::uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    double rv = 0.0, dv = 0.0;
    if (state->half != 0) {
        if (i < n) x[i] += alpha * p_hat[i];
    } else if (i < n) {
        x[i] += alpha * p_hat[i] + omega * s_hat[i];
        rv = s[i] - omega * t[i];
        r[i] = rv;
        dv = shadow[i] * rv;
    }
    sum_and_step(kSumX, i < n ? rv * rv : 0.0, dv, sh, partial, state);
}

// y = diag x + off x (the reference's apply) on an ELL copy of the off-diagonals (slot-major,
// coalesced): slot j of row r is CSR entry offset[r] + j, so the terms add in the same
// order, the same bits.
struct Ell {
    std::uint32_t rows, width;
    const std::uint8_t* degree;     // [rows]
    const std::uint32_t* col;       // [width][rows]
};

__global__ void k_csr_to_ell(Ell e, const std::uint32_t* __restrict__ offset, const double* __restrict__ off,
                             double* __restrict__ val) {
    const std::uint32_t r = blockIdx.x * kThreads + threadIdx.x;
    if (r >= e.rows) return;
    const std::uint32_t first = offset[r], deg = e.degree[r];
    for (std::uint32_t j = 0; j < e.width; ++j) val[std::size_t(j) * e.rows + r] = j < deg ? off[first + j] : 0.0;
}

// A row's product, its loads in flight together where the row is at most eight wide.
__device__ __forceinline__ double ell_row(const Ell& e, const double* __restrict__ val, const double* __restrict__ diag,
                                          const double* __restrict__ x, std::uint32_t r) {
    const std::uint32_t deg = e.degree[r];
    double sum = diag[r] * x[r];
    if (e.width <= 8) {
        double v[8], g[8];
#pragma unroll
        for (std::uint32_t j = 0; j < 8; ++j) {
            const std::size_t at = std::size_t(j < e.width ? j : 0u) * e.rows + r;
            v[j] = val[at];
            g[j] = x[e.col[at]];
        }
#pragma unroll
        for (std::uint32_t j = 0; j < 8; ++j) {
            if (j < deg) sum += v[j] * g[j];
        }
        return sum;
    }
    for (std::uint32_t j = 0; j < e.width; ++j) {
        if (j < deg) sum += val[std::size_t(j) * e.rows + r] * x[e.col[std::size_t(j) * e.rows + r]];
    }
    return sum;
}

__global__ void k_ell_apply(Ell e, const double* __restrict__ val, const double* __restrict__ diag,
                            const double* __restrict__ x, double* __restrict__ y) {
    const std::uint32_t r = blockIdx.x * kThreads + threadIdx.x;
    if (r < e.rows) y[r] = ell_row(e, val, diag, x, r);
}

// v = A p_hat and shadow . v; or t = A s_hat, t . t and t . s (`second`).
__global__ void __launch_bounds__(kThreads) k_bicg_apply(Ell e, const double* __restrict__ val, const double* __restrict__ diag,
                                                         const double* __restrict__ x, double* __restrict__ y,
                                                         const double* __restrict__ u, bool second, BicgState* state,
                                                         double* partial) {
    __shared__ double sh[kThreads];
    if (second ? state->skip_second != 0 : state->done != 0) return;
    const std::uint32_t r = blockIdx.x * kThreads + threadIdx.x;
    double yv = 0.0, uv = 0.0;
    if (r < e.rows) {
        yv = ell_row(e, val, diag, x, r);
        y[r] = yv;
        uv = u[r];
    }
    const bool on = r < e.rows;
    const double yy = yv * yv, yu = yv * uv;
    sum_and_step(second ? kSumT : kSumV, on ? (second ? yy : yu) : 0.0, on && second ? yu : 0.0, sh, partial, state);
}

// Device scratch and the scalars read back for the host's decisions.
class Scalars {
  public:
    Scalars(DeviceStore& store, std::size_t n) : blocks_(blocks_of(n)) {
        partial_ = store.alloc<double>(std::size_t(blocks_) * kQ);
        out_ = store.alloc<double>(kQ);
        host_.reset(kQ);
    }
    double* partial() { return partial_; }
    unsigned blocks() const { return blocks_; }
    // Finishes `q` partials already written.
    std::pair<double, double> read(int q, unsigned max_mask, cudaStream_t st) {
        k_finish<<<1, kThreads, 0, st>>>(blocks_, q, max_mask, partial_, out_);
        PSGB_CHECK_LAUNCH();
        PSGB_CUDA(cudaMemcpyAsync(host_.data(), out_, q * sizeof(double), cudaMemcpyDeviceToHost, st));
        PSGB_CUDA(cudaStreamSynchronize(st));
        return {host_.data()[0], q > 1 ? host_.data()[1] : 0.0};
    }

  private:
    unsigned blocks_;
    double* partial_;
    double* out_;
    PinnedDoubles host_;
};

// M^-1 x; `skip` a device word that, where set, makes it needless.
using Precondition = std::function<void(const double*, double*, const int* skip)>;

// BiCGSTAB's vectors, device state and the host's copies of it, kept with the caller's workspace.
struct BicgWork {
    double *r, *shadow, *p, *v, *p_hat, *s, *s_hat, *t;
    BicgState* state;
    BicgState* host = nullptr;          // [2], pinned
    cudaEvent_t seen[2] = {nullptr, nullptr};
    BicgWork(DeviceStore& store, std::size_t n)
        : r(store.alloc<double>(n)), shadow(store.alloc<double>(n)), p(store.alloc<double>(n)),
          v(store.alloc<double>(n)), p_hat(store.alloc<double>(n)), s(store.alloc<double>(n)),
          s_hat(store.alloc<double>(n)), t(store.alloc<double>(n)), state(store.alloc<BicgState>(1)) {
        PSGB_CUDA(cudaMallocHost(reinterpret_cast<void**>(&host), 2 * sizeof(BicgState)));
        for (cudaEvent_t& e : seen) PSGB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    BicgWork(const BicgWork&) = delete;
    BicgWork& operator=(const BicgWork&) = delete;
    ~BicgWork() {
        for (cudaEvent_t e : seen)
            if (e != nullptr) cudaEventDestroy(e);
        if (host != nullptr) cudaFreeHost(host);
    }
};

// Right-preconditioned BiCGSTAB (heat_transport.cpp:823-897): x <- A^-1 b from x = 0, A on its
// ELL copy. `ahead`: the host queues one iteration more than it has seen the state of; what is
// queued past the end finds `done` set and returns at once. A preconditioner that cannot be left
// out on the device (a V-cycle of many launches) is not queued ahead: the host reads the state
// before each one.
int bicgstab(const Ell& ell, const double* val, const double* diag, const Precondition& precondition, bool ahead,
             const double* b, double* x, double tolerance, int max_iterations, const BicgWork& w, Scalars& sc,
             cudaStream_t st) {
    const std::uint32_t n = ell.rows;
    const unsigned g = blocks_of(n);
    const int *done = &w.state->done, *skip_second = &w.state->skip_second;
    BicgState begin{};
    begin.max_iterations = max_iterations;
    begin.tolerance = tolerance;
    w.host[0] = begin;
    PSGB_CUDA(cudaMemcpyAsync(w.state, &w.host[0], sizeof(BicgState), cudaMemcpyHostToDevice, st));
    k_bicg_start<<<g, kThreads, 0, st>>>(n, b, x, w.r, w.shadow, w.p, w.v, w.state, sc.partial());
    PSGB_CHECK_LAUNCH();
    const auto read = [&]() -> const BicgState& {
        PSGB_CUDA(cudaMemcpyAsync(&w.host[0], w.state, sizeof(BicgState), cudaMemcpyDeviceToHost, st));
        PSGB_CUDA(cudaStreamSynchronize(st));
        return w.host[0];
    };
    if (!ahead && read().done != 0) return 0;
    for (int queued = 0; queued < std::max(1, max_iterations); ++queued) {
        k_bicg_p<<<g, kThreads, 0, st>>>(n, w.r, w.p, w.v, w.state);
        precondition(w.p, w.p_hat, done);
        k_bicg_apply<<<g, kThreads, 0, st>>>(ell, val, diag, w.p_hat, w.v, w.shadow, false, w.state, sc.partial());
        k_bicg_s<<<g, kThreads, 0, st>>>(n, w.r, w.v, w.s, w.state, sc.partial());
        if (ahead || read().skip_second == 0) {
            precondition(w.s, w.s_hat, skip_second);
            k_bicg_apply<<<g, kThreads, 0, st>>>(ell, val, diag, w.s_hat, w.t, w.s, true, w.state, sc.partial());
        }
        k_bicg_x<<<g, kThreads, 0, st>>>(n, x, w.r, w.p_hat, w.s_hat, w.s, w.t, w.shadow, w.state, sc.partial());
        if (!ahead) {
            PSGB_CHECK_LAUNCH();
            if (read().done != 0) break;
            continue;
        }
        PSGB_CHECK_LAUNCH();
        const int slot = queued & 1;
        PSGB_CUDA(cudaMemcpyAsync(&w.host[slot], w.state, sizeof(BicgState), cudaMemcpyDeviceToHost, st));
        PSGB_CUDA(cudaEventRecord(w.seen[slot], st));
        if (queued == 0) continue;
        PSGB_CUDA(cudaEventSynchronize(w.seen[slot ^ 1]));
        if (w.host[slot ^ 1].done != 0) return w.host[slot ^ 1].iteration;
    }
    return ahead ? read().iteration : w.host[0].iteration;
}

// ---- advection-diffusion source ----------------------------------------------------

struct Transport {
    std::uint32_t layers;
    const double* conductance;   // [entries]
    const double* outflow;       // [layers][entries]
    const double* latent;        // [nodes] or null
    double heat_capacity;
};

struct GraphView {
    std::uint32_t nodes, entries;
    const std::uint32_t* offset;
    const std::uint32_t* neighbour;
    const double* area;
};

// H_eddy and H_advective per node (heat_transport.cpp:795-813).
__global__ void k_advection_source(GraphView g, Transport tr, const double* __restrict__ mean,
                                   const double* __restrict__ energy, double* __restrict__ eddy_out,
                                   double* __restrict__ advective_out) {
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    if (a >= g.nodes) return;
    double eddy = 0.0, advective = 0.0;
    for (std::uint32_t k = g.offset[a]; k < g.offset[a + 1]; ++k) {
        const std::uint32_t b = g.neighbour[k];
        eddy += tr.conductance[k] * (mean[b] - mean[a]);
        for (std::uint32_t l = 0; l < tr.layers; ++l) {
            const double out = tr.outflow[std::size_t(l) * g.entries + k];
            const std::uint32_t upwind = out > 0.0 ? a : b;
            advective -= out * energy[std::size_t(l) * g.nodes + upwind];
        }
    }
    double e = eddy / g.area[a];
    if (tr.latent != nullptr) e -= tr.latent[a];
    eddy_out[a] = e;
    advective_out[a] = advective / g.area[a];
}

// F = h - (H_eddy + H_adv) and the block partials of sum A F^2 and max |F|.
__global__ void __launch_bounds__(kThreads) k_advection_residual(GraphView g, const double* __restrict__ h,
                                                                 const double* __restrict__ eddy,
                                                                 const double* __restrict__ advective,
                                                                 double* __restrict__ residual,
                                                                 double* __restrict__ partial) {
    __shared__ double sh[kThreads];
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    double merit = 0.0, largest = 0.0;
    if (a < g.nodes) {
        const double r = h[a] - (eddy[a] + advective[a]);
        residual[a] = r;
        merit = g.area[a] * r * r;
        largest = fabs(r);
    }
    const double s = tree_sum(merit, sh);
    const double m = tree_max(largest, sh);
    if (threadIdx.x == 0) {
        partial[blockIdx.x * kQ + 0] = s;
        partial[blockIdx.x * kQ + 1] = m;
    }
}

// The Newton matrix J = I - dH/dh on the graph's pattern and the right-hand side -F
// (heat_transport.cpp:1171-1195); the V-cycle's symmetric matrix A/theta' + K
// (heat_transport.cpp:1220-1232).
__global__ void k_advection_jacobian(GraphView g, Transport tr, const double* __restrict__ slope,
                                     const double* __restrict__ energy_slope, const double* __restrict__ residual,
                                     double* __restrict__ diagonal, double* __restrict__ off, double* __restrict__ rhs,
                                     double* __restrict__ sym_diagonal, double* __restrict__ sym_off) {
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    if (a >= g.nodes) return;
    const double inverse_area = 1.0 / g.area[a];
    double own = 0.0, conductance_sum = 0.0;
    for (std::uint32_t k = g.offset[a]; k < g.offset[a + 1]; ++k) {
        const std::uint32_t b = g.neighbour[k];
        const double G = tr.conductance[k];
        own -= G * slope[a];
        double neighbour = G * slope[b];
        for (std::uint32_t l = 0; l < tr.layers; ++l) {
            const double out = tr.outflow[std::size_t(l) * g.entries + k];
            if (out > 0.0) {
                own -= out * energy_slope[std::size_t(l) * g.nodes + a];
            } else {
                neighbour -= out * energy_slope[std::size_t(l) * g.nodes + b];
            }
        }
        off[k] = -neighbour * inverse_area;
        conductance_sum += G;
        sym_off[k] = -G;
    }
    diagonal[a] = 1.0 - own * inverse_area;
    rhs[a] = -residual[a];
    sym_diagonal[a] = g.area[a] / std_max(slope[a], 1.0e-12) + conductance_sum;
}

// scaled = A x
__global__ void k_scale_area(std::uint32_t n, const double* __restrict__ area, const double* __restrict__ x,
                             double* __restrict__ out) {
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    if (a < n) out[a] = area[a] * x[a];
}
// y /= max(theta', 1e-12)
__global__ void k_unscale_slope(std::uint32_t n, const double* __restrict__ slope, double* __restrict__ y) {
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    if (a < n) y[a] /= std_max(slope[a], 1.0e-12);
}
// leftover = x - leftover
__global__ void k_leftover(std::uint32_t n, const double* __restrict__ x, double* __restrict__ leftover) {
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    if (a < n) leftover[a] = x[a] - leftover[a];
}
__global__ void k_add(std::uint32_t n, const double* __restrict__ d, double* __restrict__ y) {
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    if (a < n) y[a] += d[a];
}
// h0 = max(initial, floor) or max(0, floor)
__global__ void k_advection_start(std::uint32_t n, const double* __restrict__ initial, const double* __restrict__ floor,
                                  double* __restrict__ h) {
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    if (a >= n) return;
    h[a] = initial != nullptr ? std_max(initial[a], floor[a]) : std_max(0.0, floor[a]);
}
// trial = max(h + step delta, floor)
__global__ void k_advection_trial(std::uint32_t n, const double* __restrict__ h, const double* __restrict__ delta,
                                  double step, const double* __restrict__ floor, double* __restrict__ trial) {
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    if (a >= n) return;
    trial[a] = std_max(h[a] + step * delta[a], floor[a]);
}
// H = eddy + advective and the block partials of sum A H, sum A|H|, sum A|H_eddy|, sum A|H_adv|
__global__ void __launch_bounds__(kThreads) k_advection_final(GraphView g, const double* __restrict__ eddy,
                                                              const double* __restrict__ advective,
                                                              double* __restrict__ out, double* __restrict__ partial) {
    __shared__ double sh[kThreads];
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    double q0 = 0.0, q1 = 0.0, q2 = 0.0, q3 = 0.0;
    if (a < g.nodes) {
        const double H = eddy[a] + advective[a];
        out[a] = H;
        const double area = g.area[a];
        q0 = area * H;
        q1 = area * fabs(H);
        q2 = area * fabs(eddy[a]);
        q3 = area * fabs(advective[a]);
    }
    const double s0 = tree_sum(q0, sh), s1 = tree_sum(q1, sh), s2 = tree_sum(q2, sh), s3 = tree_sum(q3, sh);
    if (threadIdx.x == 0) {
        partial[blockIdx.x * kQ + 0] = s0;
        partial[blockIdx.x * kQ + 1] = s1;
        partial[blockIdx.x * kQ + 2] = s2;
        partial[blockIdx.x * kQ + 3] = s3;
    }
}

// ---- the tracer ---------------------------------------------------------------------

struct Stacked {
    std::uint32_t nodes, layers, rows, entries;
    const std::uint32_t* offset;      // stacked CSR
    const std::uint32_t* neighbour;
};

// Each node's upward fluxes W_{l+1/2} (0 for the top) and |final W| (heat_transport.cpp:921-931).
__global__ void k_tracer_vertical(GraphView g, Transport tr, double* __restrict__ vertical,
                                  double* __restrict__ divergence) {
    const std::uint32_t a = blockIdx.x * kThreads + threadIdx.x;
    if (a >= g.nodes) return;
    const std::uint32_t L = tr.layers;
    double w = 0.0;
    for (std::uint32_t l = 0; l < L; ++l) {
        for (std::uint32_t k = g.offset[a]; k < g.offset[a + 1]; ++k) w -= tr.outflow[std::size_t(l) * g.entries + k];
        vertical[std::size_t(a) * L + l] = l + 1 < L ? w : 0.0;
    }
    divergence[a] = fabs(w);
}

// The stacked system's diagonal, off-diagonals and right-hand side (heat_transport.cpp:
// 960-991) and the node-major start c0.
__global__ void k_tracer_assemble(GraphView g, Transport tr, Stacked s, const double* __restrict__ mass, double dt,
                                  double exchange_scale, const double* __restrict__ vertical,
                                  const double* __restrict__ tracer, double* __restrict__ diagonal,
                                  double* __restrict__ off, double* __restrict__ rhs, double* __restrict__ start) {
    const std::uint32_t row = blockIdx.x * kThreads + threadIdx.x;
    if (row >= s.rows) return;
    const std::uint32_t L = tr.layers, a = row / L, l = row % L;
    const double rate = mass[a] / dt;
    double own = rate;
    std::uint32_t at = s.offset[row];
    for (std::uint32_t k = g.offset[a]; k < g.offset[a + 1]; ++k, ++at) {
        const double flow = tr.outflow[std::size_t(l) * g.entries + k];
        const double eddy = tr.conductance[k] * exchange_scale;
        own += std_max(flow, 0.0) + eddy;
        off[at] = -std_max(-flow, 0.0) - eddy;
    }
    const double below = l > 0 ? vertical[std::size_t(a) * L + l - 1] : 0.0;
    const double above = vertical[row];
    if (l > 0) {
        own += std_max(-below, 0.0);
        off[at++] = -std_max(below, 0.0);
    }
    if (l + 1 < L) {
        own += std_max(above, 0.0);
        off[at++] = -std_max(-above, 0.0);
    }
    diagonal[row] = own;
    const double c0 = tracer[std::size_t(l) * g.nodes + a];
    rhs[row] = rate * c0;
    start[row] = c0;
}

// residual = rhs - applied
__global__ void k_sub(std::uint32_t n, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ out) {
    const std::uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i < n) out[i] = a[i] - b[i];
}
// solved = max(0, c0 + delta)
__global__ void k_tracer_solved(std::uint32_t n, const double* __restrict__ start, const double* __restrict__ delta,
                                double* __restrict__ solved) {
    const std::uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    solved[i] = std_max(0.0, start[i] + delta[i]);
}
// block partials of sum (rhs - applied)^2 and sum rhs^2
__global__ void __launch_bounds__(kThreads) k_tracer_norms(std::uint32_t n, const double* __restrict__ rhs,
                                                           const double* __restrict__ applied,
                                                           double* __restrict__ partial) {
    __shared__ double sh[kThreads];
    const std::uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    double d = 0.0, r = 0.0;
    if (i < n) {
        d = (rhs[i] - applied[i]) * (rhs[i] - applied[i]);
        r = rhs[i] * rhs[i];
    }
    const double s0 = tree_sum(d, sh), s1 = tree_sum(r, sh);
    if (threadIdx.x == 0) {
        partial[blockIdx.x * kQ + 0] = s0;
        partial[blockIdx.x * kQ + 1] = s1;
    }
}

// The flux form of the solution (heat_transport.cpp:1042-1078), per row in the
// reference's accumulation order: faces from lower nodes (ascending), the vertical flux
// from below, the row's own faces to higher nodes (CSR order), the vertical flux up.
// Then c' = c + dt change / M, clipped at 0 (the mass added is summed in partials).
__global__ void __launch_bounds__(kThreads) k_tracer_flux_form(GraphView g, Transport tr, const double* __restrict__ mass,
                                                               double dt, double exchange_scale,
                                                               const std::uint32_t* __restrict__ face_order,
                                                               const std::uint32_t* __restrict__ lower_count,
                                                               const std::uint32_t* __restrict__ reverse,
                                                               const double* __restrict__ vertical,
                                                               const double* __restrict__ solved,
                                                               const double* __restrict__ tracer,
                                                               double* __restrict__ out, double* __restrict__ partial) {
    __shared__ double sh[kThreads];
    const std::uint32_t L = tr.layers;
    const std::uint32_t row = blockIdx.x * kThreads + threadIdx.x;
    double clipped = 0.0;
    if (row < g.nodes * L) {
        const std::uint32_t a = row / L, l = row % L;
        const std::uint32_t first = g.offset[a], split = first + lower_count[a], last = g.offset[a + 1];
        double change = 0.0;
        for (std::uint32_t idx = first; idx < split; ++idx) {   // faces b -> a, b < a
            const std::uint32_t k = face_order[idx];
            const std::uint32_t b = g.neighbour[k], kb = reverse[k];
            const std::uint32_t donor = b * L + l;
            const double flow = tr.outflow[std::size_t(l) * g.entries + kb];
            const double eddy = tr.conductance[kb] * exchange_scale;
            const double flux = (flow > 0.0 ? flow * solved[donor] : flow * solved[row]) +
                                eddy * (solved[donor] - solved[row]);
            change += flux;
        }
        if (l > 0) {
            const double w = vertical[row - 1];
            change += w > 0.0 ? w * solved[row - 1] : w * solved[row];
        }
        for (std::uint32_t idx = split; idx < last; ++idx) {    // faces a -> b, b > a
            const std::uint32_t k = face_order[idx];
            const std::uint32_t other = g.neighbour[k] * L + l;
            const double flow = tr.outflow[std::size_t(l) * g.entries + k];
            const double eddy = tr.conductance[k] * exchange_scale;
            const double flux = (flow > 0.0 ? flow * solved[row] : flow * solved[other]) +
                                eddy * (solved[row] - solved[other]);
            change -= flux;
        }
        if (l + 1 < L) {
            const double w = vertical[row];
            change -= w > 0.0 ? w * solved[row] : w * solved[row + 1];
        }
        const std::size_t at = std::size_t(l) * g.nodes + a;
        double value = tracer[at] + dt * change / mass[a];
        if (value < 0.0) {
            clipped = -(value * mass[a]);
            value = 0.0;
        }
        out[at] = value;
    }
    const double s = tree_sum(clipped, sh);
    if (threadIdx.x == 0) partial[blockIdx.x * kQ] = s;
}

}  // namespace

// ---- per-planet structures ------------------------------------------------------------

// The tracer solve's vectors, kept with its stacked system: allocating and freeing two dozen of
// them, and their pinned host copies, took 1.5 ms of every call.
struct TracerWork {
    DeviceStore store;
    double *vertical, *divergence, *diagonal, *off, *rhs, *start, *applied, *residual, *delta, *solved, *off_ell;
    Scalars scalars;
    BicgWork bicg;
    TracerWork(std::size_t rows, std::size_t nodes, std::size_t entries, std::size_t width)
        : vertical(store.alloc<double>(rows)), divergence(store.alloc<double>(nodes)), diagonal(store.alloc<double>(rows)),
          off(store.alloc<double>(entries)), rhs(store.alloc<double>(rows)), start(store.alloc<double>(rows)),
          applied(store.alloc<double>(rows)), residual(store.alloc<double>(rows)), delta(store.alloc<double>(rows)),
          solved(store.alloc<double>(rows)), off_ell(store.alloc<double>(width * rows)), scalars(store, rows),
          bicg(store, rows) {}
};

struct NonsymContext {
    DeviceStore store;
    GraphView graph{};
    Ell graph_ell{};
    std::uint32_t* face_order = nullptr;
    std::uint32_t* lower_count = nullptr;
    std::uint32_t* reverse = nullptr;
    std::unique_ptr<DeviceIlu> graph_ilu;
    struct StackedSystem {
        DeviceStore store;
        Stacked view{};
        Ell ell{};
        std::unique_ptr<DeviceIlu> ilu;
        std::unique_ptr<TracerWork> work;   // on the first solve
    };
    std::map<std::uint32_t, std::unique_ptr<StackedSystem>> stacked;
};

std::size_t device_bytes(const NonsymContext& c) {
    std::size_t bytes = c.store.bytes() + (c.graph_ilu ? c.graph_ilu->device_bytes() : 0);
    for (const auto& [layers, s] : c.stacked) {
        bytes += s->store.bytes() + (s->ilu ? s->ilu->device_bytes() : 0) + (s->work ? s->work->store.bytes() : 0);
    }
    return bytes;
}

namespace {

// The ELL shape of a CSR pattern (columns slot-major, degrees), in `store`.
Ell ell_of(DeviceStore& store, const std::vector<std::uint32_t>& offset, const std::vector<std::uint32_t>& neighbour) {
    Ell e{};
    e.rows = static_cast<std::uint32_t>(offset.size() - 1);
    for (std::uint32_t r = 0; r < e.rows; ++r) e.width = std::max(e.width, offset[r + 1] - offset[r]);
    if (e.width > 255) throw std::logic_error("non-symmetric solve: a row with more than 255 couplings");
    std::vector<std::uint8_t> degree(e.rows);
    std::vector<std::uint32_t> col(std::size_t(e.width) * e.rows, 0);
    for (std::uint32_t r = 0; r < e.rows; ++r) {
        degree[r] = static_cast<std::uint8_t>(offset[r + 1] - offset[r]);
        for (std::uint32_t j = 0; j < degree[r]; ++j) col[std::size_t(j) * e.rows + r] = neighbour[offset[r] + j];
    }
    e.degree = store.upload(degree);
    e.col = store.upload(col);
    return e;
}

NonsymContext& context(psgb_planet* h) {
    if (h->nonsym) return *h->nonsym;
    upload_planet(*h->planet);
    auto c = std::make_shared<NonsymContext>();
    const TransportGraph& g = h->planet->graph;
    const std::uint32_t n = static_cast<std::uint32_t>(g.size());
    c->graph.nodes = n;
    c->graph.entries = static_cast<std::uint32_t>(g.neighbour.size());
    c->graph.offset = c->store.upload(g.offset);
    c->graph.neighbour = c->store.upload(g.neighbour);
    c->graph.area = h->planet->dev.graph_area;
    std::vector<std::uint32_t> reverse(g.neighbour.size()), order(g.neighbour.size()), lower(n);
    for (std::uint32_t a = 0; a < n; ++a) {
        std::vector<std::pair<std::uint32_t, std::uint32_t>> below;
        std::vector<std::uint32_t> above;
        for (std::uint32_t k = g.offset[a]; k < g.offset[a + 1]; ++k) {
            const std::uint32_t b = g.neighbour[k];
            bool found = false;
            for (std::uint32_t q = g.offset[b]; q < g.offset[b + 1]; ++q) {
                if (g.neighbour[q] == a) {
                    reverse[k] = q;
                    found = true;
                }
            }
            if (!found) throw std::logic_error("transport graph is not symmetric");
            if (b < a) below.emplace_back(b, k);
            else above.push_back(k);
        }
        std::sort(below.begin(), below.end());
        std::uint32_t at = g.offset[a];
        for (const auto& [b, k] : below) order[at++] = k;
        for (std::uint32_t k : above) order[at++] = k;
        lower[a] = static_cast<std::uint32_t>(below.size());
    }
    c->reverse = c->store.upload(reverse);
    c->face_order = c->store.upload(order);
    c->lower_count = c->store.upload(lower);
    c->graph_ilu = std::make_unique<DeviceIlu>(ilu_pattern(g.offset, g.neighbour, fixed_blocks(n, 1)));
    c->graph_ell = ell_of(c->store, g.offset, g.neighbour);
    h->nonsym = c;
    return *c;
}

NonsymContext::StackedSystem& stacked_system(psgb_planet* h, std::uint32_t layers) {
    NonsymContext& c = context(h);
    auto it = c.stacked.find(layers);
    if (it != c.stacked.end()) return *it->second;
    const TransportGraph& g = h->planet->graph;
    const std::uint32_t n = static_cast<std::uint32_t>(g.size());
    // Node-major rows a L + l: the graph row's entries in this layer, then the layer below
    // and the one above (heat_transport.cpp:940-957).
    std::vector<std::uint32_t> offset{0}, neighbour;
    for (std::uint32_t a = 0; a < n; ++a) {
        for (std::uint32_t l = 0; l < layers; ++l) {
            const std::uint32_t row = a * layers + l;
            for (std::uint32_t k = g.offset[a]; k < g.offset[a + 1]; ++k) neighbour.push_back(g.neighbour[k] * layers + l);
            if (l > 0) neighbour.push_back(row - 1);
            if (l + 1 < layers) neighbour.push_back(row + 1);
            offset.push_back(static_cast<std::uint32_t>(neighbour.size()));
        }
    }
    auto s = std::make_unique<NonsymContext::StackedSystem>();
    s->view.nodes = n;
    s->view.layers = layers;
    s->view.rows = n * layers;
    s->view.entries = static_cast<std::uint32_t>(neighbour.size());
    s->view.offset = s->store.upload(offset);
    s->view.neighbour = s->store.upload(neighbour);
    s->ilu = std::make_unique<DeviceIlu>(ilu_pattern(offset, neighbour, fixed_blocks(n, layers)));
    s->ell = ell_of(s->store, offset, neighbour);
    auto& ref = *s;
    c.stacked.emplace(layers, std::move(s));
    return ref;
}

// Device copies of the caller's transport (when it passes host arrays).
struct TransportIn {
    DeviceStore store;
    Transport view{};
};

void load_transport(TransportIn& t, const psgb_advection_diffusion* in, const GraphView& g, int memory,
                    cudaStream_t st) {
    require(in != nullptr && in->conductance_W_K != nullptr && in->outflow_kg_s != nullptr, "null argument");
    require(in->heat_capacity_J_kg_K > 0.0, "the heat capacity must be positive");
    t.view.layers = in->layers;
    t.view.heat_capacity = in->heat_capacity_J_kg_K;
    const std::size_t E = g.entries;
    if (memory == PSGB_MEMORY_DEVICE) {
        t.view.conductance = in->conductance_W_K;
        t.view.outflow = in->outflow_kg_s;
        t.view.latent = in->eddy_latent_W_m2;
        return;
    }
    double* c = t.store.alloc<double>(E);
    double* o = t.store.alloc<double>(std::max<std::size_t>(1, std::size_t(in->layers) * E));
    PSGB_CUDA(cudaMemcpyAsync(c, in->conductance_W_K, E * 8, cudaMemcpyHostToDevice, st));
    if (in->layers > 0)
        PSGB_CUDA(cudaMemcpyAsync(o, in->outflow_kg_s, std::size_t(in->layers) * E * 8, cudaMemcpyHostToDevice, st));
    t.view.conductance = c;
    t.view.outflow = o;
    t.view.latent = nullptr;
    if (in->eddy_latent_W_m2 != nullptr) {
        double* e = t.store.alloc<double>(g.nodes);
        PSGB_CUDA(cudaMemcpyAsync(e, in->eddy_latent_W_m2, std::size_t(g.nodes) * 8, cudaMemcpyHostToDevice, st));
        t.view.latent = e;
    }
}

const double* input(DeviceStore& store, const double* p, std::size_t n, int memory, cudaStream_t st) {
    if (p == nullptr || memory == PSGB_MEMORY_DEVICE) return p;
    double* d = store.alloc<double>(n);
    PSGB_CUDA(cudaMemcpyAsync(d, p, n * 8, cudaMemcpyHostToDevice, st));
    return d;
}

void output(double* dst, const double* src, std::size_t n, int memory, cudaStream_t st) {
    PSGB_CUDA(cudaMemcpyAsync(dst, src, n * 8,
                              memory == PSGB_MEMORY_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st));
}

void require_memory(int memory) {
    require(memory == PSGB_MEMORY_HOST || memory == PSGB_MEMORY_DEVICE,
            "memory must be PSGB_MEMORY_HOST or PSGB_MEMORY_DEVICE");
}

}  // namespace
}  // namespace psgb

using psgb::capi::guarded;

struct psgb_incomplete_lu {
    psgb::DeviceStore store;
    std::unique_ptr<psgb::DeviceIlu> ilu;
};

extern "C" {

int psgb_incomplete_lu_create(uint32_t rows, const uint32_t* offset, const uint32_t* neighbour, const double* diagonal,
                              const double* off, const uint32_t* block_start, uint32_t blocks, double diagonal_scale,
                              psgb_incomplete_lu** out) {
    return guarded([&] {
        psgb::require(out != nullptr && offset != nullptr && diagonal != nullptr && block_start != nullptr &&
                          (offset[rows] == 0 || (neighbour != nullptr && off != nullptr)),
                      "null argument");
        *out = nullptr;
        std::vector<std::uint32_t> o(offset, offset + rows + 1), nb(neighbour, neighbour + offset[rows]),
            bs(block_start, block_start + blocks + 1);
        auto h = std::make_unique<psgb_incomplete_lu>();
        h->ilu = std::make_unique<psgb::DeviceIlu>(psgb::ilu_pattern(o, nb, bs));
        double* d = h->store.upload(std::vector<double>(diagonal, diagonal + rows));
        double* f = h->store.upload(std::vector<double>(off, off + offset[rows]));
        h->ilu->factor(d, f, diagonal_scale, nullptr);
        *out = h.release();
        return PSGB_OK;
    });
}

int psgb_incomplete_lu_solve(psgb_incomplete_lu* h, double* x, int memory, void* stream) {
    return guarded([&] {
        psgb::require(h != nullptr && x != nullptr, "null argument");
        psgb::require_memory(memory);
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        const std::size_t n = h->ilu->rows();
        if (memory == PSGB_MEMORY_DEVICE) {
            h->ilu->solve(x, x, st);
            return PSGB_OK;
        }
        psgb::DeviceStore scratch;
        double* d = scratch.alloc<double>(n);
        PSGB_CUDA(cudaMemcpyAsync(d, x, n * 8, cudaMemcpyHostToDevice, st));
        h->ilu->solve(d, d, st);
        PSGB_CUDA(cudaMemcpyAsync(x, d, n * 8, cudaMemcpyDeviceToHost, st));
        PSGB_CUDA(cudaStreamSynchronize(st));
        return PSGB_OK;
    });
}

void psgb_incomplete_lu_destroy(psgb_incomplete_lu* h) { delete h; }

int psgb_advection_diffusion_source(psgb_planet* planet, const psgb_advection_diffusion* transport,
                                    const double* mean_K, const double* energy_J_kg, double* eddy_W_m2,
                                    double* advective_W_m2, int memory, void* stream) {
    return guarded([&] {
        psgb::require(planet != nullptr && transport != nullptr && mean_K != nullptr && eddy_W_m2 != nullptr &&
                          advective_W_m2 != nullptr,
                      "null argument");
        psgb::require(energy_J_kg != nullptr || transport->layers == 0, "null argument");
        psgb::require_memory(memory);
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        psgb::NonsymContext& c = psgb::context(planet);
        const psgb::GraphView& g = c.graph;
        psgb::TransportIn tr;
        psgb::load_transport(tr, transport, g, memory, st);
        psgb::DeviceStore scratch;
        const double* m = psgb::input(scratch, mean_K, g.nodes, memory, st);
        const double* e = psgb::input(scratch, energy_J_kg, std::size_t(transport->layers) * g.nodes, memory, st);
        double* eo = memory == PSGB_MEMORY_DEVICE ? eddy_W_m2 : scratch.alloc<double>(g.nodes);
        double* ao = memory == PSGB_MEMORY_DEVICE ? advective_W_m2 : scratch.alloc<double>(g.nodes);
        psgb::k_advection_source<<<psgb::blocks_of(g.nodes), psgb::kThreads, 0, st>>>(g, tr.view, m, e, eo, ao);
        PSGB_CHECK_LAUNCH();
        if (memory == PSGB_MEMORY_HOST) {
            psgb::output(eddy_W_m2, eo, g.nodes, memory, st);
            psgb::output(advective_W_m2, ao, g.nodes, memory, st);
        }
        PSGB_CUDA(cudaStreamSynchronize(st));
        return PSGB_OK;
    });
}

int psgb_solve_implicit_tracer(psgb_planet* planet, const psgb_advection_diffusion* transport,
                               const double* layer_mass_kg, const double* tracer, double dt_s,
                               double relative_tolerance, int max_iterations, double* tracer_out,
                               psgb_tracer_result* result, int memory, void* stream) {
    return guarded([&] {
        psgb::require(planet != nullptr && transport != nullptr && layer_mass_kg != nullptr && tracer != nullptr &&
                          tracer_out != nullptr,
                      "null argument");
        psgb::require_memory(memory);
        psgb::require(transport->layers > 0 && dt_s > 0.0, "tracer transport inputs do not match the graph");
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        psgb::NonsymContext& c = psgb::context(planet);
        const psgb::GraphView& g = c.graph;
        const std::uint32_t L = transport->layers;
        psgb::NonsymContext::StackedSystem& S = psgb::stacked_system(planet, L);
        psgb::TransportIn tr;
        psgb::load_transport(tr, transport, g, memory, st);
        psgb::DeviceStore w;
        const double* mass = psgb::input(w, layer_mass_kg, g.nodes, memory, st);
        const double* c0 = psgb::input(w, tracer, std::size_t(L) * g.nodes, memory, st);
        const std::size_t rows = S.view.rows;
        const std::uint32_t urows = static_cast<std::uint32_t>(rows);
        if (!S.work) S.work = std::make_unique<psgb::TracerWork>(rows, g.nodes, S.view.entries, S.ell.width);
        psgb::TracerWork& k = *S.work;
        double *vertical = k.vertical, *divergence = k.divergence, *diagonal = k.diagonal, *off = k.off, *rhs = k.rhs,
               *start = k.start, *applied = k.applied, *residual = k.residual, *delta = k.delta, *solved = k.solved,
               *off_ell = k.off_ell;
        psgb::Scalars& sc = k.scalars;
        double* out = memory == PSGB_MEMORY_DEVICE ? tracer_out : w.alloc<double>(rows);
        const double exchange_scale = 1.0 / (transport->heat_capacity_J_kg_K * static_cast<double>(L));
        const unsigned gn = psgb::blocks_of(g.nodes), gr = psgb::blocks_of(rows);
        psgb::k_tracer_vertical<<<gn, psgb::kThreads, 0, st>>>(g, tr.view, vertical, divergence);
        PSGB_CHECK_LAUNCH();
        psgb::k_tracer_assemble<<<gr, psgb::kThreads, 0, st>>>(g, tr.view, S.view, mass, dt_s, exchange_scale, vertical,
                                                              c0, diagonal, off, rhs, start);
        PSGB_CHECK_LAUNCH();
        S.ilu->factor(diagonal, off, 1.0, st);
        psgb::k_csr_to_ell<<<gr, psgb::kThreads, 0, st>>>(S.ell, S.view.offset, off, off_ell);
        PSGB_CHECK_LAUNCH();
        const auto apply = [&](const double* x, double* y) {
            psgb::k_ell_apply<<<gr, psgb::kThreads, 0, st>>>(S.ell, off_ell, diagonal, x, y);
            PSGB_CHECK_LAUNCH();
        };
        const psgb::Precondition precondition = [&](const double* x, double* y, const int* skip) {
            S.ilu->solve(x, y, st, skip);
        };
        // A delta = b - A c0, from delta = 0.
        apply(start, applied);
        psgb::k_sub<<<gr, psgb::kThreads, 0, st>>>(urows, rhs, applied, residual);
        PSGB_CHECK_LAUNCH();
        psgb_tracer_result r{};
        r.iterations = psgb::bicgstab(S.ell, off_ell, diagonal, precondition, true, residual, delta, relative_tolerance,
                                      max_iterations, k.bicg, sc, st);
        psgb::k_tracer_solved<<<gr, psgb::kThreads, 0, st>>>(urows, start, delta, solved);
        PSGB_CHECK_LAUNCH();
        apply(solved, applied);
        psgb::k_tracer_norms<<<gr, psgb::kThreads, 0, st>>>(urows, rhs, applied, sc.partial());
        PSGB_CHECK_LAUNCH();
        const auto [residual_norm, rhs_norm] = sc.read(2, 0u, st);
        r.relative_residual = rhs_norm > 0.0 ? std::sqrt(residual_norm / rhs_norm) : 0.0;
        std::vector<double> div(g.nodes);   // the largest column divergence, below
        PSGB_CUDA(cudaMemcpyAsync(div.data(), divergence, g.nodes * 8, cudaMemcpyDeviceToHost, st));
        psgb::k_tracer_flux_form<<<gr, psgb::kThreads, 0, st>>>(g, tr.view, mass, dt_s, exchange_scale, c.face_order,
                                                               c.lower_count, c.reverse, vertical, solved, c0, out,
                                                               sc.partial());
        PSGB_CHECK_LAUNCH();
        r.clipped_kg = sc.read(1, 0u, st).first;
        for (double d : div) r.column_divergence_kg_s = std::max(r.column_divergence_kg_s, d);
        if (memory == PSGB_MEMORY_HOST) psgb::output(tracer_out, out, rows, memory, st);
        PSGB_CUDA(cudaStreamSynchronize(st));
        if (result != nullptr) *result = r;
        return PSGB_OK;
    });
}

int psgb_solve_implicit_advection_diffusion(psgb_planet* planet, const psgb_advection_diffusion* transport,
                                            const double* source_floor_W_m2, const double* initial_source_W_m2,
                                            psgb_advection_response host_response,
                                            psgb_device_advection_response device_response, void* user,
                                            const psgb_transport_settings* settings_in, double* source_out_W_m2,
                                            double* mean_out_K, double* energy_out_J_kg,
                                            psgb_advection_result* result, int memory, void* stream) {
    return guarded([&] {
        psgb::require(planet != nullptr && transport != nullptr && source_floor_W_m2 != nullptr &&
                          source_out_W_m2 != nullptr && (host_response != nullptr) != (device_response != nullptr),
                      "null argument (give exactly one of the host and device responses)");
        psgb::require_memory(memory);
        psgb_transport_settings settings;
        psgb_transport_settings_default(&settings);
        if (settings_in != nullptr) settings = *settings_in;
        psgb::require(settings.max_newton_iterations >= 0 && settings.max_line_search_halvings >= 0 &&
                          settings.max_non_monotone_steps >= 0 && settings.max_cg_iterations > 0,
                      "iteration limits must not be negative");
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        psgb::NonsymContext& c = psgb::context(planet);
        const psgb::GraphView& g = c.graph;
        const std::uint32_t n = g.nodes, L = transport->layers;
        const std::size_t nl = std::size_t(L) * n;
        psgb::TransportIn tr;
        psgb::load_transport(tr, transport, g, memory, st);
        {   // eddy conductances must be finite and non-negative (heat_transport.cpp:1094-1098)
            std::vector<double> G(g.entries);
            PSGB_CUDA(cudaMemcpyAsync(G.data(), tr.view.conductance, G.size() * 8, cudaMemcpyDeviceToHost, st));
            PSGB_CUDA(cudaStreamSynchronize(st));
            for (double v : G)
                psgb::require(v >= 0.0 && std::isfinite(v), "eddy conductances must be finite and non-negative");
        }
        psgb::DeviceStore w;
        const double* floor = psgb::input(w, source_floor_W_m2, n, memory, st);
        const double* initial = psgb::input(w, initial_source_W_m2, n, memory, st);
        struct Iterate {
            double *source, *mean, *slope, *energy, *energy_slope, *residual;
            double merit, largest;
        };
        auto make = [&] {
            return Iterate{w.alloc<double>(n), w.alloc<double>(n), w.alloc<double>(n), w.alloc<double>(std::max<std::size_t>(1, nl)),
                           w.alloc<double>(std::max<std::size_t>(1, nl)), w.alloc<double>(n), 0.0, 0.0};
        };
        Iterate current = make(), trial = make();
        double* eddy = w.alloc<double>(n);
        double* advective = w.alloc<double>(n);
        double* diagonal = w.alloc<double>(n);
        double* off = w.alloc<double>(g.entries);
        double* sym_diagonal = w.alloc<double>(n);
        double* sym_off = w.alloc<double>(g.entries);
        double* rhs = w.alloc<double>(n);
        double* delta = w.alloc<double>(n);
        double* scaled = w.alloc<double>(n);
        double* leftover = w.alloc<double>(n);
        psgb::Scalars sc(w, n);
        const psgb::BicgWork work(w, n);
        const unsigned gn = psgb::blocks_of(n);
        // host copies for a host response
        psgb::PinnedDoubles host;
        if (host_response != nullptr) host.reset(3 * std::size_t(n) + 2 * nl + 1);
        auto respond = [&](Iterate& at) {
            if (device_response != nullptr) {
                if (device_response(user, n, L, at.source, at.mean, at.slope, at.energy, at.energy_slope, st) != 0)
                    throw std::runtime_error("the advection response callback failed");
                return;
            }
            double* hs = host.data();
            double *hm = hs + n, *hsl = hm + n, *he = hsl + n, *hes = he + nl;
            PSGB_CUDA(cudaMemcpyAsync(hs, at.source, std::size_t(n) * 8, cudaMemcpyDeviceToHost, st));
            PSGB_CUDA(cudaStreamSynchronize(st));
            if (host_response(user, n, L, hs, hm, hsl, he, hes) != 0)
                throw std::runtime_error("the advection response callback failed");
            PSGB_CUDA(cudaMemcpyAsync(at.mean, hm, std::size_t(n) * 8, cudaMemcpyHostToDevice, st));
            PSGB_CUDA(cudaMemcpyAsync(at.slope, hsl, std::size_t(n) * 8, cudaMemcpyHostToDevice, st));
            if (nl > 0) {
                PSGB_CUDA(cudaMemcpyAsync(at.energy, he, nl * 8, cudaMemcpyHostToDevice, st));
                PSGB_CUDA(cudaMemcpyAsync(at.energy_slope, hes, nl * 8, cudaMemcpyHostToDevice, st));
            }
        };
        // F(h) = h - H(theta(h), s(h)) and the merit sum A F^2 (heat_transport.cpp:1111-1133).
        auto evaluate = [&](Iterate& at) {
            respond(at);
            psgb::k_advection_source<<<gn, psgb::kThreads, 0, st>>>(g, tr.view, at.mean, at.energy, eddy, advective);
            PSGB_CHECK_LAUNCH();
            psgb::k_advection_residual<<<gn, psgb::kThreads, 0, st>>>(g, at.source, eddy, advective, at.residual,
                                                                     sc.partial());
            PSGB_CHECK_LAUNCH();
            const auto [merit, largest] = sc.read(2, 0x2u, st);
            at.merit = merit;
            at.largest = largest;
        };
        psgb::k_advection_start<<<gn, psgb::kThreads, 0, st>>>(n, initial, floor, current.source);
        PSGB_CHECK_LAUNCH();
        evaluate(current);
        psgb_advection_result out{};
        int non_monotone = 0;
        double* off_ell = w.alloc<double>(std::size_t(c.graph_ell.width) * n);
        const auto apply = [&](const double* x, double* y) {
            psgb::k_ell_apply<<<gn, psgb::kThreads, 0, st>>>(c.graph_ell, off_ell, diagonal, x, y);
            PSGB_CHECK_LAUNCH();
        };
        // The V-cycle of A theta'^-1 + K on A x, divided by theta', then the block ILU of J
        // on what is left (heat_transport.cpp:1233-1249).
        const psgb::Precondition precondition = [&](const double* x, double* y, const int*) {
            psgb::k_scale_area<<<gn, psgb::kThreads, 0, st>>>(n, g.area, x, scaled);
            PSGB_CHECK_LAUNCH();
            if (psgb_multigrid_precondition(planet, PSGB_DTYPE_F64, scaled, y, PSGB_MEMORY_DEVICE, st) != PSGB_OK)
                throw std::runtime_error(psgb_last_error());
            psgb::k_unscale_slope<<<gn, psgb::kThreads, 0, st>>>(n, current.slope, y);
            PSGB_CHECK_LAUNCH();
            apply(y, leftover);
            psgb::k_leftover<<<gn, psgb::kThreads, 0, st>>>(n, x, leftover);
            PSGB_CHECK_LAUNCH();
            c.graph_ilu->solve(leftover, leftover, st);
            psgb::k_add<<<gn, psgb::kThreads, 0, st>>>(n, leftover, y);
            PSGB_CHECK_LAUNCH();
        };
        for (int iteration = 0; iteration < settings.max_newton_iterations; ++iteration) {
            if (current.largest <= settings.newton_tolerance_W_m2) break;
            psgb::k_advection_jacobian<<<gn, psgb::kThreads, 0, st>>>(g, tr.view, current.slope, current.energy_slope,
                                                                     current.residual, diagonal, off, rhs, sym_diagonal,
                                                                     sym_off);
            PSGB_CHECK_LAUNCH();
            c.graph_ilu->factor(diagonal, off, 1.0, st);
            psgb::k_csr_to_ell<<<gn, psgb::kThreads, 0, st>>>(c.graph_ell, g.offset, off, off_ell);
            PSGB_CHECK_LAUNCH();
            if (psgb_multigrid_set_matrix(planet, sym_diagonal, sym_off, PSGB_MEMORY_DEVICE, st) != PSGB_OK)
                throw std::runtime_error(psgb_last_error());
            out.linear_iterations += psgb::bicgstab(c.graph_ell, off_ell, diagonal, precondition, false, rhs, delta,
                                                    settings.cg_relative_tolerance, settings.max_cg_iterations, work, sc, st);
            // Backtracking on the merit (heat_transport.cpp:1255-1292).
            double step = 1.0;
            bool accepted = false;
            for (int halving = 0;; ++halving) {
                psgb::k_advection_trial<<<gn, psgb::kThreads, 0, st>>>(n, current.source, delta, step, floor,
                                                                      trial.source);
                PSGB_CHECK_LAUNCH();
                evaluate(trial);
                if (trial.merit < current.merit) {
                    accepted = true;
                    break;
                }
                if (halving == settings.max_line_search_halvings) {
                    if (current.largest > settings.rounding_floor_W_m2 &&
                        non_monotone < settings.max_non_monotone_steps) {
                        ++non_monotone;
                        psgb::k_advection_trial<<<gn, psgb::kThreads, 0, st>>>(n, current.source, delta, 1.0, floor,
                                                                              trial.source);
                        PSGB_CHECK_LAUNCH();
                        evaluate(trial);
                        accepted = std::isfinite(trial.merit) &&
                                   trial.merit <= settings.max_non_monotone_growth * current.merit;
                    }
                    break;
                }
                step *= 0.5;
            }
            if (!accepted) break;
            std::swap(current, trial);
            ++out.newton_iterations;
        }
        // The transport applied: the conservative source of the last iterate's theta and s.
        psgb::k_advection_source<<<gn, psgb::kThreads, 0, st>>>(g, tr.view, current.mean, current.energy, eddy,
                                                               advective);
        PSGB_CHECK_LAUNCH();
        double* H = memory == PSGB_MEMORY_DEVICE ? source_out_W_m2 : w.alloc<double>(n);
        psgb::k_advection_final<<<gn, psgb::kThreads, 0, st>>>(g, eddy, advective, H, sc.partial());
        PSGB_CHECK_LAUNCH();
        psgb::k_finish<<<1, psgb::kThreads, 0, st>>>(sc.blocks(), 4, 0u, sc.partial(), scaled);
        PSGB_CHECK_LAUNCH();
        double sums[4];
        PSGB_CUDA(cudaMemcpyAsync(sums, scaled, sizeof(sums), cudaMemcpyDeviceToHost, st));
        if (memory == PSGB_MEMORY_HOST) psgb::output(source_out_W_m2, H, n, memory, st);
        if (mean_out_K != nullptr) psgb::output(mean_out_K, current.mean, n, memory, st);
        if (energy_out_J_kg != nullptr && nl > 0) psgb::output(energy_out_J_kg, current.energy, nl, memory, st);
        PSGB_CUDA(cudaStreamSynchronize(st));
        out.consistency_residual_W_m2 = current.largest;
        out.sum_W = sums[0];
        out.absolute_sum_W = sums[1];
        out.eddy_absolute_sum_W = sums[2];
        out.advective_absolute_sum_W = sums[3];
        if (result != nullptr) *result = out;
        return PSGB_OK;
    });
}

}  // extern "C"
