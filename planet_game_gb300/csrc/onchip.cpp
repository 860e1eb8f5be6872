// Host side of the on-chip solves (onchip_plan.hpp): which planets, which cluster, where
// everything lies in a block's shared memory.
#include "onchip_plan.hpp"

#include "onchip.hpp"
#include "profile.hpp"

#include <algorithm>
#include <map>
#include <stdexcept>

namespace psgb {

OnchipPlan::~OnchipPlan() {
    for (OnchipClass& c : classes)
        if (c.list != nullptr) cudaFree(c.list);
    for (cudaStream_t s : streams) cudaStreamDestroy(s);
    for (cudaEvent_t e : done) cudaEventDestroy(e);
    if (fork != nullptr) cudaEventDestroy(fork);
}

namespace {

template <typename T>
struct Pick;
template <>
struct Pick<double> {
    static LevelView<double> view(const Batch& b, std::size_t l) { return view64(b, l); }
    static const double* inv(const DenseCoarse& D) { return D.inv64; }
};
template <>
struct Pick<float> {
    static LevelView<float> view(const Batch& b, std::size_t l) { return view32(b, l); }
    static const float* inv(const DenseCoarse& D) { return D.inv32; }
};

std::uint32_t ceil_div(std::uint32_t a, std::uint32_t b) { return (a + b - 1) / b; }

// Rows a block of `cluster` holds of a level. The fine level is shared out in whole 32-row
// warps, the reductions' unit; a coarse one row by row in the fine level's proportion, so that
// an aggregate mostly lies in the block of its members (a gather from another block takes 256
// cycles instead of 55, and a warp of them 12 cycles of the link); a level that sweeps
// block-locally in whole tiles.
std::uint32_t span_of(std::uint32_t n, unsigned cluster, bool fine, bool tiles, double share) {
    if (tiles) return ceil_div(ceil_div(n, 256u), cluster) * 256u;
    if (fine) return ceil_div(ceil_div(n, 32u), cluster) * 32u;
    return std::max(ceil_div(n, cluster), static_cast<std::uint32_t>(share * n + 0.5));
}

// The most member addresses a block holds: each of its coarse rows' padded to whole eights.
std::uint32_t members_most(const HostLevel& fine, std::uint32_t coarse_rows, std::uint32_t span) {
    std::vector<std::uint32_t> of(coarse_rows, 0), held(ceil_div(coarse_rows, span), 0);
    for (std::uint32_t a : fine.aggregate) ++of[a];
    for (std::uint32_t a = 0; a < coarse_rows; ++a) held[a / span] += ceil_div(of[a], 8u) * 8u;
    return *std::max_element(held.begin(), held.end());
}

// Shared-memory layout of a block; returns the bytes, and the offsets in
// `a` when it is given.
template <typename T>
std::size_t layout(const OnchipClass& c, OnchipArgs<T>* a) {
    std::size_t at = 0, o_r0 = 0;
    const auto take = [&](std::size_t bytes) {
        const std::size_t o = at;
        at = (at + bytes + 15) / 16 * 16;
        return static_cast<std::uint32_t>(o);
    };
    const int coarsest = static_cast<int>(c.rows.size()) - 1;
    for (int l = 0; l <= coarsest; ++l) {
        OnchipLevel<T> scratch{};
        OnchipLevel<T>& L = a != nullptr ? a->level[l] : scratch;
        const std::size_t span = c.span[l];
        if (l < coarsest) {
            // 16-byte words of a row: 6 (fine) or 8 couplings, diagonal, 1 / diagonal
            const std::size_t words = ((l == 0 ? 8 : 10) * sizeof(T) + 15) / 16;
            const bool held = l == 0 && onchip_held<T>(c.rows_per_thread);
            L.o_m = held ? 0u : take(words * span * 16);
            L.o_col = held ? 0u : take(span * (l == 0 ? 16 : 32));   // 16-bit places, or addresses
            L.o_agg = l == 0 ? 0u : take(span * 4);
            L.o_moff = take(std::size_t(c.span[l + 1]) * 4);
            L.o_mem = take(std::size_t(c.members[l]) * 4);
            L.o_r = take(span * sizeof(T));
            if (l == 0) o_r0 = L.o_r;
            L.o_y = take(span * sizeof(T));
        }
        if (l > 0) {
            L.o_x = take(span * sizeof(T));
            L.o_b = take((l == coarsest ? c.rows[l] : span) * sizeof(T));   // coarsest: every block has all of it
        }
    }
    const std::size_t dense = take(std::size_t(c.span[coarsest]) * c.rows[coarsest] * sizeof(T));
    const std::size_t phat = take(c.span[0] * sizeof(T));
    const std::size_t shat = take(c.span[0] * sizeof(T));
    // every 32-row partial of the planet, two quantities in T or one in FP64, two sets in turn;
    // the second lies where the fine residual does when it fits there (a V-cycle's phases all
    // lie between two reductions)
    const std::size_t part_bytes = std::size_t(ceil_div(c.rows[0], 256u)) * 8 * std::max(2 * sizeof(T), sizeof(double));
    const std::size_t part = take(part_bytes);
    std::size_t part2 = o_r0;
    if (part_bytes > c.span[0] * sizeof(T)) part2 = take(part_bytes);
    const std::size_t list = take(std::size_t(c.phases) * kOnchipPhaseBytes);
    if (a != nullptr) {
        a->o_list = static_cast<std::uint32_t>(list);
        a->o_dense = static_cast<std::uint32_t>(dense);
        a->o_phat = static_cast<std::uint32_t>(phat);
        a->o_shat = static_cast<std::uint32_t>(shat);
        a->o_part = static_cast<std::uint32_t>(part);
        a->o_part2 = static_cast<std::uint32_t>(part2);
    }
    return at;
}

// Spans and member bounds for a cluster size; false where a level cannot be held so.
bool spread(const Batch& b, OnchipClass& c, unsigned cluster) {
    const std::size_t depth = c.rows.size();
    c.cluster = cluster;
    c.phases = 1;
    for (std::size_t l = 0; l + 1 < depth; ++l) c.phases += b.smoother.pre_at(l) + b.smoother.post_at(l) + 2;
    if (c.phases > kOnchipMaxPhases) return false;
    c.span.assign(depth, 0);
    c.members.assign(depth, 0);
    for (std::size_t l = 0; l < depth; ++l) {
        const bool fine = l == 0;
        c.span[l] = span_of(c.rows[l], cluster, fine, l + 1 < depth && b.smoother.inner_at(l) > 1,
                            fine ? 1.0 : static_cast<double>(c.span[0]) / c.rows[0]);
        if (c.span[l] > kOnchipMaxSpan || (l + 1 < depth && b.levels[l].width > 8)) return false;
    }
    for (std::size_t l = 0; l + 1 < depth; ++l) {
        for (std::uint32_t i : c.planets)
            c.members[l] = std::max(c.members[l], members_most(b.planets[i]->hierarchy.levels[l], c.rows[l + 1], c.span[l + 1]));
    }
    return true;
}

// One fine-level phase of a block with `rows` rows, in us (measured shape of the phase: the
// barrier and gather latency, then the shared-memory reads of FP32 or the FP64 pipe).
template <typename T>
double phase_us(std::uint32_t rows) {
    return sizeof(T) == 4 ? 0.40 + 0.00035 * rows : 0.50 + 0.0023 * rows;
}

template <typename T>
void choose(const Batch& b, OnchipClass& c) {
    OnchipClass best = c;
    best.cluster = 0;
    const bool fits = c.rows.size() >= 2 && c.rows.size() <= static_cast<std::size_t>(kMaxLevels) &&
                      ceil_div(c.rows[0], kTileRows) <= kOnchipMaxTiles && b.levels[0].width == 6 &&
                      b.smoother.inner_at(0) == 1;
    for (unsigned cluster : {1u, 2u, 4u, 8u, 16u}) {
        if (!fits) break;
        OnchipClass t = c;
        if (!spread(b, t, cluster)) continue;
        // block-local sweeps: a block's threads hold all of its coarse rows, or whole tiles of them
        std::uint32_t local = 0;
        for (std::size_t l = 1; l + 1 < c.rows.size(); ++l)
            if (b.smoother.inner_at(l) > 1) local = std::max(local, t.span[l]);
        for (int r : {1, 2, 4, 7}) {
            t.rows_per_thread = r;
            t.threads = std::max(256u, ceil_div(ceil_div(t.span[0], static_cast<std::uint32_t>(r)), 32u) * 32u);
            if (local > t.threads) t.threads = ceil_div(t.threads, 256u) * 256u;
            if (t.threads <= kOnchipThreads) break;
        }
        if (t.threads > kOnchipThreads || !onchip_has<T>(t.rows_per_thread)) continue;
        t.shared_bytes = layout<T>(t, static_cast<OnchipArgs<T>*>(nullptr));
        const int active = onchip_active_clusters<T>(t.rows_per_thread, cluster, t.threads, t.shared_bytes);
        if (active <= 0) continue;
        const double waves = ceil_div(static_cast<std::uint32_t>(c.planets.size()), static_cast<std::uint32_t>(active));
        t.phase_us = waves * phase_us<T>(t.span[0]);
        if (best.cluster == 0 || t.phase_us < best.phase_us) best = t;
    }
    c = best;
}

}  // namespace

namespace {

template <typename T>
std::unique_ptr<OnchipPlan> make_plan(const Batch& b) {
    auto plan = std::make_unique<OnchipPlan>();
    std::map<std::vector<std::uint32_t>, OnchipClass> classes;
    for (std::uint32_t i = 0; i < b.instances; ++i) {
        std::vector<std::uint32_t> rows;
        for (const HostLevel& h : b.planets[i]->hierarchy.levels) rows.push_back(h.size);
        OnchipClass& c = classes[rows];
        c.rows = rows;
        c.planets.push_back(i);
    }
    // The batch goes on chip whole or not at all: with some planets left to the kernel schedule
    // its chain of launches costs the same, and the clusters take SMs from it (the 64-planet mix:
    // 11.9 ms a step without, 12.6 with its L4 and L5 planets on chip). Otherwise, whichever is
    // estimated to finish a phase of every planet first. On chip: the longest class, or all of
    // them sharing the SMs that clusters get. The kernel schedule: a launch's latency and its
    // rows' share of the GPU. Both lines are fitted to steps of 1 to 64 planets of levels 3 to 6
    // in either precision (e.g. 16 L5 planets: 1.7 against 2.3 ms FP32, 5.5 against 3.9 ms FP64).
    double longest = 0.0, shared = 0.0, rows = 0.0;
    bool fits = b.stream != nullptr;
    // the largest planets' launch first: its solves take longest
    for (auto it = classes.rbegin(); it != classes.rend() && fits; ++it) {
        OnchipClass c = it->second;
        choose<T>(b, c);
        fits = c.cluster != 0;
        longest = std::max(longest, c.phase_us);
        shared += c.planets.size() * c.cluster * phase_us<T>(c.span.empty() ? 0u : c.span[0]) / 120.0;
        rows += static_cast<double>(c.planets.size()) * c.rows[0];
        plan->classes.push_back(c);
    }
    const double launch = sizeof(T) == 4 ? 1.5 + 2.8e-6 * rows : 2.2 + 1.4e-5 * rows;
    if (!fits || std::max(longest, shared) > launch) plan->classes.clear();
    for (std::size_t k = 0; k < plan->classes.size(); ++k) {
        OnchipClass& c = plan->classes[k];
        if (plan->classes.size() == 1) break;   // every planet of the batch, in its order
        PSGB_CUDA(cudaMalloc(reinterpret_cast<void**>(&c.list), c.planets.size() * sizeof(std::uint32_t)));
        PSGB_CUDA(cudaMemcpy(c.list, c.planets.data(), c.planets.size() * sizeof(std::uint32_t), cudaMemcpyHostToDevice));
        if (k == 0) continue;
        // the other classes beside the first, on streams forked from the batch's
        int priority = 0;
        PSGB_CUDA(cudaStreamGetPriority(b.stream, &priority));
        cudaStream_t s = nullptr;
        cudaEvent_t e = nullptr;
        PSGB_CUDA(cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, priority));
        plan->streams.push_back(s);
        PSGB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        plan->done.push_back(e);
        if (plan->fork == nullptr) PSGB_CUDA(cudaEventCreateWithFlags(&plan->fork, cudaEventDisableTiming));
    }
    return plan;
}

template <typename T>
OnchipArgs<T> arguments(Batch& b, const OnchipClass& c) {
    OnchipArgs<T> a{};
    const int coarsest = static_cast<int>(c.rows.size()) - 1;
    for (int l = 0; l <= coarsest; ++l) {
        BatchLevel& L = b.levels[static_cast<std::size_t>(l)];
        const LevelView<T> v = Pick<T>::view(b, static_cast<std::size_t>(l));
        OnchipLevel<T>& o = a.level[l];
        o.col = L.col;
        o.vd = v.vd;
        o.inv = v.inv;
        o.agg = L.agg;
        o.moff = L.member_offset;
        o.member = L.member;
        o.pitch = L.rows;
        o.width = L.width;
        o.n = c.rows[static_cast<std::size_t>(l)];
        o.span = c.span[static_cast<std::size_t>(l)];
        o.pre = b.smoother.pre_at(l);
        o.post = b.smoother.post_at(l);
        o.inner = b.smoother.inner_at(l);
        o.starts_in_x = b.smoother.starts_in_x(l) ? 1 : 0;
        o.correction = v.correction;
    }
    a.coarsest = coarsest;
    a.cluster = static_cast<int>(c.cluster);
    a.planets = static_cast<std::uint32_t>(c.planets.size());
    a.instances = b.instances;
    a.list = c.list;
    a.tile_range = b.tile_range;
    a.dense_offset = b.dense.d_offset;
    a.dense_inv = Pick<T>::inv(b.dense);
    a.omega = static_cast<T>(b.smoother.omega);
    a.sc = b.scalars;
    layout<T>(c, &a);
    return a;
}

}  // namespace

template <typename T>
OnchipPlan& onchip_plan(Batch& b) {
    // the smoother decides how rows are shared out (block-local sweeps) and how many phases
    // a V-cycle has
    std::vector<int> key{static_cast<int>(sizeof(T))};
    for (std::size_t l = 0; l < b.levels.size(); ++l) {
        key.push_back(b.smoother.inner_at(l) > 1 ? 1 : 0);
        key.push_back(b.smoother.pre_at(l) + b.smoother.post_at(l));
    }
    return *b.onchip.of(key, [&] { return make_plan<T>(b); });
}

template <typename T>
void onchip_solve(Batch& b, OnchipPlan& plan, const SolveOptions& opt, const double* rhs, double* x, double inner_tol,
                  cudaStream_t st) {
    if (!plan.streams.empty()) PSGB_CUDA(cudaEventRecord(plan.fork, st));
    for (std::size_t k = 0; k < plan.classes.size(); ++k) {
        const OnchipClass& c = plan.classes[k];
        OnchipArgs<T> a = arguments<T>(b, c);
        a.fine_col = b.levels[0].col;
        a.fine_vd64 = b.levels[0].vd64;
        a.rhs64 = rhs;
        a.x64 = x;
        a.active = b.active_mask ? b.active : nullptr;
        a.tolerance = opt.tolerance;
        a.inner_tolerance = inner_tol;
        a.max_iterations = opt.max_iterations;
        a.max_refinements = opt.max_refinements;
        cudaStream_t s = k == 0 ? st : plan.streams[k - 1];
        if (k > 0) PSGB_CUDA(cudaStreamWaitEvent(s, plan.fork, 0));
        onchip_launch<T>(a, c.rows_per_thread, c.threads, c.shared_bytes, s);
        if (k > 0) PSGB_CUDA(cudaEventRecord(plan.done[k - 1], s));
    }
    for (cudaEvent_t e : plan.done) PSGB_CUDA(cudaStreamWaitEvent(st, e, 0));
}

template OnchipPlan& onchip_plan<float>(Batch&);
template OnchipPlan& onchip_plan<double>(Batch&);
template void onchip_solve<float>(Batch&, OnchipPlan&, const SolveOptions&, const double*, double*, double, cudaStream_t);
template void onchip_solve<double>(Batch&, OnchipPlan&, const SolveOptions&, const double*, double*, double, cudaStream_t);

}  // namespace psgb
