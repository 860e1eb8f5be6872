// Which planets of a batch are solved on chip, and how (onchip.hpp has the kernels).
#pragma once

#include "planet.hpp"
#include "solver.hpp"

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

namespace psgb {

// The planets of one shape (the same rows on every level) and their launch.
struct OnchipClass {
    std::vector<std::uint32_t> planets;   // indices in the batch
    std::uint32_t* list = nullptr;        // the same on the device (null: every planet of the batch)
    unsigned cluster = 0, threads = 0;    // 0: not solved on chip
    int rows_per_thread = 0;
    int phases = 0;                       // of a V-cycle
    std::size_t shared_bytes = 0;
    std::vector<std::uint32_t> rows;      // per level
    std::vector<std::uint32_t> span;      // per level: rows a block holds
    std::vector<std::uint32_t> members;   // per level: member addresses a block holds at most
    double phase_us = 0.0;                // estimate of one fine-level phase, all waves
};

struct OnchipPlan {
    std::vector<OnchipClass> classes;     // empty: the batch is not solved on chip
    ~OnchipPlan();
    OnchipPlan() = default;
    OnchipPlan(const OnchipPlan&) = delete;
    OnchipPlan& operator=(const OnchipPlan&) = delete;
    std::vector<cudaStream_t> streams;    // one per class after the first
    std::vector<cudaEvent_t> done;
    cudaEvent_t fork = nullptr;
};

// The plan of a batch in precision T under its present smoother (the batch keeps its last few).
template <typename T>
OnchipPlan& onchip_plan(Batch& b);

// Launches every class of the plan on `st` (classes beside each other on streams forked
// from it); the solves of planets that are left out of the step write their idle state.
template <typename T>
void onchip_solve(Batch& b, OnchipPlan& plan, const SolveOptions& opt, const double* rhs, double* x, double inner_tol,
                  cudaStream_t st);

}  // namespace psgb
