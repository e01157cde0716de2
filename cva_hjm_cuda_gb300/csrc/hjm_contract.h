// hjm_contract.h -- the FP64 response form as an exact-sliced contraction on
// the tensor cores (hjm_contract.cu): host interface.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "hjm_device.cuh"

namespace hjm {

constexpr int kContractTile = 128;      // paths per tile: the rows of one tcgen05 M = 128 accumulator
constexpr int kContractMaxSlots = 32;   // dates a launch carries besides date 1
constexpr int kContractExtSlots = 24;   // ... with external normals (five slices of each in tensor memory)

// One launch: the dates [lo, hi], slot r holding date hi - r (dates from
// max(lo, 2)); npad accumulator columns per slice level (two per slot, padded
// to 16); chunks of 16 evolved steps; its operand image at `image` bytes into
// the table.
struct ContractWindow {
    int lo, hi, slots, npad, chunks;
    size_t image;
};

// How a run is laid out: dates a window carries at most, and whether the table
// holds all windows' images with the FP64 responses they are cut from, or one
// image at a time and no more (compact), rebuilt before each window's launch.
// In the order of preference; the first that there is room for is taken.  10y
// swap at dt = 0.01: 3.2 MB, 1.4 MB and 0.46 MB (and three windows instead of
// one); 25y: 14 MB, 4.7 MB and 1.2 MB.  A call with a new market, 5,000 paths: 10y
// 0.19, 0.29 and 0.54 ms (convected 1.98), 25y 0.37, 0.74 and 1.50 ms (4.30); 100,000
// paths: 25y 1.93, 2.33 and 4.95 ms (29.1).
struct ContractPlan {
    int slots;
    bool compact;
};
constexpr int kContractPlans = 3;
inline ContractPlan contract_plan(int i, bool ext)
{
    return {i < 2 ? (ext ? kContractExtSlots : kContractMaxSlots) : 8, i > 0};
}

// The windows of a run of n_blocks dates (latest first): date 1, before any
// evolution, needs no slot.  w may be null; returns their number.
int contract_windows(int n_blocks, int stride, ContractPlan plan, ContractWindow* w);

// Bytes of the operand table of a run
size_t contract_table_bytes(int stride, int n_blocks, ContractPlan plan);

// Builds the table of a plan that is not compact on the stream (two launches and one per window) from the loadings sv
// [kFactors][kMaxTenor] (sqrt(dt) sigma_k; the predictor-corrector's
// N-projected ones): the impulse responses of the Euler or the three-point
// step, sliced for the contraction.  same_shape: the table holds that of the same
// run shape and scheme with other loadings, whose walk weights serve again (one
// launch and 34 us less, whatever the shape: serial FP64 latency).
cudaError_t launch_contract_table(int nt, double c, int stride, int n_blocks, bool pc, ContractPlan plan,
                                  const double* sv, bool same_shape, void* table, cudaStream_t s);

// ... and that of one window of a compact plan (two launches), bit for bit the same
// image.
cudaError_t launch_contract_window(int nt, double c, int stride, int n_blocks, bool pc, const ContractWindow& W,
                                   const double* sv, void* table, cudaStream_t s);

// External normals [path][step][3] of n_blocks blocks as launch_path_contract takes
// them, into out (as many doubles as raw; the first block's place, whose steps no
// valuation draws upon, holds the paths' scales).  Two launches.
cudaError_t launch_contract_ext(const double* raw, int64_t n_paths, int n_blocks, int stride, void* out, cudaStream_t s);

// Partial-sum rows of a run: one per tile of kContractTile paths, four for a tile
// whose steps are split over the SMs (the tiles after the last whole wave, where
// that pays); the split tiles' sums take contract_sums_bytes (0: none).  Without
// room for them (split = false, sums = null) every tile runs whole.
int64_t contract_rows(int64_t n_paths, int n_blocks, int stride, int n_sms, bool split = true);
size_t contract_sums_bytes(int64_t n_paths, int n_blocks, int stride, int n_sms, ContractPlan plan);

// The valuation's window W (the latest first): a launch over the whole tiles and one
// over the split ones with their pricing (carry [2][n_paths] doubles when there is
// more than one window).  partials: contract_rows rows of n_blocks + 3 doubles.  normals:
// launch_contract_ext's, or null for the generator.
// result[kResErr] is set if a wait in the kernel ran out.
cudaError_t launch_path_contract(int nt, const PathParams<double>& P, const ContractWindow& W, const void* table,
                                 const void* normals, double* partials, double* estore, double* carry, longlong2* sums,
                                 double* result, int n_sms, cudaStream_t s, int* launches);

// All of it: the windows of the plan, a compact one's images between them (sv and c
// as launch_contract_table's; otherwise the table is there already).
cudaError_t launch_contract(int nt, double c, bool pc, const double* sv, const PathParams<double>& P, ContractPlan plan,
                            bool have_table, void* table, const void* normals, double* partials, double* estore,
                            double* carry, longlong2* sums, double* result, int n_sms, cudaStream_t s, int* launches);

}  // namespace hjm
