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

// The windows of a run of n_blocks dates (latest first), at most
// kContractMaxSlots (ext: kContractExtSlots) slots each: date 1, before any
// evolution, needs none.  w may be null; returns their number.
int contract_windows(int n_blocks, int stride, bool ext, ContractWindow* w);

// Bytes of the operand table of a run: scales, images, and the FP64 responses
// they are cut from.
size_t contract_table_bytes(int stride, int n_blocks, bool ext);

// Builds the table on the stream (two launches and one per window) from the loadings sv
// [kFactors][kMaxTenor] (sqrt(dt) sigma_k; the predictor-corrector's
// N-projected ones): the impulse responses of the Euler or the three-point
// step, sliced for the contraction.  same_shape: the table holds that of the same
// run shape and scheme with other loadings, whose walk weights serve again (one
// launch and 34 us less, whatever the shape: serial FP64 latency).
cudaError_t launch_contract_table(int nt, double c, int stride, int n_blocks, bool pc, bool ext, const double* sv,
                                  bool same_shape, void* table, cudaStream_t s);

// External normals [path][step][3] of n_blocks blocks as launch_path_contract takes
// them, into out (as many doubles as raw; the first block's place, whose steps no
// valuation draws upon, holds the paths' scales).  Two launches.
cudaError_t launch_contract_ext(const double* raw, int64_t n_paths, int n_blocks, int stride, void* out, cudaStream_t s);

// Partial-sum rows of a run: one per tile of kContractTile paths, four for a tile
// whose steps are split over the SMs (the tiles after the last whole wave, where
// that pays); the split tiles' sums take contract_sums_bytes (0: none).  Without
// room for them (split = false, sums = null) every tile runs whole.
int64_t contract_rows(int64_t n_paths, int n_blocks, int stride, int n_sms, bool split = true);
size_t contract_sums_bytes(int64_t n_paths, int n_blocks, int stride, int n_sms, bool ext);

// The valuation: per window a launch over the whole tiles and one over the split
// ones with their pricing (carry [2][n_paths] doubles when there is more than one
// window).  partials: contract_rows rows of n_blocks + 3 doubles.  normals:
// launch_contract_ext's, or null for the generator.
// result[kResErr] is set if a wait in the kernel ran out.
cudaError_t launch_path_contract(int nt, const PathParams<double>& P, const void* table, const void* normals,
                                 double* partials, double* estore, double* carry, longlong2* sums, double* result,
                                 int n_sms, cudaStream_t s, int* launches);

}  // namespace hjm
