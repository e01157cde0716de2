// hjm_contract.cu -- the FP64 valuation's response form as a contraction on
// the tensor cores (tcgen05), for every volatility market, either time scheme
// and any number of dates.
//
// The pricing of date j reads the stochastic curve h_n = A h_{n-1} + S phi_n
// (A the upwind step, simulation_cpu.h:96-108, or the predictor-corrector's
// three-point step) only at tenor j: its value after the date's last step K_j
// and its sum over the steps, both linear in the path's normals,
//     h_K[j] = sum_{n,k} phi_{n,k} R_jk(K - n),  R_jk(l) = (A^l S_k)[j],
// and likewise with CR_jk(l) = sum_{r<=l} R_jk(r).  Over the paths of a tile
// that is a matrix product: normals [128][steps x 3] times responses
// [steps x 3][2 per date].
//
// FP64 accuracy from FP16 operands.  Each normal is cut into slices on fixed
// grids, phi = a0 + a1 2^-10 + a2 2^-20 + a3 2^-30: a0, a1, a2 multiples of
// 2^-7 (the remainder of one is scaled by 2^10 for the next, so |a1|, |a2| <=
// 4), a3 what is left, rounded to 11 bits (exact for |phi| >= 2^-15).  Each response, scaled per date by a power
// of two to at most 2^8, is cut likewise into b0 .. b3 (integers up to 2^9) and
// b4.  Every slice is exact in FP16, every product a_i b_j exact in FP32, and
// the products of one level s = i + j share one grid, so each level has an FP32
// accumulator of its own: over 12 chunks of 16 steps (576 products) levels 0
// and 1 stay below 2^21.1 grid units (rms, for the worst column), 7.5 standard
// deviations from the 2^24 up to which the accumulators add exactly; level 2's
// rounding lies 2^-40 below the curve and is met once in 10^5, levels 3 and 4's
// lies 2^-54 below.  Products of level 5 and above are dropped (2^-48).  After
// 12 chunks the five accumulators become one 64-bit integer, added to the date's
// running sum, and restart from zero.  Per-path exposures
// then lie 1e-14 of their scale from the oracle (the convected all-FP64 step:
// 5e-15; double-FP32 response sums on the FP32 pipe: 5e-14); with three slices
// fewer bits (grids 2^-12 apart, four levels) it was 6e-13.
//
// A caller's own normals (EXT) need not average out: equal or drifting ones add
// up coherently, 2^28 units at level 0 over a group.  So each path has a power of
// two of its own, which brings its normals below 8 (contract_ext_scale_kernel),
// a fifth slice for what FP32 does not hold, and levels 0 to 2 restart with every
// k-tile: 16 products of |a0| <= 2^10, |a1| <= 2^9, |a2| <= 576 with |b0| <= 2^8,
// |b1|, |b2| <= 2^9 add up to at most 2^23.9 units there, whatever the normals.
// Levels 3 and 4 go on over the group, so that the generator's own draws give its
// results bit for bit.  Constant normals of 3.65, 7.9 or 0.0039 then lie within
// 1e-13 of the exposures, where sums over whole groups lost up to 1e-7.
// Bound: the reads of levels 0 to 2 (three a chunk instead of one a group).
// 100,000 paths x 1,000 steps, 10y swap: 1.24 ms (2.28 ms for double-FP32 sums on
// the FP32 pipe; 13.4 ms with the slices cut in FP64).
//
// Roles of a CTA (one per SM, persistent over tiles of 128 paths):
//   warps 0-15   normals: Philox in registers, Box-Muller, slices; warp w holds
//                paths 32 (w % 4) + lane and half the steps of every second chunk
//                and stores the slices to the A operand in tensor memory
//                (counter-based draws: 16 warps share 128 paths);
//   warp 20      tcgen05.mma and commits, by one elected lane;
//   warp 21      B operand tiles by bulk copy (TMA) into shared memory;
//   warps 16-19  thread = path: accumulators to running sums, pricing of the
//                dates in FP64, exposures, partial sums, exposure rows.
// Accumulator columns are ordered [level][date slot]: the slices b0..b4 of a
// k-tile are consecutive rows of B, so a_s needs one instruction of (5 - s)
// npad columns (levels s..4): four instructions per 16-deep k-tile instead of
// fourteen.
//
// What bounds it: instruction issue in the sixteen normal warps, ~180 issue
// cycles per 32 path-steps (Philox's 18 wide multiplications take four each,
// the packed slicing operations two).  The matrix instructions of the 10y
// swap's 20 dates fill 1,008 of a chunk's ~2,900 cycles.  1,048,576 paths x
// 1,000 steps, FP64, 10y swap: 4.85 ms against 12.9 ms for the same sums in
// double-FP32 (a date costs no instructions per step any more); the 25y swap
// (50 dates) 17.7 ms against 92.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "hjm_contract.h"
#include "hjm_kernels.h"
#include "hjm_walk.cuh"

namespace hjm {

namespace {

constexpr int kChunk = 16;               // evolved steps per chunk: 48 = 3 x 16 contraction depth
constexpr int kFlush = 12;               // chunks per accumulator group
constexpr int kSlices = 4;                // of a normal
constexpr int kLevels = 5;                // of a response, and accumulators
constexpr int kProducers = 16;           // warps
constexpr int kMmaWarp = 20, kLoadWarp = 21;
constexpr int kThreads = 32 * 22;
constexpr int kAStages = 2, kBStages = 3;
constexpr int kTmemCols = 512;
// External normals take a fifth slice
__host__ __device__ constexpr int slices_of(bool ext) { return ext ? kSlices + 1 : kSlices; }
// 32-bit tensor-memory columns of a chunk's A slices; the A stages lie behind
// the accumulators
__host__ __device__ constexpr int a_stage_cols(bool ext) { return slices_of(ext) * 24; }
__host__ __device__ constexpr int a_col(bool ext) { return kTmemCols - kAStages * a_stage_cols(ext); }
static_assert(kLevels * 2 * kContractMaxSlots <= a_col(false) && kLevels * 2 * kContractExtSlots <= a_col(true),
              "accumulators and A stages share 512 columns");

// bytes of one chunk of the B image: 3 k-tiles of 16 x (kLevels npad) halves
__host__ __device__ constexpr size_t chunk_bytes(int npad) { return (size_t)3 * kLevels * npad * 32; }

constexpr size_t kScaleBytes = 2 * kMaxTenor * sizeof(double);  // then as many bytes of maxima

// A wait that runs out, after a second or two (every wait here is for work in
// flight, so it would be a fault of the program), ends the kernel with
// result[kResErr] set.
constexpr uint32_t kWaitNs = 1000000;
constexpr int kWaitTries = 2000;
constexpr int kSpinTries = 1 << 25;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// SLEEP: a try sleeps in hardware until the barrier turns, up to kWaitNs (it
// takes no issue slots, but wakes late); else it returns after the short
// interval of the hardware's own.
template <bool SLEEP>
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    if constexpr (SLEEP)
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(parity), "r"(kWaitNs)
            : "memory");
    else
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    return ok != 0;
}
// false when the wait ran out, here or in another warp (*abort_s)
template <bool SLEEP>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_s)
{
    if (mbar_try<SLEEP>(bar, parity)) return true;
    if constexpr (SLEEP) {
        for (int i = 0; i < kWaitTries; ++i) {
            if (*abort_s) return false;
            if (mbar_try<true>(bar, parity)) return true;
        }
    } else {
        for (int i = 0; i < kSpinTries; ++i) {
            if (mbar_try<false>(bar, parity)) return true;
            if ((i & 63) == 63 && *abort_s) return false;
        }
    }
    *abort_s = 1;
    return false;
}

__device__ __forceinline__ bool elect_one()
{
    uint32_t e;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(e));
    return e != 0;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D[128][n] (+)= A[128][16] (tensor memory) B[n][16]^T (shared memory), FP16 in, FP32 accumulators
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d),
        "r"(a), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// instruction descriptor: FP32 accumulators, FP16 operands, both K-major, M = 128
__device__ __forceinline__ uint32_t tc_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | (8u << 24); }
// shared-memory descriptor of a K-major, unswizzled tile: 8 x 16-byte core
// matrices, consecutive along n (128 bytes), `k_stride` bytes apart along k
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t addr, uint32_t k_stride)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(k_stride >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) |
           ((uint64_t)1 << 46);
}

__device__ __forceinline__ void tmem_st4(uint32_t addr, const uint32_t* r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3])
                 : "memory");
}
__device__ __forceinline__ void tmem_st2(uint32_t addr, const uint32_t* r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(r[0]), "r"(r[1])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float* r)
{
    uint32_t u[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(addr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) r[i] = __uint_as_float(u[i]);
}

constexpr float kGrid = 12582912.0f;   // 1.5 2^23: adding it rounds to integers
constexpr float kUnit = 128.0f;        // the first slice counts units of 2^-7
constexpr float kShift = 1024.0f;      // 2^10 between slices
constexpr int kTopBits = 8;            // the largest response of a date is scaled to at most 2^8

// The four slices of two normals, negated (pricing carries the sign back): -a_s
// from the constant minus the rounded sum, so that no instruction negates.
// Packed FP32 pairs throughout; every step is exact until the last conversion.
__device__ __forceinline__ void slice_pair(float2 v, uint32_t (&out)[kSlices])
{
    const float2 g = make_float2(kGrid, kGrid), m1 = make_float2(-1.0f, -1.0f), sh = make_float2(kShift, kShift),
                 un = make_float2(kUnit, kUnit);
    float2 na = __ffma2_rn(__ffma2_rn(v, un, g), m1, g);
    float2 d = __ffma2_rn(v, un, na);
#pragma unroll
    for (int s = 0; s < kSlices - 1; ++s) {
        const __half2 h = __floats2half2_rn(na.x, na.y);
        out[s] = *reinterpret_cast<const uint32_t*>(&h);
        if (s < kSlices - 2) {
            na = __ffma2_rn(__ffma2_rn(d, sh, g), m1, g);
            d = __ffma2_rn(d, sh, na);
        }
    }
    d = __fmul2_rn(d, make_float2(-kShift, -kShift));
    const __half2 h = __floats2half2_rn(d.x, d.y);
    out[kSlices - 1] = *reinterpret_cast<const uint32_t*>(&h);
}
// ... of two external normals hi + lo 2^-27 (contract_ext_kernel), with a fifth
// slice for what the fourth leaves.  lo joins at the third slice, whose units are
// 2^-27 (so |a2| <= 512 + 64); a normal that FP32 holds (lo = 0) gives the
// slices above, bit for bit.  In FP32: with FP64 operations, which share a pipe of
// 18 cycles an instruction, the slices of 100,000 paths x 950 steps took 13.4 ms.
__device__ __forceinline__ void slice_pair(float2 v, float2 lo, uint32_t (&out)[kSlices + 1])
{
    const float2 g = make_float2(kGrid, kGrid), m1 = make_float2(-1.0f, -1.0f), sh = make_float2(kShift, kShift),
                 un = make_float2(kUnit, kUnit);
    auto put = [&](int s, float2 x) {
        const __half2 h = __floats2half2_rn(x.x, x.y);
        out[s] = *reinterpret_cast<const uint32_t*>(&h);
        return h;
    };
    float2 na = __ffma2_rn(__ffma2_rn(v, un, g), m1, g);
    float2 d = __ffma2_rn(v, un, na);
    put(0, na);
    na = __ffma2_rn(__ffma2_rn(d, sh, g), m1, g);
    d = __ffma2_rn(d, sh, na);
    put(1, na);
    na = __ffma2_rn(__fadd2_rn(__ffma2_rn(d, sh, lo), g), m1, g);
    d = __fadd2_rn(__ffma2_rn(d, sh, na), lo);  // (both exact: multiples of lo's last bit below 2^8)
    put(2, na);
    d = __fmul2_rn(d, make_float2(-kShift, -kShift));
    const __half2 h = put(3, d);
    put(4, make_float2(lo.x == 0.0f ? 0.0f : (d.x - __low2float(h)) * kShift,
                       lo.y == 0.0f ? 0.0f : (d.y - __high2float(h)) * kShift));
}

// Philox4x32-10 of counter (step, 0, path): what depends on the path alone is
// formed once per tile (the first round's product of the path word and the
// second round's of the result), leaving 18 of the 20 multiplications per step.
struct PathDraw {
    uint32_t hi2, lo2;   // second round: high word (with its key) and low word of the path's product
    uint32_t y2;         // first round's low word with the second round's key
    uint32_t z1;         // path's high word with the first round's key
};
__device__ __forceinline__ PathDraw path_draw(uint64_t path, const uint32_t* rk0, const uint32_t* rk1)
{
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * (uint32_t)path;
    const uint64_t q0 = (uint64_t)0xD2511F53u * ((uint32_t)(p1 >> 32) ^ rk0[0]);
    PathDraw d;
    d.hi2 = (uint32_t)(q0 >> 32) ^ rk1[1];
    d.lo2 = (uint32_t)q0;
    d.y2 = (uint32_t)p1 ^ rk0[1];
    d.z1 = (uint32_t)(path >> 32) ^ rk1[0];
    return d;
}
__device__ __forceinline__ uint4 draw_words(const PathDraw& d, uint32_t step, const uint32_t* rk0, const uint32_t* rk1)
{
    const uint64_t p0 = (uint64_t)0xD2511F53u * step;
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * ((uint32_t)(p0 >> 32) ^ d.z1);
    uint4 c = make_uint4((uint32_t)(p1 >> 32) ^ d.y2, (uint32_t)p1, d.hi2 ^ (uint32_t)p0, d.lo2);
#pragma unroll
    for (int r = 2; r < 10; ++r) {
        const uint64_t a = (uint64_t)0xD2511F53u * c.x;
        const uint64_t b = (uint64_t)0xCD9E8D57u * c.z;
        c = make_uint4((uint32_t)(b >> 32) ^ c.y ^ rk0[r], (uint32_t)b, (uint32_t)(a >> 32) ^ c.w ^ rk1[r],
                       (uint32_t)a);
    }
    return c;
}

__device__ __forceinline__ float2 f2(float x, float y) { return make_float2(x, y); }

// A group's five level sums (integers in FP32; the last two together rounded to
// one) as one, in units of 2^-30: with the normals' 2^-7, 2^-37 of the response's
constexpr double kSumUnit = 0x1p-37;
__device__ __forceinline__ long long level_sum(float l0, float l1, float l2, float l3, float l4)
{
    return ((long long)__float2int_rn(l0) << 30) + ((long long)__float2int_rn(l1) << 20) +
           ((long long)__float2int_rn(l2) << 10) + (long long)__float2int_rn(fmaf(l4, 0x1p-10f, l3));
}
// ... as FP64: each half in the significand of a power of two (the conversion
// instruction is slow)
__device__ __forceinline__ double sum_value(long long v)
{
    const double hi = __hiloint2double(0x45300000, (int)((uint32_t)(v >> 32) ^ 0x80000000u));  // 2^84 + 2^63 + hi 2^32
    const double lo = __hiloint2double(0x43300000, (int)(uint32_t)v);                           // 2^52 + lo
    return (hi - 0x1.00000801p+84) + lo;
}

__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

}  // namespace

// Of a path with external normals: 2^e (NaN: a non-finite normal) and e
struct ExtRow {
    double scale;
    int64_t e;
};

// The launch's constants besides the path parameters.  Whole tiles [0, n_tiles)
// go to the CTAs in turn; in a split launch the accumulator groups of tiles
// [tile0, tile0 + n_tiles) are dealt to the CTAs in equal runs, and each CTA adds
// its groups' sums of a tile to sums [n_tiles][npad / 2][128], which
// contract_price_kernel then prices.
struct ContractParams {
    PathParams<double> P;
    ContractWindow W;
    int64_t tile0, n_tiles;
    longlong2* sums;  // null: whole tiles
};

// Chunks [begin, end) of a tile's accumulator groups
__host__ __device__ constexpr int group_chunk(int64_t group, int chunks)
{
    return group * kFlush < chunks ? (int)group * kFlush : chunks;
}
__host__ __device__ constexpr int tile_groups(int chunks) { return (chunks + kFlush - 1) / kFlush; }

// What a CTA works through: chunk c0 of tile first on, `chunks` chunks, tiles
// `step` apart
struct ContractRun {
    int64_t first, step, chunks;
    int c0;
};
__device__ __forceinline__ ContractRun contract_run(const ContractParams& Q)
{
    const int NC = Q.W.chunks;
    ContractRun r;
    if (!Q.sums) {
        r.first = blockIdx.x;
        r.step = gridDim.x;
        r.chunks = (blockIdx.x < Q.n_tiles ? (Q.n_tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0) * NC;
        r.c0 = 0;
        return r;
    }
    const int G = tile_groups(NC);
    const int64_t units = Q.n_tiles * G, u0 = units * blockIdx.x / gridDim.x, u1 = units * (blockIdx.x + 1) / gridDim.x;
    r.first = Q.tile0 + u0 / G;
    r.step = 1;
    r.c0 = group_chunk(u0 % G, NC);
    r.chunks = (u1 / G - u0 / G) * NC + group_chunk(u1 % G, NC) - r.c0;
    return r;
}

// The cash flow of date i from its running sums v (times the scales sx, sa; the
// slices are negated)
__device__ __forceinline__ double contract_cash_flow(const PathParams<double>& P, int i, longlong2 v, double sx,
                                                     double sa)
{
    const double x = fma(-sum_value(v.x), sx, P.psamp[i]), a = fma(-sum_value(v.y), sa, P.psum[i]);
    const double D = exp(-a * P.dt);
    const double Lb = P.m * (exp(x * P.inv_m) - 1.0);
    return D * (P.payA[i] * Lb - P.payB[i]);
}

template <bool EXT>
__global__ void __launch_bounds__(kThreads, 1)
    path_kernel_contract(const __grid_constant__ ContractParams Q, const unsigned char* __restrict__ table,
                         const float2* __restrict__ ext, const ExtRow* __restrict__ ext_row,
                         double* __restrict__ partials, double* __restrict__ estore, double* __restrict__ carry,
                         double* __restrict__ result)
{
    constexpr int kSl = slices_of(EXT), kAStageCols = a_stage_cols(EXT), kACol = a_col(EXT);
    const PathParams<double>& P = Q.P;
    const ContractWindow& W = Q.W;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[2 * kAStages + 2 * kBStages + 3];
    __shared__ uint32_t tmem_s;
    __shared__ int abort_flag, stop_flag;
    __shared__ double red_s[8];
    volatile int* abort_s = &abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lo = W.lo, hi = W.hi, npad = W.npad, NC = W.chunks;
    const size_t cb = chunk_bytes(npad);
    unsigned char* b_s = smem;                                                       // [kBStages][cb]
    longlong2* run_s = reinterpret_cast<longlong2*>(smem + kBStages * cb);            // [npad / 2][128] {value, sum}
    double* cf_s = reinterpret_cast<double*>(run_s + (size_t)(npad / 2) * kContractTile);  // [hi - lo + 3][128]

    const uint32_t a_full = smem_u32(bars), a_empty = a_full + 8 * kAStages, b_full = a_empty + 8 * kAStages,
                   b_empty = b_full + 8 * kBStages, d_full = b_empty + 8 * kBStages, d_empty = d_full + 8, drain = d_empty + 8;
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)),
                     "n"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int i = 0; i < kAStages; ++i) {
            mbar_init(a_full + 8 * i, kProducers / kAStages);
            mbar_init(a_empty + 8 * i, 1);
        }
        for (int i = 0; i < kBStages; ++i) {
            mbar_init(b_full + 8 * i, 1);
            mbar_init(b_empty + 8 * i, 1);
        }
        mbar_init(d_full, 1);
        mbar_init(d_empty, 4);
        mbar_init(drain, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_s;
    const ContractRun run = contract_run(Q);

    if (warp < kProducers) {
        // ---- normals -> A slices in tensor memory.  Two groups of 8 warps take
        // the chunks of this CTA's sequence in turn, one A stage each, so that
        // one group's waits and stores lie under the other's arithmetic; a warp
        // has 8 steps of its chunk, in two halves of 4
        const int q = warp & 3, sub = (warp >> 2) & 1, st = warp >> 3;
        const uint32_t a_addr = tmem + ((uint32_t)(32 * q) << 16) + kACol + st * kAStageCols + 12 * sub;
        const int n_last = P.n_blocks * P.stride - 1;
        uint32_t ph = 1;
        bool ok = true;
        int c = run.c0 + st;
        int64_t tile = run.first, left = (run.chunks - st + kAStages - 1) / kAStages;  // this group's chunks
        while (ok && left > 0) {
            for (; c >= NC; c -= NC) tile += run.step;
            const int64_t lp = tile * kContractTile + 32 * q + lane;
            const PathDraw pd = path_draw(P.path_offset + (uint64_t)lp, P.rk0, P.rk1);
            const int64_t lpc = lp < P.n_paths ? lp : 0;
            for (; c < NC && left > 0; c += kAStages, ph ^= 1u, --left) {
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    const int n0 = P.stride + kChunk * c + 8 * sub + 4 * half;
                    // value 3 i + k: step n0 + i, factor k; pairs of values are one column
                    uint32_t w[kSl][6];
                    if constexpr (EXT) {
                        float2 z[12];
                        const size_t np = (size_t)P.n_paths;
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int k = 0; k < 3; ++k)
                                z[3 * i + k] = __ldg(ext + (size_t)min(n0 + i, n_last) * 3 * np + k * np + lpc);
#pragma unroll
                        for (int u = 0; u < 6; ++u) {
                            uint32_t o[kSl];
                            slice_pair(f2(z[2 * u].x, z[2 * u + 1].x), f2(z[2 * u].y, z[2 * u + 1].y), o);
#pragma unroll
                            for (int s = 0; s < kSl; ++s) w[s][u] = o[s];
                        }
                    } else {
                        float z[12];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint4 u = draw_words(pd, (uint32_t)(n0 + i), P.rk0, P.rk1);
                            normals3(u, z[3 * i], z[3 * i + 1], z[3 * i + 2]);
                        }
#pragma unroll
                        for (int u = 0; u < 6; ++u) {
                            uint32_t o[kSlices];
                            slice_pair(f2(z[2 * u], z[2 * u + 1]), o);
#pragma unroll
                            for (int s = 0; s < kSlices; ++s) w[s][u] = o[s];
                        }
                    }
                    if (half == 0) {
                        ok = mbar_wait<true>(a_empty + 8 * st, ph, abort_s);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        tc_fence_after();
                    }
#pragma unroll
                    for (int s = 0; s < kSl; ++s) {
                        const uint32_t a = a_addr + 24 * s + 6 * half;
                        tmem_st4(a, &w[s][0]);
                        tmem_st2(a + 4, &w[s][4]);
                    }
                }
                if (!ok) break;
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(a_full + 8 * st);
            }
        }
    } else if (warp == kMmaWarp) {
        // ---- the matrix instructions: the warp waits as one, one elected lane issues
        const bool leader = elect_one();
        const uint32_t bs = smem_u32(b_s);
        const int64_t total = run.chunks;
        bool ok = true;
        // a_s times the response slices b_0 .. b_{levels - 1 - s} gives the
        // levels s .. 4; beyond 256 columns b_4 takes an instruction of its own
        const bool split = kLevels * npad > 256;
        uint32_t idesc[kSlices];  // (EXT: of 5 - s columns' worth, as the generator's)
#pragma unroll
        for (int s = 0; s < kSlices; ++s) idesc[s] = tc_idesc((kLevels - s - (s == 0 && split)) * npad);
        const uint32_t idesc1 = tc_idesc(npad);
        const uint64_t desc0 = tc_smem_desc(bs, kLevels * npad * 16);
        const uint32_t kt_step = (uint32_t)(kLevels * npad * 32) >> 4, stage_step = (uint32_t)cb >> 4;
        // The loop is unrolled over the six combinations of an A and a B stage, so
        // that their addresses and parities are constants or warp-uniform: the
        // issuing warp shares one scheduler with four normal warps, which its
        // instructions delay (and the barriers the other schedulers with them).
        int c = run.c0, fl = 0;  // chunk of the tile, of the accumulator group
        uint32_t ph = 0, d_ph = 1;
        int64_t g = 0;
        auto chunk = [&](auto iv) {
            constexpr int i = decltype(iv)::value, st = i % kAStages, sb = i % kBStages;
            const bool first = fl == 0;
            const bool last = fl == kFlush - 1 || c == NC - 1;
            ok = mbar_wait<false>(a_full + 8 * st, ph ^ (uint32_t)(i / kAStages & 1), abort_s) &&
                 mbar_wait<false>(b_full + 8 * sb, (uint32_t)(i / kBStages & 1), abort_s) &&
                 (EXT || !first || mbar_wait<false>(d_empty, d_ph, abort_s));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            tc_fence_after();
            if constexpr (EXT) {
                const uint64_t bd0 = desc0 + (uint64_t)(sb * stage_step);
                const uint32_t a0 = tmem + kACol + st * kAStageCols;
                const uint32_t two = idesc[3], three = idesc[2];
                for (int kt = 0; kt < 3; ++kt) {
                    const uint64_t bd = bd0 + (uint64_t)(kt * kt_step);
                    const uint32_t a = a0 + 8 * kt;
                    // levels 3 and 4: a_s times b_{3-s}, b_{4-s}
                    auto low_levels = [&](uint32_t add) {
#pragma unroll
                        for (int s = 0; s < kSlices; ++s)
                            tc_mma(tmem + 3 * npad, a + 24 * s, bd + (uint64_t)((3 - s) * npad), two, s ? 1u : add);
                        tc_mma(tmem + 4 * npad, a + 24 * kSlices, bd, idesc1, 1);
                    };
                    const bool fresh = first && kt == 0;
                    if (leader && !fresh) low_levels(1);  // (the last k-tile's reader leaves these two alone)
                    ok = __all_sync(0xffffffffu, mbar_wait<false>(d_empty, d_ph, abort_s));
                    if (!ok) return;
                    d_ph ^= 1u;
                    tc_fence_after();
                    if (leader) {
                        if (fresh) low_levels(0);
                        tc_mma(tmem, a, bd, three, 0);
                        tc_mma(tmem + npad, a + 24, bd, two, 1);
                        tc_mma(tmem + 2 * npad, a + 48, bd, idesc1, 1);
                        tc_commit(d_full);
                    }
                }
                if (leader) {
                    tc_commit(a_empty + 8 * st);
                    tc_commit(b_empty + 8 * sb);
                }
            } else if (leader) {
                const uint64_t bd0 = desc0 + (uint64_t)(sb * stage_step);
                const uint32_t a0 = tmem + kACol + st * kAStageCols;
#pragma unroll
                for (int kt = 0; kt < 3; ++kt) {
                    const uint64_t bd = bd0 + (uint64_t)(kt * kt_step);
                    const uint32_t a = a0 + 8 * kt;
                    const uint32_t add = !(first && kt == 0);
                    tc_mma(tmem, a, bd, idesc[0], add);
                    if (split)
                        tc_mma(tmem + (kLevels - 1) * npad, a, bd + (uint64_t)((kLevels - 1) * npad), idesc1, add);
#pragma unroll
                    for (int s = 1; s < kSlices; ++s) tc_mma(tmem + s * npad, a + 24 * s, bd, idesc[s], 1);
                }
                tc_commit(a_empty + 8 * st);
                tc_commit(b_empty + 8 * sb);
                if (last) tc_commit(d_full);
            }
            if (!EXT && first) d_ph ^= 1u;
            ++g;
            if (++fl == kFlush || c == NC - 1) fl = 0;
            if (++c == NC) c = 0;
        };
        static_assert(kAStages == 2 && kBStages == 3, "the unrolled period is six chunks");
        while (ok && g < total) {
            chunk(std::integral_constant<int, 0>{});
            if (ok && g < total) chunk(std::integral_constant<int, 1>{});
            if (ok && g < total) chunk(std::integral_constant<int, 2>{});
            if (ok && g < total) chunk(std::integral_constant<int, 3>{});
            if (ok && g < total) chunk(std::integral_constant<int, 4>{});
            if (ok && g < total) chunk(std::integral_constant<int, 5>{});
            ph ^= 1u;
        }
        if (!ok) {  // matrix instructions in flight end before the CTA does
            if (leader) tc_commit(drain);
            for (int i = 0; i < kWaitTries && !mbar_try<true>(drain, 0); ++i) {
            }
        }
        __syncwarp();
    } else if (warp == kLoadWarp) {
        // ---- B operand tiles by bulk copy
        if (lane == 0) {
            const uint32_t bs = smem_u32(b_s);
            const int64_t total = run.chunks;
            const unsigned char* image = table + W.image;
            int c = run.c0, st = 0;
            uint32_t ph = 1;
            int64_t g = 0;
            for (; g < total; ++g) {
                if (!mbar_wait<true>(b_empty + 8 * st, ph, abort_s)) break;
                const uint32_t bar = b_full + 8 * st;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)cb)
                             : "memory");
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        bs + (uint32_t)(st * cb)),
                    "l"(image + (size_t)c * cb), "r"((uint32_t)cb), "r"(bar)
                    : "memory");
                if (++c == NC) c = 0;
                if (++st == kBStages) {
                    st = 0;
                    ph ^= 1u;
                }
            }
            // copies in flight land before the CTA ends (all have, unless it gave up)
            for (int64_t i = g > kBStages ? g - kBStages : 0; i < g; ++i)
                for (int w = 0; w < kWaitTries && !mbar_try<true>(b_full + 8 * (int)(i % kBStages),
                                                                  (uint32_t)((i / kBStages) & 1)); ++w) {
                }
        }
        __syncwarp();
    } else {
        // ---- running sums, pricing, exposures: thread = path
        const int q = warp & 3, p = 32 * q + lane;
        const uint32_t d_addr = tmem + ((uint32_t)(32 * q) << 16);
        const double* scale = reinterpret_cast<const double*>(table);  // [date][2]
        const bool top = hi == P.n_blocks, bottom = lo == 1;
        const int B = P.n_blocks, R = B + 3;
        const int first_date = lo > 2 ? lo : 2;  // date 1 precedes any evolution
        double* e_s = cf_s + kContractTile;  // exposure row of date j: j - lo + 1 (the cash-flow row of date j + 1)
        int64_t grp = 0;
        // waits for the accumulators and adds them to the running sums of the live
        // slots (fresh: the first of them; low: levels 3 and 4 too), four slots at a
        // time, padding included (its columns are zero); false if the wait ran out
        auto drain = [&](bool fresh, auto low, int live) {
            const bool ok = mbar_wait<true>(d_full, (uint32_t)(grp & 1), abort_s);
            if (!__all_sync(0xffffffffu, ok)) return false;
            ++grp;
            tc_fence_after();
            for (int r0 = 0; r0 < live; r0 += 4) {
                float acc[kLevels][8];
#pragma unroll
                for (int s = 0; s < kLevels; ++s)
                    if (s < 3 || decltype(low)::value)
                        tmem_ld8(d_addr + s * npad + 2 * r0, acc[s]);
                    else
                        for (int i = 0; i < 8; ++i) acc[s][i] = 0.0f;
                longlong2 cell[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    cell[u] = fresh ? make_longlong2(0, 0) : run_s[(size_t)(r0 + u) * kContractTile + p];
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (r0 + 4 >= live) {  // the accumulators are read: the next group may start
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d_empty);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    cell[u].x += level_sum(acc[0][2 * u], acc[1][2 * u], acc[2][2 * u], acc[3][2 * u], acc[4][2 * u]);
                    cell[u].y += level_sum(acc[0][2 * u + 1], acc[1][2 * u + 1], acc[2][2 * u + 1], acc[3][2 * u + 1],
                                           acc[4][2 * u + 1]);
                    run_s[(size_t)(r0 + u) * kContractTile + p] = cell[u];
                }
            }
            return true;
        };
        // the accumulators of chunks [from, to), one group's: at once, or k-tile by k-tile
        auto drain_group = [&](int from, int to, bool fresh, int live) {
            if constexpr (EXT) {
                for (int i = 3 * (to - from) - 1; i > 0; --i, fresh = false)
                    if (!drain(fresh, std::false_type(), live)) return false;
            }
            return drain(fresh, std::true_type(), live);
        };
        if (Q.sums) {  // ---- split tiles: this CTA's groups of each, to the tile's sums
            int64_t left = run.chunks, tile = run.first;
            for (int c = run.c0; left > 0; c = 0, ++tile) {
                const int end = (int)min((int64_t)NC, c + left);
                left -= end - c;
                int next = first_date;
                auto skip_to = [&](int chunk) {  // dates sampled before the chunk
                    while ((next - 1) * P.stride <= kChunk * chunk) ++next;
                };
                skip_to(c);
                const int live0 = hi - next + 1;
                bool ok = true;
                for (int b = c; b < end && ok; b += kFlush) {
                    skip_to(b);
                    ok = drain_group(b, min(b + kFlush, end), b == c, hi - next + 1);
                }
                if (!ok) break;
                unsigned long long* to = reinterpret_cast<unsigned long long*>(
                    Q.sums + (size_t)(tile - Q.tile0) * (npad / 2) * kContractTile);
                for (int r = 0; r < live0; ++r) {
                    const size_t at = (size_t)r * kContractTile + p;
                    const longlong2 v = run_s[at];
                    atomicAdd(to + 2 * at, (unsigned long long)v.x);
                    atomicAdd(to + 2 * at + 1, (unsigned long long)v.y);
                }
            }
        } else {
            for (int64_t tile = blockIdx.x; tile < Q.n_tiles; tile += gridDim.x) {
                const int64_t base = tile * kContractTile, lp = base + p;
                const bool active = lp < P.n_paths;
                double rs = 1.0;
                if constexpr (EXT) rs = ext_row[active ? lp : 0].scale;
                auto price = [&](int i) {
                    double sx = 0.0, sa = 0.0;
                    longlong2 v = make_longlong2(0, 0);
                    if (i >= 2) {
                        v = run_s[(size_t)(hi - i) * kContractTile + p];
                        sx = __ldg(scale + 2 * i);
                        sa = __ldg(scale + 2 * i + 1);
                        if constexpr (EXT) {
                            sx *= rs;
                            sa *= rs;
                        }
                    }
                    cf_s[(size_t)(i - lo + 1) * kContractTile + p] = contract_cash_flow(P, i, v, sx, sa);
                };
                if (bottom) price(1);
                int next = first_date;  // the earliest date not priced yet
                for (int c = 0; c < NC; c += kFlush) {
                    if (!drain_group(c, min(c + kFlush, NC), c == 0, hi - next + 1)) break;
                    // the dates whose last step this group held
                    const int done = kChunk * min(c + kFlush, NC);
                    for (; next <= hi && (next - 1) * P.stride <= done; ++next) price(next);
                }
                // (a wait that ran out ends all four warps at the same tile)
                if (p == 0) stop_flag = *abort_s;
                epilogue_sync();
                if (stop_flag) break;
                // exposures E_j = max(sum_{i > j} cf_i, 0) of dates lo - 1 .. hi - 1
                // (and E_B = 0 for the latest window), the later dates' cash flows in carry
                const int j0 = lo - 1, j1 = top ? B : hi - 1;
                double v = 0.0, cva_c = 0.0;
                if (!top && active) {
                    v = carry[lp];
                    cva_c = carry[P.n_paths + lp];
                }
                if (top) e_s[(size_t)(B - lo + 1) * kContractTile + p] = 0.0;
                for (int j = hi - 1; j >= lo - 1; --j) {
                    v += cf_s[(size_t)(j - lo + 2) * kContractTile + p];
                    double e = (v > 0.0) ? v : 0.0;
                    if (!active) e = 0.0;
                    e_s[(size_t)(j - lo + 1) * kContractTile + p] = e;
                    cva_c = fma(P.cvaw[j], e, cva_c);
                }
                if (!bottom && active) {
                    carry[lp] = v;
                    carry[P.n_paths + lp] = cva_c;
                }
                if (bottom) {
                    const double s1 = warp_sum(cva_c), s2 = warp_sum(cva_c * cva_c);
                    if (lane == 0) {
                        red_s[q] = s1;
                        red_s[4 + q] = s2;
                    }
                }
                if (P.store_exposures) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                epilogue_sync();
                for (int j = j0 + q; j <= j1; j += 4) {
                    double sum = 0.0;
#pragma unroll
                    for (int u = 0; u < 4; ++u) sum += e_s[(size_t)(j - lo + 1) * kContractTile + lane + 32 * u];
                    sum = warp_sum(sum);
                    if (lane == 0) partials[(size_t)tile * R + j] = sum;
                }
                if (p == 127 && bottom) {
                    partials[(size_t)tile * R + B + 1] = (red_s[0] + red_s[1]) + (red_s[2] + red_s[3]);
                    partials[(size_t)tile * R + B + 2] = (red_s[4] + red_s[5]) + (red_s[6] + red_s[7]);
                }
                if (p == 0 && P.store_exposures) {
                    const int64_t cnt = (P.n_paths - base < kContractTile) ? (P.n_paths - base) : kContractTile;
                    const uint32_t bytes = (uint32_t)(((cnt + 1) / 2) * 2 * sizeof(double));
                    for (int j = j0; j <= j1; ++j) {
                        double* dst = estore + (size_t)j * (size_t)P.ld + (size_t)base;
                        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                                     "r"(smem_u32(e_s + (size_t)(j - lo + 1) * kContractTile)), "r"(bytes)
                                     : "memory");
                    }
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                }
                epilogue_sync();  // (the rows are read: the next tile may price)
            }
        }
        if (p == 0 && P.store_exposures) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid == 0 && abort_flag) result[kResErr] = 1.0;
    if (warp == kMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTmemCols) : "memory");
}

// Prices the split tiles from their sums: a CTA takes 32 paths (lane = path), its
// warps every kPriceWarps-th date: a date is ~45 FP64 instructions in a chain,
// bound by their latency until many warps share an SM's pipe (18 cycles an
// instruction).  A 128-path call of the 10y run 125 -> 117 us against four
// warps; sixteen the same.  Partial-sum rows and exposure rows as the path
// kernel's, one row per 32 paths from row0.
constexpr int kPriceWarps = 8;
template <bool EXT>
__global__ void __launch_bounds__(32 * kPriceWarps)
    contract_price_kernel(const __grid_constant__ ContractParams Q, const double* __restrict__ scale,
                          const ExtRow* __restrict__ ext_row, int64_t row0, double* __restrict__ partials,
                          double* __restrict__ estore, double* __restrict__ carry)
{
    const PathParams<double>& P = Q.P;
    const int lo = Q.W.lo, hi = Q.W.hi, B = P.n_blocks, R = B + 3;
    const bool top = hi == B, bottom = lo == 1;
    __shared__ double cf_s[kContractMaxSlots + 4][32];  // row i - lo + 1: date i, then its exposures one row up
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int in_tile = (int)(blockIdx.x & 3) * 32 + lane;
    const int64_t tile = Q.tile0 + blockIdx.x / 4, lp = tile * kContractTile + in_tile;
    const bool active = lp < P.n_paths;
    const longlong2* sums = Q.sums + (size_t)(blockIdx.x / 4) * (Q.W.npad / 2) * kContractTile + in_tile;
    double rs = 1.0;
    if constexpr (EXT) rs = ext_row[active ? lp : 0].scale;
    for (int i = lo + warp; i <= hi; i += kPriceWarps) {
        double sx = 0.0, sa = 0.0;
        longlong2 v = make_longlong2(0, 0);
        if (i >= 2) {
            v = sums[(size_t)(hi - i) * kContractTile];
            sx = __ldg(scale + 2 * i);
            sa = __ldg(scale + 2 * i + 1);
            if constexpr (EXT) {
                sx *= rs;
                sa *= rs;
            }
        }
        cf_s[i - lo + 1][lane] = contract_cash_flow(P, i, v, sx, sa);
    }
    __syncthreads();
    double(*e_s)[32] = cf_s + 1;  // exposure row of date j: j - lo + 1
    if (warp == 0) {
        double v = 0.0, cva_c = 0.0;
        if (!top && active) {
            v = carry[lp];
            cva_c = carry[P.n_paths + lp];
        }
        if (top) e_s[B - lo + 1][lane] = 0.0;
        for (int j = hi - 1; j >= lo - 1; --j) {
            v += cf_s[j - lo + 2][lane];
            double e = (v > 0.0) ? v : 0.0;
            if (!active) e = 0.0;
            e_s[j - lo + 1][lane] = e;
            cva_c = fma(P.cvaw[j], e, cva_c);
        }
        if (!bottom && active) {
            carry[lp] = v;
            carry[P.n_paths + lp] = cva_c;
        }
        if (bottom) {
            const double s1 = warp_sum(cva_c), s2 = warp_sum(cva_c * cva_c);
            if (lane == 0) {
                partials[(size_t)(row0 + blockIdx.x) * R + B + 1] = s1;
                partials[(size_t)(row0 + blockIdx.x) * R + B + 2] = s2;
            }
        }
    }
    __syncthreads();
    const int j1 = top ? B : hi - 1;
    for (int j = lo - 1 + warp; j <= j1; j += kPriceWarps) {
        const double e = e_s[j - lo + 1][lane];
        const double sum = warp_sum(e);
        if (lane == 0) partials[(size_t)(row0 + blockIdx.x) * R + j] = sum;
        if (P.store_exposures && active) estore[(size_t)j * (size_t)P.ld + (size_t)lp] = e;
    }
}

// ---------------------------------------------------------------------------
// The operand table
// ---------------------------------------------------------------------------
namespace {

struct ContractLoadings {
    double sv[kFactors][kMaxTenor];
};

// The power of two that maps a date's largest response (finite) into [2^7, 2^8), as
// a multiplier back (responses below 1e-280 count as zero), by its exponent's bits:
// FP64 instructions are what the image kernel waits for (a division and the
// exponent functions per element: 30 us for 32 dates of the 25y run against 19).
constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;
__device__ __forceinline__ int contract_exponent(unsigned long long top)
{
    const bool in = top > (unsigned long long)__double_as_longlong(1e-280) &&
                    top < kInfBits;
    return in ? (int)(top >> 52) - 1022 - kTopBits : 0;
}
__device__ __forceinline__ double power_of_two(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// One lag's walk (hjm_walk.cuh): {f_m(i), G_m(i) = sum_{r <= m} f_r(i)}, i = 0, 1, ..
// f_m are the coefficients of p^m, p = a0 + a1 z + a2 z^2: from p (p^m)' = m p' p^m,
//     (i + 1) a0 f(i+1) = (m - i) a1 f(i) + (2 m - i + 1) a2 f(i-1),
// and G those of (p^{m+1} - 1) / (p - 1), whose partial sums telescope:
//     (a1 + a2) G(i) + a2 G(i-1) = 1 - f_{m+1}(0) - .. - f_{m+1}(i),
// so a rounding fades by a2 / (a1 + a2) a step.
struct LagWalk {
    double md, f, f1, h, h1, g, tail;
    __device__ __forceinline__ LagWalk(const WalkParams& K, int m)
        : md(m), f(walk_power(K, md)), f1(0.0), h(walk_power(K, md + 1.0)), h1(0.0), g(0.0), tail(1.0)
    {
    }
    __device__ __forceinline__ double2 next(const WalkParams& K, int i)
    {
        tail -= h;
        g = fma(tail, K.inv, -(K.b2 * g));
        const double2 out = make_double2(f, g);
        const double di = i;
        const double fn = fma((md - di) * K.a1, f, (2.0 * md - di + 1.0) * K.a2 * f1) * K.rcp[i];
        const double hn = fma((md + 1.0 - di) * K.a1, h, (2.0 * md - di + 3.0) * K.a2 * h1) * K.rcp[i];
        f1 = f;
        f = fn;
        h1 = h;
        h = hn;
        return out;
    }
};

// weights[i M + m], i < n: the walks of all lags, a thread each
__global__ void contract_weights_kernel(const __grid_constant__ WalkParams K, int M, int n, double2* __restrict__ weights)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    LagWalk walk(K, m);
    for (int i = 0; i < n; ++i) weights[(size_t)i * M + m] = walk.next(K, i);
}

// A date's responses to the three factors and their running sums at lag m, the
// lags of a CTA of 128 together: v, w from the walk's weights at(i), i = 0, 1, ..
struct DateResponse {
    double v[kFactors], w[kFactors];
    template <typename At>
    __device__ __forceinline__ DateResponse(const ContractLoadings& S, const double (&dev_s)[kFactors][kMaxTenor], int L,
                                            double c, int j, int m, int m0, int lags, At at)
    {
        const double md = m;
#pragma unroll
        for (int k = 0; k < kFactors; ++k) {
            const double d = S.sv[k][L] - S.sv[k][L - 1], x = fma((double)(j - L), d, S.sv[k][L]);
            v[k] = fma(md * c, d, x);
            w[k] = (md + 1.0) * fma(0.5 * md * c, d, x);
        }
        // the walk of this block's lags ends within ten standard deviations and a
        // dozen tenors of its mean (1e-22 beyond)
        const double mean = c * (double)min(m0 + (int)blockDim.x, lags);
        const int n = min(L - 1 - j, (int)(mean + 10.0 * sqrt(mean)) + 12);
        for (int i = 0; i < n; ++i) {
            const double2 p = at(i);
#pragma unroll
            for (int k = 0; k < kFactors; ++k) {
                const double x = dev_s[k][j + i];
                v[k] = fma(p.x, x, v[k]);
                w[k] = fma(p.y, x, w[k]);
            }
        }
    }
    // its largest magnitudes into best, the CTA's into top[2 j + {0 value, 1 sum}]
    __device__ __forceinline__ void largest(double (&best)[2]) const
    {
#pragma unroll
        for (int k = 0; k < kFactors; ++k) {
            best[0] = isfinite(v[k]) ? fmax(best[0], fabs(v[k])) : __longlong_as_double(kInfBits);
            best[1] = isfinite(w[k]) ? fmax(best[1], fabs(w[k])) : __longlong_as_double(kInfBits);
        }
    }
};
// The loadings' deviations from the line through the last two tenors
__device__ __forceinline__ void load_deviations(const ContractLoadings& S, int nt, double (&dev_s)[kFactors][kMaxTenor])
{
    const int L = nt - 1;
    for (int i = threadIdx.x; i < kFactors * nt; i += blockDim.x) {
        const int k = i / nt, t = i % nt;
        dev_s[k][t] = t < L - 1 ? S.sv[k][t] - (S.sv[k][L] + (double)(t - L) * (S.sv[k][L] - S.sv[k][L - 1])) : 0.0;
    }
    __syncthreads();
}
// A CTA's (128 threads) largest magnitudes of date j into top (bits; cleared before)
__device__ __forceinline__ void store_largest(double (&best)[2], int j, unsigned long long* top)
{
    __shared__ double top_s[2][4];
    for (int o = 16; o > 0; o >>= 1) {
        best[0] = fmax(best[0], __shfl_xor_sync(0xffffffffu, best[0], o));
        best[1] = fmax(best[1], __shfl_xor_sync(0xffffffffu, best[1], o));
    }
    if ((threadIdx.x & 31) == 0) {
        top_s[0][threadIdx.x >> 5] = best[0];
        top_s[1][threadIdx.x >> 5] = best[1];
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        const double* t = top_s[threadIdx.x];
        const double x = fmax(fmax(t[0], t[1]), fmax(t[2], t[3]));
        atomicMax(top + 2 * j + threadIdx.x, (unsigned long long)__double_as_longlong(x));
    }
}

// R_jk(m) and its running sum for date j = blockIdx.y + 2 at every lag it reads
// (m < (j - 1) stride): resp[(k (B - 1) + j - 2) M + m], and the largest
// magnitude over lags and factors in top.
__global__ void __launch_bounds__(128)
    contract_response_kernel(int nt, double c, int stride, int B, const __grid_constant__ ContractLoadings S,
                             const double2* __restrict__ weights, unsigned long long* __restrict__ top,
                             double2* __restrict__ resp)
{
    __shared__ double dev_s[kFactors][kMaxTenor];
    const int M = (B - 1) * stride, j = blockIdx.y + 2, lags = (j - 1) * stride;
    const int m0 = blockIdx.x * blockDim.x, m = m0 + threadIdx.x;
    if (m0 >= lags) return;
    load_deviations(S, nt, dev_s);
    double best[2] = {0.0, 0.0};
    if (m < lags) {
        const DateResponse r(S, dev_s, nt - 1, c, j, m, m0, lags, [&](int i) { return weights[(size_t)i * M + m]; });
#pragma unroll
        for (int k = 0; k < kFactors; ++k) resp[((size_t)k * (B - 1) + (j - 2)) * M + m] = make_double2(r.v[k], r.w[k]);
        r.largest(best);
    }
    store_largest(best, j, top);
}

// The scales of the dates from their largest responses.  A date with a response that
// overflowed has a NaN for a scale and so for its values (its slices, NaN too, would
// come out of the integer sums as zero: a curve without noise).
__device__ __forceinline__ void store_scales(const unsigned long long* top, double* scale)
{
    for (int i = threadIdx.x; i < 2 * kMaxTenor; i += blockDim.x)
        scale[i] = top[i] < kInfBits ? power_of_two(contract_exponent(top[i])) * kSumUnit
                                     : __longlong_as_double(0x7ff8000000000000ll);
}
// The slices of a scaled response x into row val (value 3 i + k of a chunk: step i,
// factor k) and column col of the chunk's image: three k-tiles of 16 rows, each two
// halves of 8 that hold the kLevels npad columns slice npad + 2 slot + {0 value, 1
// sum} as consecutive 16-byte rows.
__device__ __forceinline__ void store_slices(unsigned char* image, int npad, int chunk, int val, int col, double x)
{
    const int oct = val >> 3;
    unsigned char* out = image + (size_t)chunk * chunk_bytes(npad) + (size_t)(oct >> 1) * (kLevels * npad * 32) +
                         (size_t)(oct & 1) * (kLevels * npad * 16);
#pragma unroll
    for (int s = 0; s < kLevels; ++s) {
        const double b = s < kLevels - 1 ? rint(x) : x;
        *reinterpret_cast<__half*>(out + (size_t)(s * npad + col) * 16 + 2 * (val & 7)) = __float2half_rn((float)b);
        x = (x - b) * (double)kShift;
    }
}

// The image of one window from the responses, padding included
__global__ void contract_image_kernel(int stride, int B, ContractWindow W, const unsigned long long* __restrict__ top,
                                      const double2* __restrict__ resp, double* __restrict__ scale,
                                      unsigned char* __restrict__ image)
{
    const int M = (B - 1) * stride;
    if (blockIdx.x == 0) store_scales(top, scale);
    const int64_t per_chunk = 48 * (int64_t)W.npad;
    const int64_t total = per_chunk * W.chunks;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int chunk = (int)(i / per_chunk), rem = (int)(i % per_chunk);
        const int col = (rem >> 3) % W.npad, val = 8 * ((rem >> 3) / W.npad) + (rem & 7);
        const int step = chunk * kChunk + val / 3, k = val % 3;
        const int slot = col >> 1, j = W.hi - slot;
        double x = 0.0;
        if (slot < W.slots) {
            const int lag = (j - 1) * stride - 1 - step;
            if (lag >= 0) {
                const double2 r = resp[((size_t)k * (B - 1) + (j - 2)) * M + lag];
                x = ((col & 1) ? r.y : r.x) * power_of_two(-contract_exponent(top[2 * j + (col & 1)]));
            }
        }
        store_slices(image, W.npad, chunk, val, col, x);
    }
}

// The image of one window with nothing kept beside it (blockIdx.y: the slot): every
// thread walks its own lag, first (IMAGE = false) for the dates' largest responses,
// then again for the slices (the image cleared before).  The walk's serial FP64
// chain twice and three times the FP64 work of the two kernels above: for runs that
// have no room for their scratch.
template <bool IMAGE>
__global__ void __launch_bounds__(128)
    contract_compact_kernel(int nt, double c, int stride, const __grid_constant__ ContractLoadings S,
                            const __grid_constant__ WalkParams K, ContractWindow W, unsigned long long* __restrict__ top,
                            double* __restrict__ scale, unsigned char* __restrict__ image)
{
    __shared__ double dev_s[kFactors][kMaxTenor];
    const int slot = blockIdx.y, j = W.hi - slot, lags = (j - 1) * stride;
    const int m0 = blockIdx.x * blockDim.x, m = m0 + threadIdx.x;
    if (IMAGE && blockIdx.x == 0 && slot == 0) store_scales(top, scale);
    if (m0 >= lags) return;
    load_deviations(S, nt, dev_s);
    double best[2] = {0.0, 0.0};
    if (m < lags) {
        LagWalk walk(K, m);
        const DateResponse r(S, dev_s, nt - 1, c, j, m, m0, lags, [&](int i) { return walk.next(K, i); });
        if constexpr (IMAGE) {
            const int step = lags - 1 - m;
            const double sx = power_of_two(-contract_exponent(top[2 * j])),
                         sa = power_of_two(-contract_exponent(top[2 * j + 1]));
#pragma unroll
            for (int k = 0; k < kFactors; ++k) {
                store_slices(image, W.npad, step / kChunk, 3 * (step % kChunk) + k, 2 * slot, r.v[k] * sx);
                store_slices(image, W.npad, step / kChunk, 3 * (step % kChunk) + k, 2 * slot + 1, r.w[k] * sa);
            }
        } else {
            r.largest(best);
        }
    }
    if constexpr (!IMAGE) store_largest(best, j, top);
}

// The power of two 2^e of each path: e the least that brings the evolved steps'
// normals (values first .. per_path - 1; the steps before are not drawn upon, so
// nothing that a caller leaves there may set a scale) below 2^(3 - guard), and 0
// where that is less and the largest is no smaller than 1/4: smaller ones are
// brought up.  A non-finite normal makes its own path's scale, and so its curve, a NaN.
__global__ void contract_ext_scale_kernel(const double* __restrict__ raw, int64_t n_paths, int64_t first,
                                          int64_t per_path, int guard, ExtRow* __restrict__ out)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t p = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; p < n_paths; p += warps) {
        uint32_t top = 0;  // biased exponents: 2047 of a non-finite normal
#pragma unroll 4
        for (int64_t i = first + lane; i < per_path; i += 32)
            top = max(top, ((uint32_t)(__double_as_longlong(raw[p * per_path + i]) >> 52)) & 0x7ffu);
        top = __reduce_max_sync(0xffffffffu, top);
        const int x = (int)top - 1023;
        int e = x - 2 + guard;
        if (e < 0) e = x >= -2 ? 0 : max(e, -900);
        if (lane == 0) out[p] = {top == 0x7ffu ? __longlong_as_double(0x7ff8000000000000ll) : scalbn(1.0, e), e};
    }
}

// External normals [path][step][3] -> [step][3][path] as pairs {hi, lo 2^27} of the
// scaled value hi + lo, for the evolved steps: hi its first 24 bits, lo the other 29
// rounded to 24, by integer operations on the bits.  Tiles of 32 paths x 32 values
// through shared memory.  Bound: memory (48 bytes a path-step).
__global__ void __launch_bounds__(256)
    contract_ext_kernel(const double* __restrict__ raw, int64_t n_paths, int64_t first, int64_t per_path,
                        const ExtRow* __restrict__ row, float2* __restrict__ out)
{
    __shared__ float2 tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t p0 = (int64_t)blockIdx.x * 32;
    int e[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) e[u] = p0 + ty + 8 * u < n_paths ? row[p0 + ty + 8 * u].e : 0;
    for (int64_t i0 = first + (int64_t)blockIdx.y * 32; i0 < per_path; i0 += (int64_t)gridDim.y * 32) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t p = p0 + ty + 8 * u, i = i0 + tx;
            const uint64_t b = p < n_paths && i < per_path ? (uint64_t)__double_as_longlong(raw[p * per_path + i]) : 0;
            const int f = (int)(b >> 52 & 0x7ffu), x = f - 1023 - e[u] + 127;  // x: FP32's biased exponent
            const uint32_t sign = (uint32_t)(b >> 63) << 31;
            float hi = 0.0f, lo = 0.0f;
            if (f > 0 && x > 0) {  // (else nothing beside the path's scale; x <= 129 by the choice of e)
                hi = __uint_as_float(sign | (uint32_t)x << 23 | (uint32_t)(b >> 29 & 0x7fffffu));
                // the low 29 bits in units of 2^(x - 127 - 52), times 2^27
                const int y = x - 52 + 27;
                if (y > 0) lo = (float)(uint32_t)(b & 0x1fffffffu) * __uint_as_float(sign | (uint32_t)y << 23);
            }
            tile[tx][ty + 8 * u] = f2(hi, lo);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t i = i0 + ty + 8 * u;
            if (i < per_path && p0 + tx < n_paths) out[(size_t)i * (size_t)n_paths + (size_t)(p0 + tx)] = tile[ty + 8 * u][tx];
        }
        __syncthreads();
    }
}

size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

constexpr size_t contract_smem(int npad, int dates)
{
    const size_t need = kBStages * chunk_bytes(npad) + sizeof(longlong2) * (size_t)(npad / 2) * kContractTile +
                        sizeof(double) * (size_t)(dates + 2) * kContractTile;
    // more than half an SM's shared memory: one CTA per SM, which takes all of its tensor memory
    return std::max<size_t>(need, 120 * 1024);
}
// the largest window: kContractMaxSlots dates and date 1
constexpr size_t kContractSmemMost = contract_smem(2 * kContractMaxSlots, kContractMaxSlots + 1);

}  // namespace

int contract_windows(int n_blocks, int stride, ContractPlan plan, ContractWindow* w)
{
    const int most = plan.slots;
    int n = 0;
    size_t image = align_up(2 * kScaleBytes);
    for (int hi = n_blocks; hi >= 1;) {
        const int lo = hi - 1 <= most ? 1 : hi - most + 1;
        ContractWindow x;
        x.lo = lo;
        x.hi = hi;
        x.slots = std::max(hi - std::max(lo, 2) + 1, 0);
        x.npad = std::max((2 * x.slots + 15) / 16 * 16, 16);
        x.chunks = ((hi - 1) * stride + kChunk - 1) / kChunk;
        x.image = image;
        if (!plan.compact) image += align_up((size_t)x.chunks * chunk_bytes(x.npad));
        if (w) w[n] = x;
        ++n;
        hi = lo - 1;
    }
    return n;
}

size_t contract_table_bytes(int stride, int n_blocks, ContractPlan plan)
{
    ContractWindow w[kMaxTenor];
    const int n = contract_windows(n_blocks, stride, plan, w);
    size_t end = 0;
    for (int i = 0; i < n; ++i) end = std::max(end, w[i].image + align_up((size_t)w[i].chunks * chunk_bytes(w[i].npad)));
    if (plan.compact) return end;
    const size_t dates = std::max(n_blocks - 1, 1), lags = dates * stride;
    return end + sizeof(double2) * lags * (kFactors * dates + kMaxTenor);
}

static bool table_shape_ok(int nt, int n_blocks, int stride)
{
    return nt >= 35 && nt <= kMaxTenor && n_blocks >= 1 && n_blocks < nt && stride >= 1;
}

cudaError_t launch_contract_table(int nt, double c, int stride, int n_blocks, bool pc, ContractPlan plan,
                                  const double* sv, bool same_shape, void* table, cudaStream_t s)
{
    if (!table_shape_ok(nt, n_blocks, stride) || plan.compact) return cudaErrorInvalidValue;
    ContractLoadings S;
    std::memcpy(S.sv, sv, sizeof(S.sv));
    ContractWindow w[kMaxTenor];
    const int n = contract_windows(n_blocks, stride, plan, w);
    if (n_blocks == 1) return cudaSuccess;  // date 1 alone: nothing evolves
    double* scale = (double*)table;
    unsigned long long* top = (unsigned long long*)((unsigned char*)table + kScaleBytes);
    double2* resp = (double2*)((unsigned char*)table + w[n - 1].image +
                               align_up((size_t)w[n - 1].chunks * chunk_bytes(w[n - 1].npad)));
    const int M = (n_blocks - 1) * stride;
    double2* weights = resp + (size_t)M * kFactors * (n_blocks - 1);
    const WalkParams K = walk_params(c, pc);
    cudaError_t e = cudaMemsetAsync(top, 0, kScaleBytes, s);
    if (e != cudaSuccess) return e;
    if (!same_shape) contract_weights_kernel<<<(M + 63) / 64, 64, 0, s>>>(K, M, nt - 3, weights);
    contract_response_kernel<<<dim3((M + 127) / 128, n_blocks - 1), 128, 0, s>>>(nt, c, stride, n_blocks, S, weights,
                                                                                 top, resp);
    for (int i = 0; i < n; ++i) {
        if (w[i].chunks == 0) continue;
        const int64_t total = 48 * (int64_t)w[i].npad * w[i].chunks;
        contract_image_kernel<<<(unsigned)std::min<int64_t>((total + 255) / 256, 1216), 256, 0, s>>>(
            stride, n_blocks, w[i], top, resp, scale, (unsigned char*)table + w[i].image);
    }
    return cudaGetLastError();
}

cudaError_t launch_contract_window(int nt, double c, int stride, int n_blocks, bool pc, const ContractWindow& W,
                                   const double* sv, void* table, cudaStream_t s)
{
    if (!table_shape_ok(nt, n_blocks, stride)) return cudaErrorInvalidValue;
    if (W.slots == 0) return cudaSuccess;  // date 1 alone: nothing evolves
    ContractLoadings S;
    std::memcpy(S.sv, sv, sizeof(S.sv));
    const WalkParams K = walk_params(c, pc);
    double* scale = (double*)table;
    unsigned long long* top = (unsigned long long*)((unsigned char*)table + kScaleBytes);
    unsigned char* image = (unsigned char*)table + W.image;
    // (the image lies behind the scales and the largest responses)
    cudaError_t e = cudaMemsetAsync(table, 0, W.image + (size_t)W.chunks * chunk_bytes(W.npad), s);
    if (e != cudaSuccess) return e;
    const dim3 grid(((W.hi - 1) * stride + 127) / 128, W.slots);
    contract_compact_kernel<false><<<grid, 128, 0, s>>>(nt, c, stride, S, K, W, top, scale, image);
    contract_compact_kernel<true><<<grid, 128, 0, s>>>(nt, c, stride, S, K, W, top, scale, image);
    return cudaGetLastError();
}

cudaError_t launch_contract_ext(const double* raw, int64_t n_paths, int n_blocks, int stride, void* out, cudaStream_t s)
{
    if (stride < 2) return cudaErrorInvalidValue;  // (the rows lie where the first block's normals would)
    const int64_t first = (int64_t)stride * 3, per_path = first * n_blocks;
    // a path's running sums stay below 2^62: values x 2^10 2^8 2^30 units
    int guard = 0;
    while ((per_path - first) >> (14 + guard) > 0) ++guard;
    ExtRow* row = (ExtRow*)out;
    contract_ext_scale_kernel<<<(unsigned)std::min<int64_t>((n_paths + 7) / 8, 4096), 256, 0, s>>>(raw, n_paths, first,
                                                                                                   per_path, guard, row);
    if (n_blocks > 1) {
        const int64_t gx = (n_paths + 31) / 32, tiles = (per_path - first + 31) / 32;
        const int64_t gy = std::max<int64_t>(1, std::min<int64_t>(tiles, 4096 / gx));
        contract_ext_kernel<<<dim3((unsigned)gx, (unsigned)gy), 256, 0, s>>>(raw, n_paths, first, per_path, row,
                                                                             (float2*)out);
    }
    return cudaGetLastError();
}

// Tiles whose steps are split over all SMs: those left over after the whole
// waves, when dealing their groups costs less than a wave of whole tiles.  Decided
// on the whole run's groups, so every window (and an external-normals run's other
// windows) splits the same paths.  Two groups' time covers the second launch and
// the pricing kernel.  FP64 calls: 128 paths 10y 189 -> 124 us, 5,000 paths 185 ->
// 151 us, 5,000 paths 25y 471 -> 296 us, 100,003 paths 30y 2.73 -> 2.46 ms.
static int64_t split_tiles(int64_t n_paths, int n_blocks, int stride, int n_sms)
{
    const int64_t tiles = (n_paths + kContractTile - 1) / kContractTile, rest = tiles % n_sms;
    const int G = tile_groups(((n_blocks - 1) * stride + kChunk - 1) / kChunk);
    return rest > 0 && (rest * G + n_sms - 1) / n_sms + 2 <= G ? rest : 0;
}

int64_t contract_rows(int64_t n_paths, int n_blocks, int stride, int n_sms, bool with_split)
{
    const int64_t split = with_split ? split_tiles(n_paths, n_blocks, stride, n_sms) : 0;
    return (n_paths + kContractTile - 1) / kContractTile + 3 * split;
}

size_t contract_sums_bytes(int64_t n_paths, int n_blocks, int stride, int n_sms, ContractPlan plan)
{
    ContractWindow w[kMaxTenor];
    const int n = contract_windows(n_blocks, stride, plan, w);
    int npad = 0;
    for (int i = 0; i < n; ++i) npad = std::max(npad, w[i].npad);
    return sizeof(longlong2) * (size_t)split_tiles(n_paths, n_blocks, stride, n_sms) * (npad / 2) * kContractTile;
}

cudaError_t launch_path_contract(int nt, const PathParams<double>& P, const ContractWindow& W, const void* table,
                                 const void* normals, double* partials, double* estore, double* carry, longlong2* sums,
                                 double* result, int n_sms, cudaStream_t s, int* launches)
{
    if (!path_tenor_supported(nt) || P.n_blocks < 1 || P.n_blocks >= nt || P.stride < 1) return cudaErrorInvalidValue;
    if ((W.lo != 1 || W.hi != P.n_blocks) && !carry) return cudaErrorInvalidValue;
    const float2* ext = (const float2*)normals;
    const ExtRow* ext_row = (const ExtRow*)normals;
    auto kernel = ext ? path_kernel_contract<true> : path_kernel_contract<false>;
    auto price = ext ? contract_price_kernel<true> : contract_price_kernel<false>;
    cudaError_t e = allow_dynamic_smem(kernel, kContractSmemMost);
    if (e != cudaSuccess) return e;
    ContractParams Q;
    Q.P = P;
    Q.W = W;
    const int64_t tiles = (P.n_paths + kContractTile - 1) / kContractTile;
    const int64_t split = sums ? split_tiles(P.n_paths, P.n_blocks, P.stride, n_sms) : 0, whole = tiles - split;
    const size_t smem = contract_smem(W.npad, W.hi - W.lo + 1);
    int count = 0;
    if (whole > 0) {
        Q.tile0 = 0;
        Q.n_tiles = whole;
        Q.sums = nullptr;
        kernel<<<(unsigned)std::min<int64_t>(whole, n_sms), kThreads, smem, s>>>(
            Q, (const unsigned char*)table, ext, ext_row, partials, estore, carry, result);
        ++count;
    }
    if (split > 0) {
        Q.tile0 = whole;
        Q.n_tiles = split;
        Q.sums = sums;
        const int64_t groups = split * tile_groups(W.chunks);
        if (groups > 0) {
            e = cudaMemsetAsync(sums, 0, sizeof(longlong2) * (size_t)split * (W.npad / 2) * kContractTile, s);
            if (e != cudaSuccess) return e;
            kernel<<<(unsigned)std::min<int64_t>(groups, n_sms), kThreads, smem, s>>>(
                Q, (const unsigned char*)table, ext, ext_row, partials, estore, carry, result);
            ++count;
        }
        price<<<(unsigned)(4 * split), 32 * kPriceWarps, 0, s>>>(Q, (const double*)table, ext_row, whole, partials,
                                                                estore, carry);
        ++count;
    }
    *launches += count;
    return cudaGetLastError();
}

cudaError_t launch_contract(int nt, double c, bool pc, const double* sv, const PathParams<double>& P, ContractPlan plan,
                            bool have_table, void* table, const void* normals, double* partials, double* estore,
                            double* carry, longlong2* sums, double* result, int n_sms, cudaStream_t s, int* launches)
{
    ContractWindow w[kMaxTenor];
    const int n = contract_windows(P.n_blocks, P.stride, plan, w);
    *launches = 0;
    for (int i = 0; i < n; ++i) {
        if (!have_table) {
            const cudaError_t e = launch_contract_window(nt, c, P.stride, P.n_blocks, pc, w[i], sv, table, s);
            if (e != cudaSuccess) return e;
            *launches += w[i].slots > 0 ? 2 : 0;
        }
        const cudaError_t e = launch_path_contract(nt, P, w[i], table, normals, partials, estore, carry, sums, result,
                                                   n_sms, s, launches);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace hjm
