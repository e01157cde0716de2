// hjm_forward.cu -- fused Monte Carlo path kernel and reductions.
//
// One launch of path_kernel replaces the reference's whole GPU pipeline
// (simulation_gpu.cu:956-1179): cuRAND normal buffer (:1057-1071), 2,500
// single-step launches each followed by cudaDeviceSynchronize (:724-796, or
// the 50-step kernel4 variant :471-669), the exposure kernel (:803-882) and
// the cuBLAS gemv column sum (:889-933).  One thread owns one Monte Carlo
// path for its whole life: the curve sits in registers, normals come from
// Philox in registers, the numeraire of each 0.5y block end is priced on the
// spot, and the per-path exposure profile is reduced inside the CTA.
//
// Semantics follow the reference CPU path (simulation_cpu.h:188-296), which
// the reference's shared-memory GPU kernel also reproduces (xls RMSE 0.0):
//   * block 0 (steps 0..stride-1) holds the curve at spot (simulation_cpu.h:212);
//   * after block b the numeraire of tenor i = b+1 is sampled: forward f[i] and
//     discount exp(-dt * sum of f[i] over all steps so far) (simulation_cpu.h:248-250);
//   * cash flow of date i: D_i * N * alpha_i * (L_i - K), L = m (e^{f/m} - 1);
//     exposure E_j = max(sum_{i>j} cf_i, 0) (simulation_cpu.h:279-295).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "hjm_device.cuh"
#include "hjm_kernels.h"
#include "hjm_pairs.cuh"
#include "hjm_epilogue.cuh"

namespace hjm {

// Shared-memory layout of the FP64 path kernel (dynamic), per CTA of
// kFp64Cta threads, column tid private to its thread until the epilogue:
//   cf_s   [B+1] double   cash flows of the sampled dates
//   acc_s  [B+1] double   FP64 discount sums of the stochastic part per tenor
//   work_s [2(B+2)] double  curve at block start / end, then exposures
//   red_s  [2 * kFp64Cta/32] double  CVA statistics

__host__ __device__ inline size_t path_smem_bytes(int nt, int n_blocks, bool mixed)
{
    (void)nt;
    (void)mixed;
    const size_t rows = (size_t)n_blocks + 1;
    size_t b = rows * kFp64Cta * 8;  // cf_s
    b += rows * kFp64Cta * 8;        // acc_s
    b = (b + 127) & ~(size_t)127;
    b += 2 * (rows + 1) * kFp64Cta * 8;  // work_s
    b += 2 * (kFp64Cta / 32) * 8;        // red_s
    return b;
}

// Discount sums by block-sum recovery.  Over one block of Euler steps
// n = n0 .. n0+stride-1 the states h_n = A h_{n-1} + xi_n sum to
//     (I - A) H = sum_n xi_n - A (h_end - h_start),   H = sum_n h_n,
// and (I - A) H [t] = c (H[t] - H[t+1]) for t below the last tenor.  So with
// one tenor accumulated directly (H[B], the last tenor still to be sampled),
//     H[t] = H[t+1] + (Xi[t] - (A d)[t]) / c,  d = h_end - h_start,
// gives every block sum the discount needs in O(B) FP64 operations per block
// instead of one FP64 addition per tenor per step (the FP64 pipe is the bound).
// Exact in exact arithmetic; in FP64 the recovered sums differ from step-by-
// step accumulation by ~1e-14 relative.
//
// Polynomial volatility (POLY).  When sqrt(dt) sigma_k(T) = sum_d svc[k][d] T^d
// with degree <= 2, the noise of a step is xi = alpha + beta T + gamma T^2 and
// the convection operator maps that basis into itself up to one last-tenor
// term:  A 1 = 1,  A T = T + c dtau 1,  A T^2 = T^2 + 2 c dtau T + c dtau^2 1
// - 2 c dtau^2 e_L.  Writing h = S 1 + U T + W T^2 + hc, the Euler step becomes
//     S <- S + c dtau U + c dtau^2 W + alpha,   U <- U + 2 c dtau W + beta,
//     W <- W + gamma,   hc <- A hc - 2 c dtau^2 W e_L   (old U, W on the right),
// exact in exact arithmetic: the curve is advanced in full, with the
// convection of hc per tenor instead of 5 operations, plus a dozen per step.
// With the growth scaling of PathParams (v = h / (1-c)^j) the convection is
// one FMA per tenor, and the table form four.
// FORM: kFormTable (volatility table), kFormPoly (quadratic factors) or
// kFormPolyTri (factor k of degree <= k, as the synthetic workloads' factors: the noise
// projection then skips the three zero coefficients).
template <int NT, bool EXT, int FORM>
__global__ void __launch_bounds__(kFp64Cta, 4)
    path_kernel_fp64(const __grid_constant__ PathParams<double> P, const double* __restrict__ ext,
                     double* __restrict__ partials, double* __restrict__ estore)
{
    constexpr int kCta = kFp64Cta;
    constexpr int L = NT - 1;
    constexpr bool POLY = FORM != kFormTable;
    constexpr bool TRI = FORM == kFormPolyTri;
    constexpr int kGroup = 8;                      // dead-tenor skipping granularity (4 measured slower)
    constexpr int kGroups = (L + kGroup - 1) / kGroup;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x;
    const int B = P.n_blocks;
    const int rows = B + 1;
    double* cf_s = reinterpret_cast<double*>(smem);
    double* acc_s = cf_s + (size_t)rows * kCta;
    size_t off = ((size_t)rows * kCta * 16 + 127) & ~(size_t)127;
    double* work_s = reinterpret_cast<double*>(smem + off);
    double* red_s = work_s + (size_t)2 * (rows + 1) * kCta;

    const int64_t cta_base = (int64_t)blockIdx.x * kCta;
    const int64_t lp = cta_base + tid;            // path index within this launch
    const bool active = lp < P.n_paths;
    const uint64_t gpath = P.path_offset + (uint64_t)lp;

    // stochastic part of the curve (POLY: its convected remainder hc); zero
    // through block 0 (spot hold)
    double h[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) h[t] = 0.0;
    double S = 0.0, U = 0.0, W = 0.0;  // POLY: parallel, tilt and curvature parts
    for (int i = 0; i < rows; ++i) acc_s[i * kCta + tid] = 0.0;
    double* hs_s = work_s;
    double* he_s = work_s + (size_t)(rows + 1) * kCta;
    for (int t = 0; t <= B + 1; ++t) hs_s[t * kCta + tid] = 0.0;

    double g = 1.0;  // the kernel holds v; h = g v
    auto value_at = [&](int i) -> double {
        double v = g * select_reg<NT, double>(h, i);
        if (POLY) v += fma(P.tau[i], fma(P.tau[i], W, U), S);
        return v;
    };
    // price date i from the sampled numeraire (x_i, D_i)
    auto sample = [&](int i) {
        const double x = P.psamp[i] + value_at(i);
        const double a = P.psum[i] + acc_s[i * kCta + tid];
        const double D = exp(-a * P.dt);
        const double Lb = P.m * (exp(x * P.inv_m) - 1.0);
        cf_s[i * kCta + tid] = D * (P.payA[i] * Lb - P.payB[i]);
    };

    sample(1);
    const double c = P.c, rr = P.rr;
    for (int b = 1; b < B; ++b) {
        double f0 = 0.0, f1 = 0.0, f2 = 0.0;  // block sums of phi_k
        double sS = 0.0, sU = 0.0, sW = 0.0;  // POLY: block sums of S, U, W
        // anchor: hb = sum_s h_s[B] = g_end * Tb with Tb <- (1 + rr) Tb + v[B]
        // (g_s = g_end (1 + rr)^(stride - s)), one FMA per step
        double Tb = 0.0;
        double ig = P.igblk[b];          // table form: (1 + rr)^n'
        // tenors <= b are never read again (date b was sampled; the upwind step
        // carries information from high to low tenors only): their groups of
        // kGroup tenors are skipped, which changes no output bit
        const int live = b + 1;
        double mig = P.m2k2 * P.igblk[b];  // polynomial form: -2 c dtau^2 (1 + rr)^n'
        for (int s = 0; s < P.stride; ++s) {
            const int n = b * P.stride + s;
            double phi0, phi1, phi2;
            draw_phi<double, EXT>(ext, gpath, active ? lp : 0, P.n_paths, n, P.rk0, P.rk1, phi0, phi1, phi2);
            // in place, ascending (h[t+1] is still the old value); the last
            // tenor, which reads h[L-1], first
            if constexpr (POLY) {
                // the noise projection folded into the updates of S, U, W:
                // S' = S + c dtau U + c dtau^2 W + sum_k svc[k][0] phi_k, etc.
                // (old U, W on the right; factor k of degree <= k drops 3 terms)
                mig *= P.ip;
                const double hl = fma(mig, W, fma(rr, fma(2.0, h[L], -h[L - 1]), h[L]));  // + scaled source
#pragma unroll
                for (int gi = 0; gi < kGroups; ++gi) {
                    // uniform: skip groups of dead tenors, and (polynomial form)
                    // the exact zeros below the remainder's front: driven only
                    // at the last tenor from zero, after k steps it is nonzero
                    // on tenors >= L - k only
                    const int front = L - 1 - ((b - 1) * P.stride + s);
                    if (kGroup * gi + kGroup > (live > front ? live : front)) {
#pragma unroll
                        for (int j = 0; j < kGroup; ++j) {
                            const int t = kGroup * gi + j;
                            if (t < L) h[t] = fma(rr, h[t + 1], h[t]);
                        }
                    }
                }
                h[L] = hl;
                double Sn = fma(P.svc[0][0], phi0, fma(P.k2, W, fma(P.k1, U, S)));
                Sn = fma(P.svc[2][0], phi2, fma(P.svc[1][0], phi1, Sn));
                double Un = fma(P.svc[2][1], phi2, fma(P.svc[1][1], phi1, fma(2.0 * P.k1, W, U)));
                double Wn = fma(P.svc[2][2], phi2, W);
                if constexpr (!TRI) {
                    Un = fma(P.svc[0][1], phi0, Un);
                    Wn = fma(P.svc[1][2], phi1, fma(P.svc[0][2], phi0, Wn));
                }
                S = Sn;
                U = Un;
                W = Wn;
                sS += S;
                sU += U;
                sW += W;
            } else {
                ig *= P.ip;
                const double p0 = phi0 * ig, p1 = phi1 * ig, p2 = phi2 * ig;
                double xl = fma(P.sv[0][L], p0, h[L]);
                xl = fma(P.sv[1][L], p1, xl);
                xl = fma(P.sv[2][L], p2, xl);
                const double hl = fma(rr, fma(2.0, h[L], -h[L - 1]), xl);
#pragma unroll
                for (int gi = 0; gi < kGroups; ++gi) {
                    if (kGroup * gi + kGroup > live) {
#pragma unroll
                        for (int j = 0; j < kGroup; ++j) {
                            const int t = kGroup * gi + j;
                            if (t < L) {
                                double x = fma(P.sv[0][t], p0, h[t]);
                                x = fma(P.sv[1][t], p1, x);
                                x = fma(P.sv[2][t], p2, x);
                                h[t] = fma(rr, h[t + 1], x);
                            }
                        }
                    }
                }
                h[L] = hl;
                f0 += phi0;
                f1 += phi1;
                f2 += phi2;
            }
            Tb = fma(P.ip, Tb, select_reg<NT, double>(h, B));
        }
        g = P.gblk[b + 1];  // (1 + rr)^-(b stride): the scale at the block end
        const double hb = g * Tb;
#pragma unroll
        for (int t = 0; t < NT; ++t)
            if (t <= B + 1) he_s[t * kCta + tid] = g * h[t];
        auto poly_part = [&](int t) -> double {
            return POLY ? fma(P.tau[t], fma(P.tau[t], sW, sU), sS) : 0.0;
        };
        double Hn = hb;
        acc_s[B * kCta + tid] += Hn + poly_part(B);
        double dn = he_s[B * kCta + tid] - hs_s[B * kCta + tid];
        for (int t = B - 1; t > b; --t) {
            const double d = he_s[t * kCta + tid] - hs_s[t * kCta + tid];
            const double xi = POLY ? 0.0 : fma(P.sv[2][t], f2, fma(P.sv[1][t], f1, P.sv[0][t] * f0));
            const double ad = fma(c, dn - d, d);
            Hn = fma(xi - ad, P.inv_c, Hn);
            acc_s[t * kCta + tid] += Hn + poly_part(t);
            dn = d;
        }
        double* tmp = hs_s;
        hs_s = he_s;
        he_s = tmp;
        sample(b + 1);
    }

    fp64_epilogue<kCta>(P, cf_s, work_s, red_s, partials, estore, cta_base, active);
}

// Mixed precision with packed FP32x2 arithmetic.  The curve of one path is held
// as H = ceil(NT/2) float2 pairs, pair p = {h[p], h[p+H]}: the upwind neighbour
// h[t+1] of every tenor lies in the same component of pair p+1, so each packed
// FMA (__ffma2_rn) advances two tenors: with the growth scaling of PathParams
// the polynomial form's step is one packed FMA per pair, the table form's four.
// Only the seam pair (p = H-1, whose .x neighbour is pair 0's .y), the pair
// holding the last tenor (backward difference) and the padding tenor of an odd
// grid take scalar fix-ups.
// ---------------------------------------------------------------------------
// Mixed-precision discount sums: FP32 block sums by the same recovery as the
// FP64 kernel, but anchored at tenor 1 and run upwards,
//     H[t+1] = H[t] - (sum_k sv[k][t] Phi_k - (A d)[t]) / c,   t = 1 .. B-1,
// so a block costs O(B) scalar FP32 operations and four additions per step
// (Phi_k and H[1]) instead of an addition per tenor per step; the FP32 block
// sums are then folded into FP64 per tenor.  The recovered sums differ from
// step-by-step FP32 accumulation by ~1e-6 relative (the FP32 rounding of the
// Euler steps divided by c), far inside the mixed-precision tolerance.
//
// Shared memory per thread: acc (B+1) FP64 discount sums, whose slot i holds
// date i's cash flow once tenor i is sampled; hs (B+2) FP32 curve at the block
// start, reused for the exposure tile at the end.
// Occupancy: 512 threads per SM by the registers (<= 128 per thread).
template <int NT, bool EXT, int C>
__global__ void __launch_bounds__(C, 512 / C)
    path_kernel_mixed(const __grid_constant__ MixedParams M, const double* __restrict__ ext,
                      double* __restrict__ partials, float* __restrict__ estore)
{
    const PathParams<float>& P = M.P;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x;
    const int B = P.n_blocks;
    const int rows = B + 1;
    double* acc_s = reinterpret_cast<double*>(smem);                      // [B+1][C]
    float* hs_s = reinterpret_cast<float*>(smem + (size_t)rows * C * 8);  // [B+2][C]
    double* red_s = reinterpret_cast<double*>(
        smem + (((size_t)rows * C * 8 + (size_t)(rows + 1) * C * 4 + 7) & ~(size_t)7));

    const int64_t cta_base = (int64_t)blockIdx.x * C;
    const int64_t lp = cta_base + tid;
    const bool active = lp < P.n_paths;
    const uint64_t gpath = P.path_offset + (uint64_t)lp;

    MixedPath<NT, false> x;
    x.reset();
    for (int i = 0; i < rows; ++i) acc_s[i * C + tid] = 0.0;
    for (int t = 0; t <= B + 1; ++t) hs_s[t * C + tid] = 0.f;

    auto sample = [&](int i) {
        const double xv = P.psamp[i] + (double)x.value(P, i);
        const double a = P.psum[i] + acc_s[i * C + tid];
        const float D = expf((float)(-a * P.dt));
        const float mm = (float)P.m;
        const float L = mm * expm1f((float)xv / mm);
        const float cf = D * ((float)P.payA[i] * L - (float)P.payB[i]);
        acc_s[i * C + tid] = (double)cf;  // cash flow of date i
    };

    sample(1);
    // normals drawn one step ahead, so that the generator's dependent chain
    // overlaps the curve update (the last step redraws itself, unused)
    const int n_last = B * P.stride - 1;
    const int64_t lpc = active ? lp : 0;
    float q0, q1, q2;
    draw_phi<float, EXT>(ext, gpath, lpc, P.n_paths, min(P.stride, n_last), P.rk0, P.rk1, q0, q1, q2);
    for (int b = 1; b < B; ++b) {
        BlockSums bs;
        bs.reset();
        x.begin_block(P, b);
        for (int s = 0; s < P.stride; ++s) {
            const int n = b * P.stride + s;
            const float phi0 = q0, phi1 = q1, phi2 = q2;
            draw_phi<float, EXT>(ext, gpath, lpc, P.n_paths, min(n + 1, n_last), P.rk0, P.rk1, q0, q1, q2);
            x.step(M, phi0, phi1, phi2);
            bs.add(x, phi0, phi1, phi2);
        }
        // block sums of tenors 2 .. B; fold (b, B] into FP64
        block_sums_up<NT, false>(x, hs_s, tid, C, P, bs, B, [&](int t, float Ht) {
            if (t > b) acc_s[t * C + tid] += as_f64(Ht);
        });
        // the block-end curve is the next block's start
#pragma unroll
        for (int t = 1; t < NT; ++t)
            if (t <= B + 1) hs_s[t * C + tid] = x.rem(t);
        sample(b + 1);
    }

    mixed_epilogue<double, C>(P, acc_s, hs_s, red_s, partials, estore, cta_base, active);
}

// The convected form of the polynomial factors on the tenors that matter.  In
// block b (from step b stride on) the remainder
// * holds nothing that counts below the tenor its source has reached (2^-46 per
//   unit of the source, MixedParams::win; 2^-30 would make the windows only half
//   a tenor narrower), and
// * is read by no later date at or below tenor b: information moves down the
//   tenors only,
// so a block convects tenors S0 .. L, S0 the largest window start (thirds of
// the tenors) at or below either bound: 28 of 51 tenors on average on the 25y
// swap.  The discount sums telescope (LongSums): no per-tenor sums and no
// block starts in shared memory, 0.25 KB per path at 60 dates instead of 0.5, so
// the registers bound the occupancy (16 warps per SM instead of 14).
// 512k paths: 25y quadratic 7.15 -> 5.95 ms, 25y cubic 7.66 -> 6.23, the
// 61-tenor netting set 9.61 -> 7.39 (with the windows alone 6.54 and 9.53); 15y at
// 256k paths 2.14 -> 1.94, the 10y swap convected 1.37 -> 1.30.
// Steps unrolled by 2: 7.0 ms by 1 on the cubic run, 6.6 by 3.
// CTAs of 64 paths, as the adjoint's (the same partial sums; 128 run as fast).
constexpr int kConvCta = 64;
template <int NT, bool EXT, bool CUB>
__global__ void __launch_bounds__(kConvCta, 512 / kConvCta)
    path_kernel_mixed_conv(const __grid_constant__ MixedParams M, const double* __restrict__ ext,
                           double* __restrict__ partials, float* __restrict__ estore)
{
    constexpr int C = kConvCta;
    const PathParams<float>& P = M.P;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x;
    const int B = P.n_blocks;
    float* cf_s = reinterpret_cast<float*>(smem);  // [B+2][C]: cash flows, then exposures one row up
    double* red_s = reinterpret_cast<double*>(smem + (size_t)(B + 2) * C * sizeof(float));

    const int64_t cta_base = (int64_t)blockIdx.x * C;
    const int64_t lp = cta_base + tid;
    const bool active = lp < P.n_paths;
    const uint64_t gpath = P.path_offset + (uint64_t)lp;

    MixedPath<NT, true, CUB> x;
    x.reset();
    LongSums<NT, CUB> z;
    z.reset();
    auto price = [&](int i, float value, double sum) {
        const double xv = P.psamp[i] + (double)value;
        const double a = P.psum[i] + sum;
        const float D = expf((float)(-a * P.dt));
        const float mm = (float)P.m;
        const float L = mm * expm1f((float)xv / mm);
        cf_s[i * C + tid] = D * ((float)P.payA[i] * L - (float)P.payB[i]);
    };
    price(1, 0.f, 0.0);
    // normals drawn one step ahead, so that the generator's dependent chain
    // overlaps the curve update (the last step redraws itself, unused)
    const int n_last = B * P.stride - 1;
    const int64_t lpc = active ? lp : 0;
    float q0, q1, q2;
    draw_phi<float, EXT>(ext, gpath, lpc, P.n_paths, min(P.stride, n_last), P.rk0, P.rk1, q0, q1, q2);
    auto block = [&](auto s0_c, int b) {
        constexpr int S0 = decltype(s0_c)::value;
        float sR = 0.f, sS = 0.f, sU = 0.f, sW = 0.f, sX = 0.f;
        x.begin_block(P, b);
#pragma unroll 2
        for (int s = 0; s < P.stride; ++s) {
            const int n = b * P.stride + s;
            const float phi0 = q0, phi1 = q1, phi2 = q2;
            draw_phi<float, EXT>(ext, gpath, lpc, P.n_paths, min(n + 1, n_last), P.rk0, P.rk1, q0, q1, q2);
            x.template step<S0>(M, phi0, phi1, phi2);
            sR = fmaf(x.g, pair_tenor<NT>(x.h, S0), sR);
            sS += x.S;
            sU += x.U;
            sW += x.W;
            if constexpr (CUB) sX += x.X;
        }
        z.fold(sR, sS, sU, sW, sX);
        float value;
        double sum;
        z.template read<S0>(x, P, S0, b + 1, value, sum);
        price(b + 1, value, sum);
    };
    constexpr int W1 = conv_window(NT, 0), W2 = conv_window(NT, 1);
    for (int b = 1; b < B; ++b) {
        const int w = window_start<NT>(M, b);
        if (w != z.start) z.move(x, P, w);
        if (w == W2)
            block(std::integral_constant<int, W2>(), b);
        else if (w == W1)
            block(std::integral_constant<int, W1>(), b);
        else
            block(std::integral_constant<int, 1>(), b);
    }
    mixed_epilogue<float, C>(P, cf_s, cf_s + C, red_s, partials, estore, cta_base, active);
}

__host__ __device__ inline size_t mixed_smem_bytes(int nt, int n_blocks, int cta = kCta)
{
    (void)nt;
    const size_t rows = (size_t)n_blocks + 1;
    const size_t head = rows * cta * 8 + (rows + 1) * cta * 4;
    return ((head + 7) & ~(size_t)7) + 2 * (cta / 32) * 8;
}

inline size_t conv_smem_bytes(int n_blocks)  // path_kernel_mixed_conv
{
    return (size_t)(n_blocks + 2) * kConvCta * sizeof(float) + 2 * (kConvCta / 32) * 8;
}

// Paths per CTA of the mixed kernels.  The table step keeps FP64 sums per tenor,
// so with many dates its shared memory bounds the occupancy and 64-thread CTAs
// pack an SM more finely (25y on 51 tenors: 79 KB per CTA of 128, 2 per SM; 5
// of 64, 10 warps instead of 8).  Otherwise the registers bound it, whatever
// the CTA size.
constexpr int kMixedSmallCta = 64;
inline int mixed_cta(int nt, int n_blocks, bool poly)
{
    if (poly) return kConvCta;
    return mixed_smem_bytes(nt, n_blocks) > (size_t)228 * 1024 / 4 ? kMixedSmallCta : kCta;
}

void pack_mixed_params(int nt, const PathParams<float>& P, MixedParams& M)
{
    std::memset(&M, 0, sizeof(M));
    M.P = P;
    const int H = (nt + 1) / 2;
    for (int k = 0; k < kFactors; ++k)
        for (int p = 0; p < H; ++p) {
            M.svp[k][p].x = P.sv[k][p];
            M.svp[k][p].y = (H + p < nt) ? P.sv[k][H + p] : 0.0f;
        }
    M.rp = make_float2(P.rr, P.rr);
    for (int k = 0; k < kFactors; ++k)
        for (int d = 0; d < 3; ++d) M.svcf[k][d] = (float)P.svc[k][d];
    M.k1f = (float)P.k1;
    M.k2f = (float)P.k2;
}

// ---------------------------------------------------------------------------
// Deterministic column sums of the CTA partials (Neumaier-compensated FP64):
// blockIdx.x the column, blockIdx.y one of gridDim.y row ranges, fixed
// assignment of rows to threads, fixed tree order.  Replaces the cuBLAS gemv with
// a ones vector (simulation_gpu.cu:889-933) and the host vAdd/saxpy
// (simulation_gpu.cu:941-951, 1157-1179).  The last CTA to finish (a counter in
// the cleared result block) adds the ranges of each column and forms EE, CVA, its
// standard error and dCVA/dhazard.  Bound: the FP64 pipe (18 cycles an
// instruction and SM), so 256 threads a CTA (the tree's additions grow with
// them: 25 us with 1,024) and up to six row ranges.  40 rows: 21 -> 16 us (two
// launches before), 8,192 rows 38 -> 22 us, 32,768 rows 88 -> 33 us.
// ---------------------------------------------------------------------------
constexpr int kReduceThreads = 256;
constexpr int kReduceRows = 1024;   // rows a range has at least
constexpr int kReduceRanges = 6;    // a column's ranges (23 columns of the 10y swap: 138 CTAs)

__device__ __forceinline__ void neumaier_add(double& s, double& comp, double x)
{
    const double t = s + x;
    comp += (fabs(s) >= fabs(x)) ? ((s - t) + x) : ((x - t) + s);
    s = t;
}

// The compensated sum of the warp's pairs, in every lane, in a fixed order
__device__ __forceinline__ void neumaier_warp(double& s, double& comp)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_down_sync(0xffffffffu, s, o), c = __shfl_down_sync(0xffffffffu, comp, o);
        comp += c;
        neumaier_add(s, comp, x);
    }
}

__global__ void __launch_bounds__(kReduceThreads)
    reduce_columns(double* partials, int64_t n_rows, int R, double* __restrict__ sums,
                   const __grid_constant__ FinalParams F, double* __restrict__ result)
{
    constexpr int kWarps = kReduceThreads / 32;
    __shared__ double ss[kWarps], cs[kWarps];
    __shared__ bool last_s;
    const int col = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5, ranges = gridDim.y;
    const int64_t per = (n_rows + ranges - 1) / ranges, begin = per * blockIdx.y, end = min(begin + per, n_rows);
    double s = 0.0, comp = 0.0;
    for (int64_t r = begin + t; r < end; r += 4 * kReduceThreads) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t q = r + u * kReduceThreads;
            v[u] = q < end ? partials[(size_t)q * R + col] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) neumaier_add(s, comp, v[u]);
    }
    neumaier_warp(s, comp);
    if (lane == 0) {
        ss[warp] = s;
        cs[warp] = comp;
    }
    __syncthreads();
    if (t == 0) {
        for (int w = 1; w < kWarps; ++w) {
            comp += cs[w];
            neumaier_add(s, comp, ss[w]);
        }
        // (a range's sum into its first row, which this CTA alone has read)
        (ranges > 1 ? partials + (size_t)begin * R : sums)[col] = s + comp;
        __threadfence();
        last_s = atomicAdd(reinterpret_cast<uint32_t*>(result + kResCount), 1u) == gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    if (ranges > 1) {
        for (int c = t; c < R; c += kReduceThreads) {
            double a = 0.0, ca = 0.0;
            for (int g = 0; g < ranges; ++g) neumaier_add(a, ca, __ldcg(partials + (size_t)(per * g) * R + c));
            sums[c] = a + ca;
        }
        __syncthreads();
    }
    if (warp != 0) return;
    auto sums_at = [&](int c) { return __ldcg(sums + c); };  // (written by this CTA or others)
    const int B = F.n_blocks;
    const double inv_n = 1.0 / (double)F.n_paths;
    double cva = 0.0, dcva = 0.0;
#pragma unroll
    for (int u = 0; u < kMaxTenor / 32; ++u) {
        const int j = lane + 32 * u;
        const double ee = (j <= B) ? sums_at(j) * inv_n : 0.0;
        result[kResEE + j] = ee;
        cva = fma(F.cvaw[j], ee, cva);
        dcva = fma(F.dcvaw[j], ee, dcva);
    }
    cva = warp_sum(cva);
    dcva = warp_sum(dcva);
    if (lane == 0) {
        const double s1 = sums_at(B + 1), s2 = sums_at(B + 2);
        const double n = (double)F.n_paths;
        const double var = (n > 1.0) ? fmax((s2 - s1 * s1 / n) / (n - 1.0), 0.0) : 0.0;
        result[kResCVA] = cva;
        result[kResCVAStderr] = sqrt(var / n);
        result[kResDCVADHazard] = dcva;
        result[kResCVAPathMean] = s1 * inv_n;
    }
}

// ---------------------------------------------------------------------------
// Diagnostics: the device's normals and raw Philox words; layout transposes.
// ---------------------------------------------------------------------------
__global__ void dump_normals_kernel(int64_t n_paths, uint64_t path_offset, int n_steps, uint32_t k0, uint32_t k1,
                                    double* __restrict__ out)
{
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n_paths * (int64_t)n_steps) return;
    const int64_t p = idx / n_steps;
    const int n = (int)(idx % n_steps);
    const uint4 w = philox4x32_10(normals_counter(path_offset + (uint64_t)p, (uint32_t)n), k0, k1);
    float z0, z1, z2;
    normals3(w, z0, z1, z2);
    out[idx * 3 + 0] = (double)z0;
    out[idx * 3 + 1] = (double)z1;
    out[idx * 3 + 2] = (double)z2;
}

__global__ void philox_words_kernel(int64_t n_paths, uint64_t path_offset, uint32_t step, uint32_t k0, uint32_t k1,
                                    uint32_t* __restrict__ out)
{
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_paths) return;
    const uint4 w = philox4x32_10(normals_counter(path_offset + (uint64_t)p, step), k0, k1);
    out[p * 4 + 0] = w.x;
    out[p * 4 + 1] = w.y;
    out[p * 4 + 2] = w.z;
    out[p * 4 + 3] = w.w;
}

// [path][step][3] -> [step][3][path] so that the path kernel reads coalesced
__global__ void transpose_normals_kernel(const double* __restrict__ in, int64_t n_paths, int n_steps,
                                         double* __restrict__ out)
{
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t total = n_paths * (int64_t)n_steps * 3;
    if (idx >= total) return;
    const int64_t p = idx % n_paths;
    const int64_t rest = idx / n_paths;  // = n * 3 + k
    out[idx] = in[(size_t)p * n_steps * 3 + (size_t)rest];
}

// [date][ld] of T -> [date][n_paths] of double
template <typename T>
__global__ void widen_exposures_kernel(const T* __restrict__ in, int64_t ld, int64_t n_paths, int n_dates,
                                       double* __restrict__ out)
{
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n_paths * (int64_t)n_dates) return;
    const int64_t j = idx / n_paths, p = idx % n_paths;
    out[idx] = (double)in[(size_t)j * ld + p];
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
template <int NT, bool EXT, int FORM>
static cudaError_t launch_fp64_t(const PathParams<double>& P, const double* ext, double* partials, double* estore,
                                 cudaStream_t s)
{
    const size_t smem = path_smem_bytes(NT, P.n_blocks, false);
    auto k = path_kernel_fp64<NT, EXT, FORM>;
    cudaError_t e = allow_dynamic_smem(k);
    if (e != cudaSuccess) return e;
    const int64_t grid = (P.n_paths + kFp64Cta - 1) / kFp64Cta;
    k<<<(unsigned)grid, kFp64Cta, smem, s>>>(P, ext, partials, estore);
    return cudaGetLastError();
}

template <int NT>
static cudaError_t launch_fp64_nt(const PathParams<double>& P, bool poly, const double* ext, double* partials,
                                  double* estore, cudaStream_t s)
{
    const bool tri = poly && P.svc[0][1] == 0.0 && P.svc[0][2] == 0.0 && P.svc[1][2] == 0.0;
    if (ext) return tri    ? launch_fp64_t<NT, true, kFormPolyTri>(P, ext, partials, estore, s)
                    : poly ? launch_fp64_t<NT, true, kFormPoly>(P, ext, partials, estore, s)
                           : launch_fp64_t<NT, true, kFormTable>(P, ext, partials, estore, s);
    return tri    ? launch_fp64_t<NT, false, kFormPolyTri>(P, ext, partials, estore, s)
           : poly ? launch_fp64_t<NT, false, kFormPoly>(P, ext, partials, estore, s)
                  : launch_fp64_t<NT, false, kFormTable>(P, ext, partials, estore, s);
}

cudaError_t launch_path_fp64(int nt, const PathParams<double>& P, bool poly, const double* ext, double* partials,
                             double* estore, cudaStream_t s)
{
    if (nt == 51) return launch_fp64_nt<51>(P, poly, ext, partials, estore, s);
    if (nt == 61) return launch_fp64_nt<61>(P, poly, ext, partials, estore, s);
    return cudaErrorInvalidValue;
}

template <int NT, bool EXT>
static cudaError_t launch_mixed_t(const MixedParams& M, bool poly, bool cub, const double* ext, double* partials,
                                  float* estore, cudaStream_t s)
{
    const int B = M.P.n_blocks, cta = mixed_cta(NT, B, poly);
    auto k = cub    ? path_kernel_mixed_conv<NT, EXT, true>
             : poly ? path_kernel_mixed_conv<NT, EXT, false>
             : cta == kMixedSmallCta ? path_kernel_mixed<NT, EXT, kMixedSmallCta>
                                     : path_kernel_mixed<NT, EXT, kCta>;
    const size_t smem = poly ? conv_smem_bytes(B) : mixed_smem_bytes(NT, B, cta);
    cudaError_t e = allow_dynamic_smem(k);
    if (e != cudaSuccess) return e;
    const int64_t grid = (M.P.n_paths + cta - 1) / cta;
    k<<<(unsigned)grid, cta, smem, s>>>(M, ext, partials, estore);
    return cudaGetLastError();
}

template <int NT>
static cudaError_t launch_mixed_nt(const MixedParams& M, bool poly, bool cub, const double* ext, double* partials,
                                   float* estore, cudaStream_t s)
{
    return ext ? launch_mixed_t<NT, true>(M, poly, cub, ext, partials, estore, s)
               : launch_mixed_t<NT, false>(M, poly, cub, ext, partials, estore, s);
}

cudaError_t launch_path_mixed(int nt, const MixedParams& M, bool poly, const double* ext, double* partials,
                              float* estore, cudaStream_t s, bool cub)
{
    if (nt == 51) return launch_mixed_nt<51>(M, poly || cub, cub, ext, partials, estore, s);
    if (nt == 61) return launch_mixed_nt<61>(M, poly || cub, cub, ext, partials, estore, s);
    return cudaErrorInvalidValue;
}

bool path_tenor_supported(int nt) { return nt == 51 || nt == 61; }

size_t path_smem(int nt, int n_blocks, bool mixed)
{
    return mixed ? mixed_smem_bytes(nt, n_blocks) : path_smem_bytes(nt, n_blocks, false);  // the larger form
}

int path_cta(bool mixed, int nt, int n_blocks, bool poly)
{
    return mixed ? mixed_cta(nt, n_blocks, poly) : kFp64Cta;
}

cudaError_t launch_reduce(double* partials, int64_t n_rows, int R, double* sums, const FinalParams& F, double* result,
                          cudaStream_t s)
{
    const int64_t ranges = std::max<int64_t>(1, std::min(n_rows / kReduceRows, (int64_t)kReduceRanges));
    reduce_columns<<<dim3((unsigned)R, (unsigned)ranges), kReduceThreads, 0, s>>>(partials, n_rows, R, sums, F, result);
    return cudaGetLastError();
}

cudaError_t launch_dump_normals(int64_t n_paths, uint64_t path_offset, int n_steps, uint32_t k0, uint32_t k1,
                                double* out, cudaStream_t s)
{
    const int64_t total = n_paths * (int64_t)n_steps;
    dump_normals_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(n_paths, path_offset, n_steps, k0, k1, out);
    return cudaGetLastError();
}

cudaError_t launch_philox_words(int64_t n_paths, uint64_t path_offset, uint32_t step, uint32_t k0, uint32_t k1,
                                uint32_t* out, cudaStream_t s)
{
    philox_words_kernel<<<(unsigned)((n_paths + 255) / 256), 256, 0, s>>>(n_paths, path_offset, step, k0, k1, out);
    return cudaGetLastError();
}

cudaError_t launch_transpose_normals(const double* in, int64_t n_paths, int n_steps, double* out, cudaStream_t s)
{
    const int64_t total = n_paths * (int64_t)n_steps * 3;
    transpose_normals_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(in, n_paths, n_steps, out);
    return cudaGetLastError();
}

cudaError_t launch_widen_exposures(const void* in, bool fp64, int64_t ld, int64_t n_paths, int n_dates, double* out,
                                   cudaStream_t s)
{
    const int64_t total = n_paths * (int64_t)n_dates;
    const unsigned g = (unsigned)((total + 255) / 256);
    if (fp64)
        widen_exposures_kernel<double><<<g, 256, 0, s>>>((const double*)in, ld, n_paths, n_dates, out);
    else
        widen_exposures_kernel<float><<<g, 256, 0, s>>>((const float*)in, ld, n_paths, n_dates, out);
    return cudaGetLastError();
}

}  // namespace hjm
