// hjm_adjoint_run.cu -- the adjoint of the CVA in one pass over the steps.
//
// The adjoint in the response form (Euler step, quadratic factors, the sampled
// states kept: checkpoint_every = 0), in one pass over the steps.  The forward
// values are the mixed valuation's response form (path_kernel_mixed_resp,
// hjm_mresp.cu: the parts S, U, W as FP32 scalars, the remainder as FP32
// impulse-response sums in NS date slots, the same operations in the same
// order, so the path's cash flows are the valuation's).
//
// A date's sampled forward x_i and discount sum a_i are linear in the loadings
// a_kd of factor k on T^d, so their derivatives run along with the path
// instead of a reverse sweep that draws every normal a second time.  With
//     r0 = sum phi_k,  r1 = sum r0,  r2 = sum r1,  r3 = sum r2
// (each step adds the values before it) and t the date's tenor,
//     dx/da_k0 = r0
//     dx/da_k1 = t r0 + k1 r1                                (k1 = c dtau)
//     dx/da_k2 = t^2 r0 + (2 k1 t + k2) r1 + 2 k1^2 r2 + Y_kx   (k2 = c dtau^2)
// and the discount sum's are the same with r0 + r1, r1 + r2, r2 + r3 and Y_ky
// in place of r0, r1, r2 and Y_kx: the parts' update rules with a unit
// loading.  Y_k = sum_n {kappa G_j, kappa CG_j}(n) r0(n) is the remainder's
// response to W = r0: the table row and the slots of A, once per factor.
// The twelve sums of a date go to memory (a part of sens per CTA, rewritten
// tile by tile, 71 MB for 20 dates: 95 MB of write-backs to DRAM at 262,144 paths, reads
// from the second-level cache) until the seeds {xbar_i, abar_i}, which need the exposures
// of the whole path, weigh them.
//
// Bounds: the generator (115 of ~165 issue cycles per 32 path-steps), then the
// packed FMAs of Y.  10y swap, 1M paths: 8.35 ms -> 5.75 ms against the
// two-pass form; 12y (16 slots), 512k paths: 6.37 -> 4.83 ms; 5,000 paths: 0.58 ->
// 0.38 ms.  Eight CTAs per SM with the widest loop unrolled by 2: by 5 its
// three bodies outgrow the instruction cache (6.15 ms); seven CTAs leave one
// scheduler a warp more (6.69), six take 5.85.  Slots dropped by quarters
// instead of halves: 5.77 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "hjm_adjoint.cuh"
#include "hjm_device.cuh"
#include "hjm_kernels.h"
#include "hjm_pairs.cuh"

namespace hjm {

struct AdjRespLayout {
    size_t cf, xs, ds, red, total;
};

__host__ __device__ inline AdjRespLayout adj_resp_layout(int B, int R)
{
    AdjRespLayout L;
    const size_t rows = (size_t)B + 1;
    L.cf = 0;
    L.xs = align128((rows + 1) * kAdjCta * 4);
    L.ds = align128(L.xs + rows * kAdjCta * 4);
    L.red = align128(L.ds + rows * kAdjCta * 4);
    L.total = align128(L.red + (size_t)(kAdjCta / 32) * R * 8);
    return L;
}

// A path's derivatives with respect to the loadings.
template <int NS>
struct PathSens {
    float2 Y[kFactors][NS];  // {hc at date j's tenor, its running sum} per unit of factor k's T^2 loading, slot B - j
    float r0[kFactors], r1[kFactors], r2[kFactors], r3[kFactors];

    __device__ __forceinline__ void reset()
    {
#pragma unroll
        for (int k = 0; k < kFactors; ++k) {
            r0[k] = r1[k] = r2[k] = r3[k] = 0.f;
#pragma unroll
            for (int r = 0; r < NS; ++r) Y[k][r] = make_float2(0.f, 0.f);
        }
    }
    // a step's responses of slots 2u, 2u + 1 (before its sums)
    __device__ __forceinline__ void respond(int u, float2 e0, float2 e1)
    {
#pragma unroll
        for (int k = 0; k < kFactors; ++k) {
            const float2 p2 = make_float2(r0[k], r0[k]);
            Y[k][2 * u] = __ffma2_rn(e0, p2, Y[k][2 * u]);
            Y[k][2 * u + 1] = __ffma2_rn(e1, p2, Y[k][2 * u + 1]);
        }
    }
    __device__ __forceinline__ void advance(float phi0, float phi1, float phi2)
    {
        const float ph[kFactors] = {phi0, phi1, phi2};
#pragma unroll
        for (int k = 0; k < kFactors; ++k) {
            r3[k] += r2[k];
            r2[k] += r1[k];
            r1[k] += r0[k];
            r0[k] += ph[k];
        }
    }
    // the sums at the date of block b's end
    __device__ __forceinline__ void store(float4* sens_p, int b) const
    {
#pragma unroll
        for (int k = 0; k < kFactors; ++k)
            sens_p[((size_t)(b - 1) * kFactors + k) * kAdjCta] = make_float4(r0[k], r1[k], r2[k], r3[k]);
    }
};

// A tile's end, for both forward forms: exposures (cash flows cf, rows 1..B of
// kAdjCta columns; e_s may lie one row above a float cf), EE and CVA sums,
// seeds, the coefficients' sums and the partial row `out`.
template <int NS>
__device__ __forceinline__ void adjoint_tile_end(const MixedParams& M, const float* cf_s, float* e_s, float* xs_s,
                                                 float* ds_s, double* red_s, const float4* sens_p,
                                                 const PathSens<NS>& sn, bool active, double* __restrict__ out)
{
    constexpr int C = kAdjCta;
    const PathParams<float>& P = M.P;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int B = P.n_blocks, R = 3 * B + 12;
    double v = 0.0, cva_c = 0.0;
    e_s[B * C + tid] = 0.f;
    for (int j = B - 1; j >= 0; --j) {
        v += (double)cf_s[(j + 1) * C + tid];
        double e = (v > 0.0) ? v : 0.0;
        if (!active) e = 0.0;
        e_s[j * C + tid] = (float)e;
        cva_c = fma(P.cvaw[j], e, cva_c);
    }
    __syncthreads();
    for (int j = warp; j <= B; j += C / 32) {
        double sum = 0.0;
#pragma unroll
        for (int q = 0; q < C / 32; ++q) sum += (double)e_s[j * C + lane + 32 * q];
        sum = warp_sum(sum);
        if (lane == 0) out[j] = sum;
    }
    {
        const double s1 = warp_sum(cva_c), s2 = warp_sum(cva_c * cva_c);
        if (lane == 0) {
            red_s[warp * R + B + 1] = s1;
            red_s[warp * R + B + 2] = s2;
        }
    }

    // per-date seeds from cfbar_i = sum_{j<i} w_j [E_j > 0], and the
    // coefficients' sums in FP32 pairs (hi + lo)
    float hi[3 * kFactors] = {}, lo[3 * kFactors] = {};
    auto add = [&](int q, float val) {
        const float t = hi[q] + val, z = t - hi[q];
        lo[q] += (hi[q] - (t - z)) + (val - z);
        hi[q] = t;
    };
    float cfbar = 0.f;
    for (int i = 1; i <= B; ++i) {
        const int j = i - 1;
        if (e_s[j * C + tid] > 0.f) cfbar += (float)P.cvaw[j];
        if (!active) cfbar = 0.f;
        float xb, ab;
        date_seeds(P, i, (double)xs_s[i * C + tid], ds_s[i * C + tid], cfbar, xb, ab);
        xs_s[i * C + tid] = xb;
        ds_s[i * C + tid] = ab;
        if (i == 1) continue;
        const float ti = P.tau[i];
        const float t2 = ti * ti, t1 = fmaf(2.f * M.k1f, ti, M.k2f), t0 = 2.f * M.k1f * M.k1f;
#pragma unroll
        for (int k = 0; k < kFactors; ++k) {
            const float4 m = sens_p[((size_t)(i - 2) * kFactors + k) * C];
            const float v0 = fmaf(xb, m.x, ab * (m.x + m.y));
            const float v1 = fmaf(xb, m.y, ab * (m.y + m.z));
            const float v2 = fmaf(xb, m.z, ab * (m.z + m.w));
            add(3 * k, v0);
            add(3 * k + 1, fmaf(ti, v0, M.k1f * v1));
            add(3 * k + 2, fmaf(t2, v0, fmaf(t1, v1, t0 * v2)));
        }
    }
    // the remainder's share of the T^2 loadings
    {
        float c2[kFactors] = {};
#pragma unroll
        for (int r = 0; r < NS; ++r) {
            const int j = B - r;
            if (j >= 2) {
                const float xb = xs_s[j * C + tid], ab = ds_s[j * C + tid];
#pragma unroll
                for (int k = 0; k < kFactors; ++k) c2[k] = fmaf(xb, sn.Y[k][r].x, fmaf(ab, sn.Y[k][r].y, c2[k]));
            }
        }
#pragma unroll
        for (int k = 0; k < kFactors; ++k) add(3 * k + 2, c2[k]);
    }

    // columns as adjoint_kernel's: [0..B] EE, B+1/B+2 CVA stats, E xbar_i,
    // E abar_i (i = 1..B), the 9 coefficient columns
    const int cx = B + 3, ca = 2 * B + 3, cc = 3 * B + 3;
    for (int i = 1; i <= B; ++i) {
        const double sx = warp_sum((double)xs_s[i * C + tid]);
        const double sa = warp_sum((double)ds_s[i * C + tid]);
        if (lane == 0) {
            red_s[warp * R + cx + i - 1] = sx;
            red_s[warp * R + ca + i - 1] = sa;
        }
    }
#pragma unroll
    for (int q = 0; q < 3 * kFactors; ++q) {
        const double sum = warp_sum((double)hi[q] + (double)lo[q]);
        if (lane == 0) red_s[warp * R + cc + q] = sum;
    }
    __syncthreads();
    for (int col = B + 1 + tid; col < R; col += C) {
        double sum = 0.0;
        for (int w = 0; w < C / 32; ++w) sum += red_s[w * R + col];
        out[col] = sum;
    }
}

// CTAs per SM: four warps per scheduler with 8 slots (128 registers), two with
// 16 (255 registers; five CTAs spill, 6.8 ms at 512k paths of the 12y swap)
constexpr int adj_resp_ctas(int ns) { return ns <= 8 ? 8 : 4; }

template <int NS>
__global__ void __launch_bounds__(kAdjCta, adj_resp_ctas(NS))
    adjoint_kernel_resp(const __grid_constant__ MixedParams M, const RespLive live,
                        const float4* __restrict__ resp, float4* __restrict__ sens, double* __restrict__ partials,
                        int64_t n_tiles)
{
    constexpr int C = kAdjCta;
    const PathParams<float>& P = M.P;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x;
    const int B = P.n_blocks;
    const int R = 3 * B + 12;
    const AdjRespLayout Ly = adj_resp_layout(B, R);
    float* cf_s = reinterpret_cast<float*>(smem + Ly.cf);  // [B+2][C]: cash flows, then exposures one row up
    float* xs_s = reinterpret_cast<float*>(smem + Ly.xs);  // [B+1][C]: x_i, then xbar_i
    float* ds_s = reinterpret_cast<float*>(smem + Ly.ds);  // [B+1][C]: D_i, then abar_i
    double* red_s = reinterpret_cast<double*>(smem + Ly.red);  // [warp][R]
    float4* sens_p = sens + (size_t)blockIdx.x * (B - 1) * kFactors * C + tid;  // [date - 2][factor][C]
    const int stride = P.stride;
    const int n_last = B * stride - 1;

    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const int64_t lp = tile * C + tid;
        const bool active = lp < P.n_paths;
        const uint64_t gpath = P.path_offset + (uint64_t)lp;

        float2 A[NS];  // {hc at date j's tenor, its running sum}, slot B - j
#pragma unroll
        for (int r = 0; r < NS; ++r) A[r] = make_float2(0.f, 0.f);
        PathSens<NS> sn;
        sn.reset();
        float S = 0.f, U = 0.f, W = 0.f;
        double zS = 0.0, zU = 0.0, zW = 0.0;
        auto price = [&](int i, float2 rc) {
            const float ti = P.tau[i];
            const float pv = fmaf(ti, fmaf(ti, W, U), S);
            const double xv = P.psamp[i] + (double)(rc.x + pv);
            const double td = (double)ti;
            const double a = P.psum[i] + (double)rc.y + fma(td, fma(td, zW, zU), zS);
            const float D = expf((float)(-a * P.dt));
            const float mm = (float)P.m;
            const float L = mm * expm1f((float)xv / mm);
            cf_s[i * C + tid] = D * ((float)P.payA[i] * L - (float)P.payB[i]);
            xs_s[i * C + tid] = (float)xv;
            ds_s[i * C + tid] = D;
        };
        price(1, make_float2(0.f, 0.f));
        float q0, q1, q2;
        draw_phi<float, false>(nullptr, gpath, lp, P.n_paths, min(stride, n_last), P.rk0, P.rk1, q0, q1, q2);
        float sS, sU, sW;
        auto steps = [&](auto live_c, int b) {  // (the values as path_kernel_mixed_resp's)
            constexpr int LIVE = decltype(live_c)::value;
            const float4* row = resp + (size_t)b * stride * (NS / 2);
#pragma unroll(NS == 8 && LIVE == NS ? 2 : 5)
            for (int s = 0; s < stride; ++s) {
                const int n = b * stride + s;
                const float phi0 = q0, phi1 = q1, phi2 = q2;
                draw_phi<float, false>(nullptr, gpath, lp, P.n_paths, min(n + 1, n_last), P.rk0, P.rk1, q0, q1, q2);
                const float2 w2 = make_float2(W, W);
                const float4* rr = row + (size_t)s * (NS / 2);
#pragma unroll
                for (int u = 0; u < LIVE / 2; ++u) {
                    const float4 e = __ldg(rr + u);
                    const float2 e0 = make_float2(e.x, e.y), e1 = make_float2(e.z, e.w);
                    A[2 * u] = __ffma2_rn(e0, w2, A[2 * u]);
                    A[2 * u + 1] = __ffma2_rn(e1, w2, A[2 * u + 1]);
                    sn.respond(u, e0, e1);
                }
                float Sn = fmaf(M.svcf[0][0], phi0, fmaf(M.k2f, W, fmaf(M.k1f, U, S)));
                Sn = fmaf(M.svcf[2][0], phi2, fmaf(M.svcf[1][0], phi1, Sn));
                float Un = fmaf(M.svcf[1][1], phi1, fmaf(M.svcf[0][1], phi0, fmaf(2.0f * M.k1f, W, U)));
                Un = fmaf(M.svcf[2][1], phi2, Un);
                const float Wn = fmaf(M.svcf[2][2], phi2, fmaf(M.svcf[1][2], phi1, fmaf(M.svcf[0][2], phi0, W)));
                S = Sn;
                U = Un;
                W = Wn;
                sS += S;
                sU += U;
                sW += W;
                sn.advance(phi0, phi1, phi2);
            }
        };
        for (int b = 1; b < B; ++b) {
            sS = sU = sW = 0.f;
            if (b < live.half)
                steps(std::integral_constant<int, NS>(), b);
            else if (b < live.none)
                steps(std::integral_constant<int, NS / 2>(), b);
            else
                steps(std::integral_constant<int, 0>(), b);
            zS += (double)sS;
            zU += (double)sU;
            zW += (double)sW;
            const int r = B - (b + 1);
            price(b + 1, r < NS ? select_reg<NS, float2>(A, r) : make_float2(0.f, 0.f));
            sn.store(sens_p, b);
        }

        adjoint_tile_end<NS>(M, cf_s, cf_s + C, xs_s, ds_s, red_s, sens_p, sn, active, partials + (size_t)tile * R);
        __syncthreads();  // (the next tile writes the rows and sums just read)
    }
}

// The same for the convected form (checkpoint_every > 0 where the dates the
// remainder reaches fit the slots): the values are path_kernel_mixed_conv's
// (stepped whole, which leaves the window's tenors as they are), the derivatives
// as above, so no state is kept and no normal drawn twice.
//
// Checkpoints every 32 steps on the 10y swap, 256k paths: 4.45 ms with the
// state written, the segments recomputed and the sweep -> 2.00 ms (of which
// the convected valuation is 1.3); 12y (16 slots) 3.01 ms.  Whole warps per
// scheduler: 6 CTAs with 8 slots (168 registers; 7 take 2.96 ms, 4 2.42),
// 4 with 16 or with 61 tenors; steps unrolled by 2 (by 1 2.18, by 5 2.20).  The
// window's start as a constant of the loop: selected per step 2.16 ms.
constexpr int adj_conv_ctas(int ns, int nt) { return ns <= 8 && nt <= 56 ? 6 : 4; }

template <int NS, int NT>
__global__ void __launch_bounds__(kAdjCta, adj_conv_ctas(NS, NT))
    adjoint_kernel_conv(const __grid_constant__ MixedParams M, const RespLive live,
                        const float4* __restrict__ resp, float4* __restrict__ sens, double* __restrict__ partials,
                        int64_t n_tiles)
{
    constexpr int C = kAdjCta;
    constexpr int W1 = conv_window(NT, 0), W2 = conv_window(NT, 1);
    const PathParams<float>& P = M.P;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x;
    const int B = P.n_blocks;
    const int R = 3 * B + 12;
    const AdjRespLayout Ly = adj_resp_layout(B, R);
    float* cf_s = reinterpret_cast<float*>(smem + Ly.cf);
    float* xs_s = reinterpret_cast<float*>(smem + Ly.xs);
    float* ds_s = reinterpret_cast<float*>(smem + Ly.ds);
    double* red_s = reinterpret_cast<double*>(smem + Ly.red);
    // (in shared memory: read and written once a block)
    LongSums<NT, false>& z = reinterpret_cast<LongSums<NT, false>*>(smem + align128(Ly.total))[tid];
    float4* sens_p = sens + (size_t)blockIdx.x * (B - 1) * kFactors * C + tid;
    const int stride = P.stride;
    const int n_last = B * stride - 1;

    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const int64_t lp = tile * C + tid;
        const bool active = lp < P.n_paths;
        const uint64_t gpath = P.path_offset + (uint64_t)lp;
        MixedPath<NT, true> x;
        x.reset();
        PathSens<NS> sn;
        sn.reset();
        z.reset();
        auto price = [&](int i, float value, double sum) {
            const double xv = P.psamp[i] + (double)value;
            const double a = P.psum[i] + sum;
            const float D = expf((float)(-a * P.dt));
            const float mm = (float)P.m;
            const float L = mm * expm1f((float)xv / mm);
            cf_s[i * C + tid] = D * ((float)P.payA[i] * L - (float)P.payB[i]);
            xs_s[i * C + tid] = (float)xv;
            ds_s[i * C + tid] = D;
        };
        price(1, 0.f, 0.0);
        float q0, q1, q2;
        draw_phi<float, false>(nullptr, gpath, lp, P.n_paths, min(stride, n_last), P.rk0, P.rk1, q0, q1, q2);
        BlockSums bs;
        // block b with the first LIVE slots' responses, on the tenors from S0 (0:
        // on all, the window's start w selected)
        auto steps = [&](auto live_c, auto s0_c, int b, int w) {
            constexpr int LIVE = decltype(live_c)::value, S0 = decltype(s0_c)::value;
            const float4* row = resp + (size_t)b * stride * (NS / 2);
#pragma unroll 2
            for (int s = 0; s < stride; ++s) {
                const int n = b * stride + s;
                const float phi0 = q0, phi1 = q1, phi2 = q2;
                draw_phi<float, false>(nullptr, gpath, lp, P.n_paths, min(n + 1, n_last), P.rk0, P.rk1, q0, q1, q2);
                const float4* rr = row + (size_t)s * (NS / 2);
#pragma unroll
                for (int u = 0; u < LIVE / 2; ++u) {
                    const float4 e = __ldg(rr + u);
                    sn.respond(u, make_float2(e.x, e.y), make_float2(e.z, e.w));
                }
                sn.advance(phi0, phi1, phi2);
                x.template step<S0>(M, phi0, phi1, phi2);
                bs.add_at(x, S0        ? pair_tenor<NT>(x.h, S0)
                             : w == W2 ? pair_tenor<NT>(x.h, W2)
                                       : pair_tenor<NT>(x.h, W1));
            }
        };
        for (int b = 1; b < B; ++b) {
            bs.reset();
            const int w = window_start<NT>(M, b);
            if (w != z.start) z.move(x, P, w);
            x.begin_block(P, b);
            using std::integral_constant;
            const integral_constant<int, NS> all;
            const integral_constant<int, NS / 2> half;
            const integral_constant<int, 0> none;
            const integral_constant<int, 1> whole;
            if (b < live.none && w > 1)
                steps(all, none, b, w);
            else if (b < live.half)
                steps(all, whole, b, w);
            else if (b < live.none)
                steps(half, whole, b, w);
            else if (w == 1)
                steps(none, whole, b, w);
            else if (w == W1)
                steps(none, integral_constant<int, W1>(), b, w);
            else
                steps(none, integral_constant<int, W2>(), b, w);
            z.fold(bs.H1, bs.sS, bs.sU, bs.sW, 0.f);
            float value;
            double sum;
            z.template read<1>(x, P, z.start, b + 1, value, sum);
            price(b + 1, value, sum);
            sn.store(sens_p, b);
        }
        adjoint_tile_end<NS>(M, cf_s, cf_s + C, xs_s, ds_s, red_s, sens_p, sn, active, partials + (size_t)tile * R);
        __syncthreads();  // (the next tile writes the rows and sums just read)
    }
}

// (the convected form's running sums behind the layout)
size_t adjoint_resp_smem(int n_blocks, int conv_nt)
{
    return adj_resp_layout(n_blocks, 3 * n_blocks + 12).total + (conv_nt ? sizeof(LongSums<51, false>) * kAdjCta : 0);
}

// conv_nt: the tenors of the convected forward form, 0 for the response form

int adjoint_resp_grid(int64_t n_paths, int ns, int conv_nt, int n_sms)
{
    const int ctas = conv_nt ? adj_conv_ctas(ns, conv_nt) : adj_resp_ctas(ns);
    return (int)std::min((n_paths + kAdjCta - 1) / kAdjCta, (int64_t)n_sms * ctas);
}

size_t adjoint_resp_sens_bytes(int n_blocks, int grid)
{
    return sizeof(float4) * kFactors * kAdjCta * (size_t)(n_blocks - 1) * (size_t)grid;
}

cudaError_t launch_adjoint_resp(const AdjParams& A, int ns, int conv_nt, const RespLive& live, const float4* table,
                                float4* sens, int grid, double* partials, cudaStream_t s)
{
    const int B = A.M.P.n_blocks;
    if ((ns != 8 && ns != 16) || B < 1 || B >= kMaxTenor || A.M.P.stride < 1 || grid < 1) return cudaErrorInvalidValue;
    decltype(&adjoint_kernel_resp<8>) k = nullptr;
    if (conv_nt == 0) k = ns == 8 ? adjoint_kernel_resp<8> : adjoint_kernel_resp<16>;
    if (conv_nt == 51) k = ns == 8 ? adjoint_kernel_conv<8, 51> : adjoint_kernel_conv<16, 51>;
    if (conv_nt == 61) k = ns == 8 ? adjoint_kernel_conv<8, 61> : adjoint_kernel_conv<16, 61>;
    if (!k) return cudaErrorInvalidValue;
    const size_t smem = adjoint_resp_smem(B, conv_nt);
    cudaError_t e = allow_dynamic_smem(k);
    if (e != cudaSuccess) return e;
    const int64_t tiles = (A.M.P.n_paths + kAdjCta - 1) / kAdjCta;
    k<<<(unsigned)grid, kAdjCta, smem, s>>>(A.M, live, table, sens, partials, tiles);
    return cudaGetLastError();
}

}  // namespace hjm
