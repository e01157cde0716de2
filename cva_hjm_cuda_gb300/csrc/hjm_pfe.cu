// hjm_pfe.cu -- PFE: the exact k-th smallest exposure of every date column.
//
// Exposures are >= +0, so the order of their IEEE bits as integers is the numeric
// order and selection works on the bits.
//   * Few paths (a column fits one CTA's shared memory): one launch, one CTA
//     per date, a radix selection in shared memory.
//   * Otherwise three launches and one read of the store.  pfe_bracket draws a
//     strided sample of 16,384 keys per date and takes the two sample values six
//     standard deviations either side of the wanted rank; pfe_split counts the
//     keys below the bracket and at its two ends and copies those strictly
//     inside it (a percent or two) to a buffer; pfe_pick selects among them.
//     Keys equal to an end are only counted, so heavily tied columns (most
//     exposures zero) need no buffer at all.  A bracket that misses the rank, or
//     more keys inside it than the buffer holds, makes pfe_pick select from the
//     whole column: the result is exact for any data.
// Bound: few paths, the passes' barriers and launch; many, the store's one read
// and the two single-CTA selections around it.  The radix selection over the
// store it replaces read it three times in 24 launches.  PFE of 21 dates:
// 5,000 paths FP64 350 -> 14 us, 1,048,576 FP64 445 -> 129 us (bracket 46, split
// 43 = 4.1 TB/s, pick 27), 4,194,304 FP32 768 -> 219 us (49, 75 = 4.7 TB/s, 84).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <limits>
#include <type_traits>

#include "hjm_kernels.h"

namespace hjm {

namespace {

constexpr int kThreads = 1024;   // of the selecting CTAs
constexpr int kDigit = 11;
constexpr int kBins = 1 << kDigit;
constexpr int kSample = 16384;   // keys per date the bracket is drawn from
constexpr int kList = 256;       // candidates ranked by comparison
constexpr size_t kColumnBytes = 200 * 1024;  // a column up to this size is selected from shared memory

template <typename K>
constexpr K kTop = std::numeric_limits<K>::max();

struct SelectScratch {
    uint32_t hist[kBins];
    int64_t list[kList];
    int64_t ends[2][kThreads / 32];
    uint32_t warp[kThreads / 32];
    uint32_t digit, before, count, n;
    int64_t out;
};

// Calls f(key) for every key, four loads in flight per thread; every thread of
// the CTA makes every call (key = none beyond the end).
template <typename K, typename F>
__device__ __forceinline__ void for_keys(const K* keys, int64_t m, K none, F f)
{
    for (int64_t base = threadIdx.x; base - threadIdx.x < m; base += 4 * kThreads) {
        K v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t i = base + u * kThreads;
            v[u] = i < m ? keys[i] : none;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) f(v[u]);
    }
}

// The key of rank k (from 0) among m keys >= 0, by all threads of the CTA: the
// keys' range first, then 2,048 equal parts of the range holding the rank, until
// the keys in it are few enough to rank by comparison (ties by position, so
// exactly one has the rank) or all equal.
template <typename K>
__device__ K block_select(const K* keys, int64_t m, uint64_t k, SelectScratch& S)
{
    using U = std::make_unsigned_t<K>;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const K none = -1;
    K lo = kTop<K>, hi = 0;
    for_keys(keys, m, none, [&](K v) {
        if (v >= 0) {
            lo = v < lo ? v : lo;
            hi = v > hi ? v : hi;
        }
    });
    for (int o = 16; o > 0; o >>= 1) {
        const K a = __shfl_xor_sync(0xffffffffu, lo, o), b = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
    }
    __syncthreads();  // (the scratch's last use)
    if (lane == 0) {
        S.ends[0][warp] = lo;
        S.ends[1][warp] = hi;
    }
    __syncthreads();
    lo = (K)S.ends[0][lane];
    hi = (K)S.ends[1][lane];
    for (int o = 16; o > 0; o >>= 1) {
        const K a = __shfl_xor_sync(0xffffffffu, lo, o), b = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
    }
    // the keys v with (U)(v - lo) >> width == 0 hold the rank
    int width = lo == hi ? 0 : 64 - __clzll((long long)(hi - lo));
    while (width > 0) {
        const int shift = width > kDigit ? width - kDigit : 0;
        for (int i = t; i < kBins; i += kThreads) S.hist[i] = 0;
        __syncthreads();
        for_keys(keys, m, none, [&](K v) {
            const U d = (U)(v - lo);
            const bool take = v >= lo && (width >= 8 * (int)sizeof(K) || (d >> width) == 0);
            const uint32_t digit = (uint32_t)(d >> shift);
            const uint32_t active = __ballot_sync(0xffffffffu, take);
            if (take) {  // one atomic per distinct digit of the warp
                const uint32_t peers = __match_any_sync(active, digit);
                if (lane == __ffs(peers) - 1) atomicAdd(&S.hist[digit], (uint32_t)__popc(peers));
            }
        });
        __syncthreads();
        // the part whose cumulative count passes k: prefix sum, two parts a thread
        const uint32_t h0 = S.hist[2 * t], h1 = S.hist[2 * t + 1];
        uint32_t incl = h0 + h1;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) S.warp[warp] = incl;
        __syncthreads();
        uint32_t sums = S.warp[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, sums, o);
            if (lane >= o) sums += v;
        }
        const uint32_t prev = __shfl_sync(0xffffffffu, sums, warp > 0 ? warp - 1 : 0);
        const uint64_t before = (uint64_t)(warp > 0 ? prev : 0) + incl - (h0 + h1);
        if (before <= k && k < before + h0 + h1) {
            const bool second = k >= before + h0;
            S.digit = 2 * t + second;
            S.before = (uint32_t)(before + (second ? h0 : 0));
            S.count = second ? h1 : h0;
            S.n = 0;
        }
        __syncthreads();
        lo += (K)((U)S.digit << shift);
        k -= S.before;
        width = shift;
        const uint32_t count = S.count;
        __syncthreads();
        if (width > 0 && count <= kList) {
            for_keys(keys, m, none, [&](K v) {
                if (v >= lo && ((U)(v - lo) >> width) == 0) S.list[atomicAdd(&S.n, 1u)] = v;
            });
            __syncthreads();
            if (t < (int)count) {
                const int64_t v = S.list[t];
                uint32_t rank = 0;
                for (uint32_t j = 0; j < count; ++j) rank += (S.list[j] < v) || (S.list[j] == v && (int)j < t);
                if (rank == k) S.out = v;
            }
            __syncthreads();
            return (K)S.out;
        }
    }
    return lo;
}

__device__ __forceinline__ double key_value(int64_t k) { return __longlong_as_double((long long)k); }
__device__ __forceinline__ double key_value(int32_t k) { return (double)__int_as_float(k); }

// One CTA per date; the dates beyond are zero
template <typename K>
__device__ void write_result(double* result, int date, int n_dates, K key)
{
    if (threadIdx.x == 0) result[kResPFE + date] = key_value(key);
    if (date == 0)
        for (int j = n_dates + threadIdx.x; j < kMaxTenor; j += blockDim.x) result[kResPFE + j] = 0.0;
}

template <typename K>
__global__ void __launch_bounds__(kThreads)
    pfe_column(const K* __restrict__ keys, int64_t ld, int n, int n_dates, uint64_t k, double* __restrict__ result)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SelectScratch S;
    K* col = reinterpret_cast<K*>(smem);
    const K* src = keys + (size_t)blockIdx.x * (size_t)ld;
    for (int i = threadIdx.x; i < n; i += kThreads) col[i] = src[i];
    __syncthreads();
    write_result(result, blockIdx.x, n_dates, block_select(col, n, k, S));
}

// The bracket of one date from keys 0, step, 2 step, ...: sample ranks r0 and r1
// (r0 < 0 or r1 >= n_sample: open at that end, beyond every key)
template <typename K>
__global__ void __launch_bounds__(kThreads)
    pfe_bracket(const K* __restrict__ keys, int64_t ld, int64_t step, int n_sample, int r0, int r1,
                SelState* __restrict__ st)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SelectScratch S;
    K* col = reinterpret_cast<K*>(smem);
    const K* src = keys + (size_t)blockIdx.x * (size_t)ld;
#pragma unroll 4
    for (int i = threadIdx.x; i < n_sample; i += kThreads) col[i] = src[(size_t)i * (size_t)step];
    __syncthreads();
    SelState x = {};
    x.lo = r0 < 0 ? -1 : (int64_t)block_select(col, n_sample, (uint64_t)r0, S);
    x.hi = r1 >= n_sample ? (int64_t)kTop<K> : (int64_t)block_select(col, n_sample, (uint64_t)r1, S);
    if (threadIdx.x == 0) st[blockIdx.x] = x;
}

// Counts at the bracket's ends and above its lower end; the keys strictly
// inside it to the date's buffer (beyond its capacity they are only counted),
// gathered per CTA in shared memory first.  Most keys of a high quantile lie
// below the bracket: they take a load and a comparison, four keys a load (rows
// are padded to four).
template <typename K>
__global__ void __launch_bounds__(256)
    pfe_split(const K* __restrict__ keys, int64_t ld, int64_t n, SelState* __restrict__ st, K* __restrict__ buf,
              int64_t cap)
{
    struct alignas(16) Quad {
        K k[4];
    };
    constexpr uint32_t kGather = 4096;
    __shared__ K gather[kGather];
    __shared__ uint32_t n_gather, n_lo, n_hi, n_above;
    __shared__ unsigned long long at_s;
    const int date = blockIdx.y;
    const K lo = (K)st[date].lo, hi = (K)st[date].hi;
    const Quad* col = reinterpret_cast<const Quad*>(keys + (size_t)date * (size_t)ld);
    K* out = buf + (size_t)date * (size_t)cap;
    if (threadIdx.x == 0) n_gather = n_lo = n_hi = n_above = 0;
    __syncthreads();
    uint32_t at_lo = 0, at_hi = 0, above = 0;
    auto rest = [&](K v) {  // v >= lo
        if (v == lo) {
            ++at_lo;
        } else if (v < hi) {
            const uint32_t at = atomicAdd(&n_gather, 1u);
            if (at < kGather) {
                gather[at] = v;
            } else {
                const int64_t pos = (int64_t)atomicAdd(&st[date].inside, 1ull);
                if (pos < cap) out[pos] = v;
            }
        } else if (v == hi) {
            ++at_hi;
        } else {
            ++above;
        }
    };
    const int64_t quads = n / 4, stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll 2
    for (int64_t i = first; i < quads; i += stride) {
        const Quad v = col[i];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v.k[u] >= lo) rest(v.k[u]);
    }
    if (first < n - 4 * quads) {  // the row's last few keys
        const K v = keys[(size_t)date * (size_t)ld + (size_t)(4 * quads + first)];
        if (v >= lo) rest(v);
    }
    at_lo = __reduce_add_sync(0xffffffffu, at_lo);
    at_hi = __reduce_add_sync(0xffffffffu, at_hi);
    above = __reduce_add_sync(0xffffffffu, above);
    if ((threadIdx.x & 31) == 0) {
        if (at_lo) atomicAdd(&n_lo, at_lo);
        if (at_hi) atomicAdd(&n_hi, at_hi);
        if (above) atomicAdd(&n_above, above);
    }
    __syncthreads();
    const uint32_t m = min(n_gather, kGather);
    if (threadIdx.x == 0) {
        at_s = m ? atomicAdd(&st[date].inside, (unsigned long long)m) : 0ull;
        if (n_lo) atomicAdd(&st[date].at_lo, (unsigned long long)n_lo);
        if (n_hi) atomicAdd(&st[date].at_hi, (unsigned long long)n_hi);
        if (n_above) atomicAdd(&st[date].above, (unsigned long long)n_above);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
        const int64_t pos = (int64_t)at_s + i;
        if (pos < cap) out[pos] = gather[i];
    }
}

template <typename K>
__global__ void __launch_bounds__(kThreads)
    pfe_pick(const K* __restrict__ keys, int64_t ld, int64_t n, int n_dates, uint64_t k, const SelState* __restrict__ st,
             const K* __restrict__ buf, int64_t cap, double* __restrict__ result)
{
    __shared__ SelectScratch S;
    const int date = blockIdx.x;
    const SelState x = st[date];
    const uint64_t below = (uint64_t)n - x.at_lo - x.inside - x.at_hi - x.above, r = k - below;
    K key;
    if (k >= below && r < x.at_lo) {
        key = (K)x.lo;
    } else if (k >= below && r - x.at_lo < x.inside && (int64_t)x.inside <= cap) {
        key = block_select(buf + (size_t)date * (size_t)cap, (int64_t)x.inside, r - x.at_lo, S);
    } else if (k >= below && r - x.at_lo >= x.inside && r - x.at_lo - x.inside < x.at_hi) {
        key = (K)x.hi;
    } else {  // the bracket missed the rank, or overflowed: the whole column
        key = block_select(keys + (size_t)date * (size_t)ld, n, k, S);
    }
    write_result(result, date, n_dates, key);
}

bool fits_column(int64_t n, size_t key_bytes) { return (size_t)n * key_bytes <= kColumnBytes; }

// candidates a date's buffer holds: several times the 1.5 % the bracket of the
// 97.5 % quantile takes (4.7 % for the median)
int64_t capacity(int64_t n) { return (n / 12 + 1023) / 1024 * 1024; }

template <typename K>
cudaError_t select_t(const K* keys, int64_t ld, int64_t n, int n_dates, uint64_t k, SelState* st, K* buf,
                     size_t buf_bytes, double* result, int n_sms, cudaStream_t s, int* launches)
{
    if (fits_column(n, sizeof(K))) {
        const size_t smem = (size_t)n * sizeof(K);
        cudaError_t e = allow_dynamic_smem(pfe_column<K>, kColumnBytes);
        if (e != cudaSuccess) return e;
        pfe_column<K><<<n_dates, kThreads, smem, s>>>(keys, ld, (int)n, n_dates, k, result);
        *launches = 1;
        return cudaGetLastError();
    }
    // (n > 25,000 here: the sample is a proper one)
    const int m = (int)std::min<int64_t>(n, kSample);
    const int64_t step = n / m;
    const double q = ((double)k + 0.5) / (double)n;
    const double mid = q * m, half = 6.0 * std::sqrt((double)m * q * (1.0 - q)) + 8.0;
    const int r0 = (int)std::floor(mid - half), r1 = (int)std::ceil(mid + half);
    const size_t smem = (size_t)m * sizeof(K);
    cudaError_t e = allow_dynamic_smem(pfe_bracket<K>, kSample * sizeof(K));
    if (e != cudaSuccess) return e;
    pfe_bracket<K><<<n_dates, kThreads, smem, s>>>(keys, ld, step, m, r0, r1, st);
    // eight CTAs per SM over all dates, each with at least a few thousand keys
    const int64_t gx = std::max<int64_t>(1, std::min<int64_t>((n + 4095) / 4096, (int64_t)n_sms * 8 / n_dates));
    const int64_t cap = std::min<int64_t>(capacity(n), (int64_t)(buf_bytes / (sizeof(K) * (size_t)n_dates)));
    pfe_split<K><<<dim3((unsigned)gx, (unsigned)n_dates), 256, 0, s>>>(keys, ld, n, st, buf, cap);
    pfe_pick<K><<<n_dates, kThreads, 0, s>>>(keys, ld, n, n_dates, k, st, buf, cap, result);
    *launches = 3;
    return cudaGetLastError();
}

}  // namespace

size_t pfe_scratch_bytes(int64_t n, int n_dates, bool fp64_keys)
{
    const size_t key = fp64_keys ? 8 : 4;
    return fits_column(n, key) ? 0 : key * (size_t)capacity(n) * (size_t)n_dates;
}

cudaError_t launch_pfe(const void* estore, bool fp64_keys, int64_t ld, int64_t n_paths, int n_dates, uint64_t k0,
                       SelState* st, void* scratch, size_t scratch_bytes, double* result, int n_sms, cudaStream_t s,
                       int* launches)
{
    return fp64_keys ? select_t((const int64_t*)estore, ld, n_paths, n_dates, k0, st, (int64_t*)scratch,
                                scratch_bytes, result, n_sms, s, launches)
                     : select_t((const int32_t*)estore, ld, n_paths, n_dates, k0, st, (int32_t*)scratch,
                                scratch_bytes, result, n_sms, s, launches);
}

}  // namespace hjm
