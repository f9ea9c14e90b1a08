// One-off calibration kernels: the exact integer histogram of block-normalised gradients, the
// block-period scores and the Lloyd-Max accumulation / MSE kernels.
//
// Reference behaviour:
//   histogram   kernels/exact_histogram_fused_kernel.cu:17-85
//   scores      kernels/period_variance_kernel.cu:13-165 and the host post-ops at :242, :311-317, :392-395
//   Lloyd-Max   kernels/lloyd_max_fused_kernel.cu:50-195
//
// All of them are one read of the gradient from HBM (the reference reads it twice per kernel and,
// for the adjacent-log score, twice per candidate period; here once per candidate that no other one
// divides, one to six per tensor). A warp owns a block; the second look at
// a block's elements, where one is needed, comes from L1.
#include "common.cuh"

#include <string.h>

#include <algorithm>
#include <new>
#include <vector>

namespace gefen {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

static int persistent_grid(long long groups, int groups_per_cta, int ctas_per_sm) {
    long long ctas = (groups + groups_per_cta - 1) / groups_per_cta;
    const long long cap = static_cast<long long>(sm_count()) * ctas_per_sm;
    if (ctas > cap) ctas = cap;
    if (ctas < 1) ctas = 1;
    return static_cast<int>(ctas);
}

// NaN-ignoring max |g| over one block, by one warp (GROUP=32) or one CTA (GROUP=256).
template <typename S, int GROUP>
__device__ __forceinline__ float block_absmax(const S* g, long long period, int tig, float* red) {
    float m = 0.0f;
    for (long long i = tig; i < period; i += GROUP) m = fmaxf(m, fabsf(ScalarIO<S>::load(g + i)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (GROUP > 32) {
        __syncthreads();
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
        m = red[0];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) m = fmaxf(m, red[w]);
    }
    return m;
}

// ------------------------------------------------------------------------------- vector access
// Eight consecutive elements (16 bytes of a 2-byte type, 32 bytes of fp32) as floats; the pointer is
// 16-byte aligned. Calibration reads every block twice: the second look hits L1.
template <typename S> __device__ __forceinline__ void load8(const S* p, float (&f)[8]);
template <> __device__ __forceinline__ void load8<float>(const float* p, float (&f)[8]) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&f)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
}
template <> __device__ __forceinline__ void load8<__half>(const __half* p, float (&f)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        f[2 * i] = v.x;
        f[2 * i + 1] = v.y;
    }
}
template <> __device__ __forceinline__ void load8<double>(const double* p, float (&f)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = static_cast<float>(p[i]);
}

// NaN-ignoring max |v| over the eight elements at p, folded into m (fmaxf semantics, as block_absmax).
template <typename S> __device__ __forceinline__ float absmax8(const S* p, float m) {
    float f[8];
    load8<S>(p, f);
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(f[i]));
    return m;
}
// bf16: two elements per instruction on the packed pipe (max of two bf16 values is exact; NaN loses).
template <> __device__ __forceinline__ float absmax8<__nv_bfloat16>(const __nv_bfloat16* p, float m) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162 a = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const __nv_bfloat162 b = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    const __nv_bfloat162 c = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&raw.z));
    const __nv_bfloat162 d = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&raw.w));
    const __nv_bfloat162 top = __hmax2(__hmax2(a, b), __hmax2(c, d));
    return fmaxf(m, fmaxf(__low2float(top), __high2float(top)));
}

// x = v / absmax as the reference divides (IEEE), through the block's reciprocal where that is exact.
struct BlockDivider {
    float absmax, rinv;
    bool fast, nonzero;
    __device__ __forceinline__ explicit BlockDivider(float a) : absmax(a) {
        nonzero = a > 0.0f;
        fast = div_range_ok(a);
        rinv = fast ? 1.0f / a : 0.0f;
    }
    __device__ __forceinline__ float operator()(float v) const {
        if (fast) return div_by_block_constant(v, absmax, rinv);
        return nonzero ? v / absmax : 0.0f;
    }
    // The two cases apart, for loops that decide once per block which one they need (the choice is the same
    // for every element of a block; a test per element costs a branch per element).
    __device__ __forceinline__ float quick(float v) const { return div_by_block_constant(v, absmax, rinv); }
    __device__ __forceinline__ float careful(float v) const { return nonzero ? v / absmax : 0.0f; }
};

// ------------------------------------------------------------------------------- histogram
// bin = clamp(floor((g/absmax + 1) * bins/2), 0, bins-1); counts are integers and therefore
// independent of the order of accumulation. One warp per block (VEC: 128-bit loads, eight elements
// per lane and access) or one CTA per very long block. Every element is one shared-memory atomic
// on the CTA's histogram: the values of a block are bell-shaped over a few hundred bins, so the
// lanes of a warp rarely meet in one bin, and the hardware serialises those that do.
template <typename S, int GROUP, bool VEC, bool POW2>
__global__ void __launch_bounds__(kThreads) histogram_kernel(const S* __restrict__ g, long long period,
                                                             long long num_blocks, int bins,
                                                             unsigned long long* __restrict__ counts) {
    __shared__ unsigned int hist[4096 + 1];   // one spare counter for x == 1 (see below)
    __shared__ float red[kWarps];
    for (int i = threadIdx.x; i <= bins; i += kThreads) hist[i] = 0u;
    __syncthreads();

    const int lane = threadIdx.x & 31;
    const int tig = GROUP == 32 ? lane : static_cast<int>(threadIdx.x);
    const long long group0 = GROUP == 32 ? static_cast<long long>(blockIdx.x) * kWarps + (threadIdx.x >> 5)
                                         : static_cast<long long>(blockIdx.x);
    const long long stride = GROUP == 32 ? static_cast<long long>(gridDim.x) * kWarps : static_cast<long long>(gridDim.x);
    const float scale = 0.5f * static_cast<float>(bins);
    const int last_bin = bins - 1;
    unsigned long long since_flush = 0;

    for (long long b = group0; b < num_blocks; b += stride) {
        const S* gb = g + b * period;
        if (VEC) {   // GROUP == 32, period a multiple of 8, 16-byte aligned blocks
            const int nchunks = static_cast<int>(period >> 3);
            float m = 0.0f;
            for (int c = lane; c < nchunks; c += 32) m = absmax8<S>(gb + 8 * c, m);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            const BlockDivider divide(m);
            auto second_look = [&](auto quotient) {
                for (int c = lane; c < nchunks; c += 32) {
                    float f[8];
                    load8<S>(gb + 8 * c, f);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        // |x| <= 1 (or x is NaN), so (x + 1) * scale lies in [0, bins]: the floor is a truncation,
                        // NaN maps to bin 0, and x == 1 lands in the spare counter hist[bins], folded into the
                        // last bin at the end (the reference's upper clamp). With a power-of-two scale the sum and
                        // the product round as one fused multiply-add does (scaling by 2^k commutes with rounding).
                        const float x = quotient(f[i]);
                        const float y = POW2 ? fmaf(x, scale, scale) : (x + 1.0f) * scale;
                        atomicAdd(&hist[__float2uint_rz(y)], 1u);
                    }
                }
            };
            // (measured: deciding the kind of division once per block pays for 2-byte elements, 0.485 -> 0.518 of the
            // copy bandwidth on bf16; for fp32 the per-element form is the faster one, 0.684 against 0.589)
            if (sizeof(S) != 2) second_look([&](float v) { return divide(v); });
            else if (divide.fast) second_look([&](float v) { return divide.quick(v); });
            else second_look([&](float v) { return divide.careful(v); });
        } else {
            const float absmax = block_absmax<S, GROUP>(gb, period, tig, red);
            for (long long i = tig; i < period; i += GROUP) {
                const float v = ScalarIO<S>::load(gb + i);
                float x = 0.0f;
                if (absmax > 0.0f) x = v / absmax;
                int bin = static_cast<int>(floorf((x + 1.0f) * scale));
                bin = bin < 0 ? 0 : (bin > last_bin ? last_bin : bin);
                atomicAdd(&hist[bin], 1u);
            }
        }
        since_flush += static_cast<unsigned long long>(period);
        if (GROUP > 32 && since_flush > 0x7fffffffull) {  // keep the 32-bit counters from wrapping
            __syncthreads();
            for (int i = threadIdx.x; i < bins; i += kThreads) {
                if (hist[i]) { atomicAdd(&counts[i], static_cast<unsigned long long>(hist[i])); hist[i] = 0u; }
            }
            __syncthreads();
            since_flush = 0;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) { hist[last_bin] += hist[bins]; hist[bins] = 0u; }
    __syncthreads();
    for (int i = threadIdx.x; i < bins; i += kThreads) {
        if (hist[i]) atomicAdd(&counts[i], static_cast<unsigned long long>(hist[i]));
    }
}

// The histograms of many tensors in one launch, and their float32 sum in the tensors' order. A unit of work is a run of
// blocks of one tensor (about 256 k elements, whose counts are then added to the tensor's row).
struct HistEntry {
    const void* values;
    long long period, nb;
    long long first_unit;
    int dtype, vec;
};
__host__ __device__ inline long long hist_unit_blocks(long long period) {
    const long long blocks = (1 << 18) / period;
    return blocks < kWarps ? (period > 8192 ? 1 : kWarps) : blocks;
}
template <typename S>
__device__ __forceinline__ void hist_unit(const HistEntry& e, long long unit, int bins, bool pow2, unsigned int* hist, float* red) {
    const float scale = 0.5f * static_cast<float>(bins);
    const int last_bin = bins - 1;
    const S* values = static_cast<const S*>(e.values);
    const long long per = hist_unit_blocks(e.period), first = unit * per;
    const long long end = first + per < e.nb ? first + per : e.nb;
    const int lane = threadIdx.x & 31;
    auto count_scalar = [&](const S* gb, float absmax, int index, int stride) {
        for (long long i = index; i < e.period; i += stride) {
            const float v = ScalarIO<S>::load(gb + i);
            float x = 0.0f;
            if (absmax > 0.0f) x = v / absmax;
            int bin = static_cast<int>(floorf((x + 1.0f) * scale));
            bin = bin < 0 ? 0 : (bin > last_bin ? last_bin : bin);
            atomicAdd(&hist[bin], 1u);
        }
    };
    if (e.period > 8192) {   // the whole CTA on one block at a time
        for (long long b = first; b < end; ++b) {
            const S* gb = values + b * e.period;
            const float absmax = block_absmax<S, kThreads>(gb, e.period, threadIdx.x, red);
            count_scalar(gb, absmax, threadIdx.x, kThreads);
        }
        return;
    }
    for (long long b = first + (threadIdx.x >> 5); b < end; b += kWarps) {
        const S* gb = values + b * e.period;
        if (!e.vec) {
            count_scalar(gb, block_absmax<S, 32>(gb, e.period, lane, red), lane, 32);
            continue;
        }
        if constexpr (sizeof(S) < 8) {   // as histogram_kernel's vector form
            const int nchunks = static_cast<int>(e.period >> 3);
            float m = 0.0f;
            for (int c = lane; c < nchunks; c += 32) m = absmax8<S>(gb + 8 * c, m);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            const BlockDivider divide(m);
            auto second_look = [&](auto quotient) {
                for (int c = lane; c < nchunks; c += 32) {
                    float f[8];
                    load8<S>(gb + 8 * c, f);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float x = quotient(f[i]);
                        const float y = pow2 ? fmaf(x, scale, scale) : (x + 1.0f) * scale;
                        atomicAdd(&hist[__float2uint_rz(y)], 1u);
                    }
                }
            };
            // (once per block in every type: here fp32 gains too, 134 M values in blocks of 64 / 768 / 2048 0.587 / 0.163 /
            // 0.159 ms against 0.726 / 0.185 / 0.179 with a choice per element)
            if (divide.fast) second_look([&](float v) { return divide.quick(v); });
            else second_look([&](float v) { return divide.careful(v); });
        }
    }
}
__global__ void __launch_bounds__(kThreads) histogram_many_kernel(const HistEntry* __restrict__ table, int n, long long units, int bins,
                                                                  unsigned long long* __restrict__ rows) {
    __shared__ unsigned int hist[4096 + 1];
    __shared__ float red[kWarps];
    const bool pow2 = (bins & (bins - 1)) == 0 && bins >= 2;
    for (long long u = blockIdx.x; u < units; u += gridDim.x) {
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (table[mid].first_unit <= u) lo = mid; else hi = mid - 1;
        }
        const HistEntry& e = table[lo];
        for (int i = threadIdx.x; i <= bins; i += kThreads) hist[i] = 0u;
        __syncthreads();
        switch (e.dtype) {
            case GEFEN_B200_F32: hist_unit<float>(e, u - e.first_unit, bins, pow2, hist, red); break;
            case GEFEN_B200_F16: hist_unit<__half>(e, u - e.first_unit, bins, pow2, hist, red); break;
            case GEFEN_B200_BF16: hist_unit<__nv_bfloat16>(e, u - e.first_unit, bins, pow2, hist, red); break;
            default: hist_unit<double>(e, u - e.first_unit, bins, pow2, hist, red); break;
        }
        __syncthreads();
        if (threadIdx.x == 0) { hist[bins - 1] += hist[bins]; hist[bins] = 0u; }   // x == 1, see histogram_kernel
        __syncthreads();
        unsigned long long* row = rows + static_cast<long long>(lo) * bins;
        for (int i = threadIdx.x; i < bins; i += kThreads)
            if (hist[i]) atomicAdd(&row[i], static_cast<unsigned long long>(hist[i]));
        __syncthreads();
    }
}
__global__ void __launch_bounds__(kThreads) histogram_total_kernel(const long long* __restrict__ rows, int n, int bins, float* __restrict__ total) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= bins) return;
    float t = 0.0f;
    for (int r = 0; r < n; ++r) t += static_cast<float>(rows[static_cast<long long>(r) * bins + i]);
    total[i] = t;
}

// ------------------------------------------------------------------------------- period scores
// Sum over one block of log(x + eps) in fp64, x = v*v in fp64 unless the input is already squared
// (reference: period_variance_kernel.cu:124-139). `invalid` counts non-positive log inputs.
template <typename S, bool SQUARED>
__device__ __forceinline__ double log_term(const S* p, double eps, unsigned long long& invalid) {
    const double raw = static_cast<double>(ScalarIO<S>::load(p));
    const double x = (SQUARED ? raw : raw * raw) + eps;
    if (x <= 0.0) { ++invalid; return 0.0; }
    return log(x);
}

// period >= 64: one warp per block. period < 64: one thread per block.
template <typename S, bool SQUARED>
__global__ void __launch_bounds__(kThreads) block_logsum_kernel(const S* __restrict__ values, long long period,
                                                                long long num_blocks, double eps,
                                                                double* __restrict__ sums,
                                                                unsigned long long* __restrict__ invalid_out) {
    unsigned long long invalid = 0;
    if (period >= 64) {
        const int lane = threadIdx.x & 31;
        const long long w0 = static_cast<long long>(blockIdx.x) * kWarps + (threadIdx.x >> 5);
        const long long stride = static_cast<long long>(gridDim.x) * kWarps;
        for (long long b = w0; b < num_blocks; b += stride) {
            const S* vb = values + b * period;
            double acc = 0.0;
            for (long long i = lane; i < period; i += 32) acc += log_term<S, SQUARED>(vb + i, eps, invalid);
            acc = warp_sum(acc);
            if (lane == 0) sums[b] = acc;
        }
    } else {
        const long long t0 = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
        const long long stride = static_cast<long long>(gridDim.x) * kThreads;
        for (long long b = t0; b < num_blocks; b += stride) {
            const S* vb = values + b * period;
            double acc = 0.0;
            for (long long i = 0; i < period; ++i) acc += log_term<S, SQUARED>(vb + i, eps, invalid);
            sums[b] = acc;
        }
    }
    if (invalid) atomicAdd(invalid_out, invalid);
}

// partial[c] = sum over this CTA's slice of |S[j+1]/P - S[j]/P|, fixed order => reproducible.
__global__ void __launch_bounds__(kThreads) adjacent_diff_partial_kernel(const double* __restrict__ sums,
                                                                         long long num_pairs, double period,
                                                                         double* __restrict__ partial) {
    __shared__ double red[kWarps];
    const long long per_cta = (num_pairs + gridDim.x - 1) / gridDim.x;
    const long long begin = static_cast<long long>(blockIdx.x) * per_cta;
    long long end = begin + per_cta;
    if (end > num_pairs) end = num_pairs;
    double acc = 0.0;
    for (long long j = begin + threadIdx.x; j < end; j += kThreads) {
        const double cur = sums[j] / period;
        const double nxt = sums[j + 1] / period;
        acc += fabs(nxt - cur);
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kWarps; ++w) t += red[w];
        partial[blockIdx.x] = t;
    }
}

__global__ void adjacent_diff_final_kernel(const double* __restrict__ partial, int n_partial, double num_pairs,
                                           const unsigned long long* __restrict__ invalid,
                                           double* __restrict__ stats) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < n_partial; ++i) t += partial[i];
        stats[0] = t / num_pairs;
        stats[1] = static_cast<double>(*invalid);
    }
}

// ------------------------------------------------------------------------------- scan of many periods
// All candidate periods of many tensors in a handful of launches. The block sums of a candidate are formed from those
// of a smaller candidate that divides it; the candidates that no other one divides ("bases": 8, 9 and 12 for a tensor
// of 768 x 2304 elements) read the tensor themselves.
//
// A base takes one logarithm per block, not per element: the sum of log x_i is the logarithm of the product, which is
// kept as a mantissa in [1, 2) and an exponent (split off every eight factors; with 2^-120 <= eps <= 2^100 and
// |g| < 2^63 eight factors neither overflow nor underflow, other values take their own logarithm). One rounding of 2^-53 per factor is
// less than what adding up logarithms of about -25 costs (2^-49 per term). Two double-precision operations per
// element remain, and the tensor is read once per base instead of a double per element written and read back.
// An element moves the exponent by at most 128: 32 bits (E = int) hold it for blocks below kCtaPeriod, the longer blocks
// count in 64 (zeros in fp32 with eps = 1e-12 leave 32 bits at 430 M elements per block).
template <typename E> struct LogProduct {
    double mantissa, slow;
    E exponent;
    __device__ __forceinline__ LogProduct() : mantissa(1.0), slow(0.0), exponent(0) {}
    __device__ __forceinline__ void split() {
        const int hi = __double2hiint(mantissa);
        exponent += (hi >> 20) - 1023;
        mantissa = __hiloint2double((hi & 0x000FFFFF) | 0x3FF00000, __double2loint(mantissa));
    }
    // |f| as a double, built from the bits (the conversion instruction runs at a quarter of the arithmetic's rate).
    // Subnormal and zero values come out as at most 2^-126, whose square vanishes beside eps >= 2^-120.
    static __device__ __forceinline__ double magnitude(uint32_t bits) {
        return __hiloint2double(static_cast<int>(((bits & 0x7FFFFFFFu) >> 3) + 0x38000000u), static_cast<int>(bits << 29));
    }
    // up to eight values; the first n count
    template <bool SQUARED>
    __device__ __forceinline__ void add(const float (&f)[8], int n, double eps, bool eps_ok, unsigned long long& invalid) {
        uint32_t most = 0u;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t bits = __float_as_uint(f[i]) & (SQUARED ? 0xFFFFFFFFu : 0x7FFFFFFFu);   // (negative: largest)
            most = i < n && bits > most ? bits : most;
        }
        if (eps_ok && most < (SQUARED ? 0x71800000u : 0x5F000000u)) {   // 2^100 / 2^63; NaN and infinity are above
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const double v = magnitude(__float_as_uint(f[i]));
                const double x = SQUARED ? v + eps : fma(v, v, eps);
                mantissa *= i < n ? x : 1.0;
            }
            split();
        } else {
            for (int i = 0; i < n; ++i) slow += log_term<float, SQUARED>(f + i, eps, invalid);
        }
    }
    template <int LANES> __device__ __forceinline__ void combine() {
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            mantissa *= __shfl_xor_sync(0xffffffffu, mantissa, o);   // at most 2^32
            exponent += __shfl_xor_sync(0xffffffffu, exponent, o);
            slow += __shfl_xor_sync(0xffffffffu, slow, o);
        }
    }
    __device__ __forceinline__ double value() const { return log(mantissa) + (static_cast<double>(exponent) * 0.693147180559945309417 + slow); }
};

struct ScanBase {
    const void* values;
    long long dst;         // offset of its sums (in doubles from the scratch base)
    long long period, nb;
    long long first_unit;  // in the index space of the launch
    int dtype, tensor;
    int count_invalid;     // one base per tensor counts the non-positive logarithm inputs
    int vec;               // eight elements per load
};
struct ScanCandidate {
    long long src;         // offset of the sums that this candidate is regrouped from
    long long dst;         // offset of its own sums
    long long ratio;       // period / parent period; 0: a base
    long long nb;          // blocks of this period
    long long first_unit;  // of its level's regrouping launch
    long long first_partial;   // number of its first partial sum
    double period;
    int n_partial;
    int tensor;
};

constexpr int kThreadPeriod = 64;       // shorter blocks: one thread each,
constexpr int kGroupPeriod = 512;       // shorter ones: eight lanes each; longer ones: one warp (blocks of 167 elements by
                                        // whole warps spent most of their time on the warp's reduction and logarithm:
                                        // the scan of 383 M bf16 elements 2.06 -> 1.63 ms),
constexpr int kCtaPeriod = 16384;       // from here on one CTA
static_assert(128ll * kCtaPeriod < (1ll << 31), "a 32-bit exponent holds the product of a shorter block");
// Blocks of one unit of work (a CTA's turn).
__host__ __device__ inline long long base_unit_blocks(long long period) {
    if (period < kThreadPeriod) return 2 * kThreads;
    if (period >= kCtaPeriod) return 1;
    return period >= 1024 ? kWarps : (period >= kGroupPeriod ? kWarps * 4 : kThreads / 8 * 2);
}

template <typename S> __device__ __forceinline__ float scan_value(const S* p) { return ScalarIO<S>::load(p); }

// The product over elements first, first + stride, ... (stride counted in elements; VEC: runs of eight) of one block.
template <typename S, bool SQUARED, typename E>
__device__ __forceinline__ void block_product(const S* v, long long period, int index, int count, bool vec, double eps, bool eps_ok,
                                              LogProduct<E>& p, unsigned long long& invalid) {
    if constexpr (sizeof(S) == 8) {
        for (long long i = index; i < period; i += count) p.slow += log_term<S, SQUARED>(v + i, eps, invalid);
    } else {
        float f[8];
        if (vec) {
            for (long long c = index; c < period / 8; c += count) {
                load8<S>(v + 8 * c, f);
                p.template add<SQUARED>(f, 8, eps, eps_ok, invalid);
            }
        } else {
            for (long long i0 = index; i0 < period; i0 += 8LL * count) {
                const long long left = (period - i0 + count - 1) / count;
                const int n = left < 8 ? static_cast<int>(left) : 8;
#pragma unroll
                for (int u = 0; u < 8; ++u) f[u] = u < n ? scan_value(v + i0 + static_cast<long long>(u) * count) : 0.0f;
                p.template add<SQUARED>(f, n, eps, eps_ok, invalid);
            }
        }
    }
}

template <typename S, bool SQUARED>
__device__ __forceinline__ void scan_base_unit(const ScanBase& b, long long unit, double eps, bool eps_ok, double* sums,
                                               unsigned long long& invalid) {
    const S* values = static_cast<const S*>(b.values);
    const long long period = b.period, first = unit * base_unit_blocks(period);
    if (period < kThreadPeriod) {
        for (int r = 0; r < 2; ++r) {
            const long long j = first + r * kThreads + threadIdx.x;
            if (j >= b.nb) return;
            LogProduct<int> p;
            block_product<S, SQUARED>(values + j * period, period, 0, 1, b.vec != 0, eps, eps_ok, p, invalid);
            sums[j] = p.value();
        }
    } else if (period < kGroupPeriod) {
        const long long end = first + base_unit_blocks(period) < b.nb ? first + base_unit_blocks(period) : b.nb;
        for (long long j0 = first; j0 < end; j0 += kThreads / 8) {   // uniform over the CTA: the groups shuffle together
            const long long j = j0 + (threadIdx.x >> 3);
            LogProduct<int> p;
            if (j < end) block_product<S, SQUARED>(values + j * period, period, threadIdx.x & 7, 8, b.vec != 0, eps, eps_ok, p, invalid);
            p.template combine<8>();
            if (j < end && (threadIdx.x & 7) == 0) sums[j] = p.value();
        }
    } else if (period < kCtaPeriod) {
        const int lane = threadIdx.x & 31;
        const long long end = first + base_unit_blocks(period) < b.nb ? first + base_unit_blocks(period) : b.nb;
        for (long long j = first + (threadIdx.x >> 5); j < end; j += kWarps) {
            LogProduct<int> p;
            block_product<S, SQUARED>(values + j * period, period, lane, 32, b.vec != 0, eps, eps_ok, p, invalid);
            p.template combine<32>();
            if (lane == 0) sums[j] = p.value();
        }
    } else {
        __shared__ double red[kWarps];
        LogProduct<long long> p;
        block_product<S, SQUARED>(values + first * period, period, threadIdx.x, kThreads, b.vec != 0, eps, eps_ok, p, invalid);
        p.template combine<32>();
        __syncthreads();   // the previous unit's sum has been read
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = p.value();
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < kWarps; ++w) t += red[w];
            sums[first] = t;
        }
    }
}

// Entry of a table sorted by `key` (the first unit of each entry) that holds `unit`.
template <typename T, typename F> __device__ __forceinline__ int find_entry(const T* table, int n, long long unit, F key) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (key(table[mid]) <= unit) lo = mid; else hi = mid - 1;
    }
    return lo;
}

template <bool SQUARED>
__global__ void __launch_bounds__(kThreads) scan_base_kernel(double* __restrict__ scratch, const ScanBase* __restrict__ table, int n,
                                                             long long units, double eps, unsigned long long* __restrict__ invalid_out) {
    // 2^-120; squared inputs: 2^-70 (zeros and subnormal values count as up to 2^-126 themselves, not squared)
    // up to 2^100: a factor stays below 2^127, eight of them and the mantissa below 2^1017
    const bool eps_ok = eps >= (SQUARED ? 8.470329472543003e-22 : 7.52316384526264e-37) && eps <= 1.2676506002282294e30;
    for (long long u = blockIdx.x; u < units; u += gridDim.x) {
        const ScanBase& b = table[find_entry(table, n, u, [](const ScanBase& e) { return e.first_unit; })];
        const long long unit = u - b.first_unit;
        double* sums = scratch + b.dst;
        unsigned long long invalid = 0;
        switch (b.dtype) {
            case GEFEN_B200_F32: scan_base_unit<float, SQUARED>(b, unit, eps, eps_ok, sums, invalid); break;
            case GEFEN_B200_F16: scan_base_unit<__half, SQUARED>(b, unit, eps, eps_ok, sums, invalid); break;
            case GEFEN_B200_BF16: scan_base_unit<__nv_bfloat16, SQUARED>(b, unit, eps, eps_ok, sums, invalid); break;
            default: scan_base_unit<double, SQUARED>(b, unit, eps, eps_ok, sums, invalid); break;
        }
        if (invalid != 0 && b.count_invalid) atomicAdd(&invalid_out[b.tensor], invalid);
    }
}

constexpr int kRegroupUnit = 4 * kThreads;   // outputs of a unit whose outputs are formed by one thread each
__host__ __device__ inline long long regroup_units(long long ratio, long long nb) {
    return ratio >= 64 ? (nb + kWarps - 1) / kWarps : (nb + kRegroupUnit - 1) / kRegroupUnit;
}
// One level: out[j] = sum of `ratio` consecutive sums of the parent, added left to right.
__global__ void __launch_bounds__(kThreads) scan_regroup_kernel(double* __restrict__ scratch, const ScanCandidate* __restrict__ table,
                                                                int n, long long units) {
    for (long long u = blockIdx.x; u < units; u += gridDim.x) {
        const ScanCandidate& c = table[find_entry(table, n, u, [](const ScanCandidate& e) { return e.first_unit; })];
        const double* in = scratch + c.src;
        double* out = scratch + c.dst;
        const long long ratio = c.ratio, nb = c.nb, unit = u - c.first_unit;
        if (ratio >= 64) {
            const int lane = threadIdx.x & 31;
            const long long j = unit * kWarps + (threadIdx.x >> 5);
            if (j >= nb) continue;
            double acc = 0.0;
            for (long long i = lane; i < ratio; i += 32) acc += in[j * ratio + i];
            acc = warp_sum(acc);
            if (lane == 0) out[j] = acc;
        } else {
            for (int r = 0; r < kRegroupUnit / kThreads; ++r) {
                const long long j = unit * kRegroupUnit + r * kThreads + threadIdx.x;
                if (j >= nb) break;
                double acc = 0.0;
                for (long long i = 0; i < ratio; ++i) acc += in[j * ratio + i];
                out[j] = acc;
            }
        }
    }
}

// Partial sums of |S[j+1] - S[j]| (the mean difference is that over the period), cut by the candidate's own number of
// partials: reproducible.
__global__ void __launch_bounds__(kThreads) scan_partial_kernel(const double* __restrict__ scratch, const ScanCandidate* __restrict__ table,
                                                                int n, double* __restrict__ partials) {
    __shared__ double red[kWarps];
    const long long u = blockIdx.x;
    const ScanCandidate& c = table[find_entry(table, n, u, [](const ScanCandidate& e) { return e.first_partial; })];
    const double* sums = scratch + c.dst;
    const long long num_pairs = c.nb - 1;
    const long long per = (num_pairs + c.n_partial - 1) / c.n_partial;
    const long long begin = (u - c.first_partial) * per;
    const long long end = begin + per < num_pairs ? begin + per : num_pairs;
    double acc = 0.0;
    for (long long j = begin + threadIdx.x; j < end; j += kThreads) acc += fabs(sums[j + 1] - sums[j]);
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kWarps; ++w) t += red[w];
        partials[u] = t;
    }
}

// stats[candidate] = (score, invalid inputs of its tensor); one warp per candidate. `place`: where in stats.
__global__ void __launch_bounds__(kThreads) scan_final_kernel(const double* __restrict__ partials, const ScanCandidate* __restrict__ table,
                                                              const int* __restrict__ place, int n,
                                                              const unsigned long long* __restrict__ invalid, double* __restrict__ stats) {
    const int i = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (i >= n) return;
    const ScanCandidate& c = table[i];
    const int lane = threadIdx.x & 31;
    double t = 0.0;
    for (int k = lane; k < c.n_partial; k += 32) t += partials[c.first_partial + k];
    t = warp_sum(t);
    if (lane == 0) {
        stats[2 * place[i]] = t / c.period / static_cast<double>(c.nb - 1);
        stats[2 * place[i] + 1] = static_cast<double>(invalid[c.tensor]);
    }
}

// Mean within-block variance / coefficient of variation of x (= v or v*v), fp32 sums
// (reference: period_variance_kernel.cu:13-106). One warp per block.
template <typename S, bool SQUARED, bool COV>
__global__ void __launch_bounds__(kThreads) block_moment_kernel(const S* __restrict__ values, long long period,
                                                                long long num_blocks, double* __restrict__ stats) {
    const int lane = threadIdx.x & 31;
    const long long w0 = static_cast<long long>(blockIdx.x) * kWarps + (threadIdx.x >> 5);
    const long long stride = static_cast<long long>(gridDim.x) * kWarps;
    for (long long b = w0; b < num_blocks; b += stride) {
        const S* vb = values + b * period;
        float sx = 0.0f, sx2 = 0.0f;
        for (long long i = lane; i < period; i += 32) {
            const float v = ScalarIO<S>::load(vb + i);
            const float x = SQUARED ? v : v * v;
            sx += x;
            sx2 = fmaf(x, x, sx2);
        }
        sx = warp_sum(sx);
        sx2 = warp_sum(sx2);
        if (lane == 0) {
            const float mean = sx / static_cast<float>(period);
            float var = sx2 / static_cast<float>(period);
            var -= mean * mean;
            if (var < 0.0f) var = 0.0f;
            if (!COV) {
                atomicAdd(stats, static_cast<double>(var));
            } else if (mean < 0.0f) {
                atomicAdd(stats + 2, 1.0);
            } else if (mean > 0.0f) {
                atomicAdd(stats, static_cast<double>(sqrtf(var) / mean));
                atomicAdd(stats + 1, 1.0);
            }
        }
    }
}

// ------------------------------------------------------------------------------- Lloyd-Max
// Both kernels assign every normalised value to its codebook entry with the rule of the step kernels
// (nearest entry, left on ties; reference: lloyd_max_fused_kernel.cu:16-48), through the codebook
// workspace staged in shared memory: one table read and one compare per value, the binary search
// over the thresholds only for the few undecidable cells.
struct LloydTables {
    const float* cb;
    const float* thr;
    const unsigned char* lut;
    int k;
    __device__ __forceinline__ int entry(float x) const {
        // the table covers [-1, 1]; values outside it (non-finite gradients) take the exact rule
        if (!(fabsf(x) <= 1.0f)) return entry_exact(x, thr, cb, k);
        bool slow;
        const int e = lut_query(x, lut, &slow);
        return slow ? entry_exact(x, thr, cb, k) : e;
    }
};

__device__ __forceinline__ LloydTables stage_lloyd_tables(const unsigned char* ws, unsigned char* smem) {
    const uint4* src = reinterpret_cast<const uint4*>(ws);
    uint4* dst = reinterpret_cast<uint4*>(smem);
    for (int i = threadIdx.x; i < GEFEN_B200_CODEBOOK_WS_BYTES / 16; i += blockDim.x) dst[i] = src[i];
    __syncthreads();
    LloydTables t;
    t.cb = reinterpret_cast<const float*>(smem + kWsCodebookOff);
    t.thr = reinterpret_cast<const float*>(smem + kWsThresholdOff);
    t.lut = smem + kWsLutOff;
    t.k = reinterpret_cast<const int*>(smem + kWsMetaOff)[0];
    return t;
}

// (x + 1) * 2^24 rounded to an integer in [0, 2^25] for |x| <= 1 (non-finite values, which only non-finite
// gradients produce, count as x = 0 in the sum; their count is still taken).
__device__ __forceinline__ unsigned int lloyd_fixed(float x) {
    const float scaled = x * 16777216.0f;
    const int q = (fabsf(scaled) <= 16777216.0f) ? __float2int_rn(scaled) : 0;
    return static_cast<unsigned int>(q + 16777216);
}

// E-step: per codebook entry, the sum of the normalised values assigned to it and their count
// (reference: lloyd_max_fused_kernel.cu:50-118). Sums are fp32 atomics (order-dependent in the
// reference too); counts are exact.
template <typename S, int GROUP, bool VEC>
__global__ void __launch_bounds__(kThreads) lloyd_accumulate_kernel(const S* __restrict__ g, long long period,
                                                                    long long num_blocks, const unsigned char* ws,
                                                                    int k, float* __restrict__ sums,
                                                                    unsigned long long* __restrict__ counts) {
    __shared__ __align__(16) unsigned char tables[GEFEN_B200_CODEBOOK_WS_BYTES];
    // Per-entry sums are kept in shared memory in fixed point, as the 64-bit sum of (x + 1) * 2^24 in two 32-bit
    // words: float and 64-bit additions to shared memory are compare-and-swap loops, 32-bit integer ones are
    // native. An element costs one add to the low word (whose returned old value tells a carry, which then
    // goes to the high word: once per ~128 elements of an entry) and one to the count; the offset count * 2^24
    // comes off at the flush. The sum does not depend on the order of the additions, values of magnitude 2^-1
    // or more are exact and smaller ones are within 2^-25.
    __shared__ unsigned int slo[kMaxCodebook];
    __shared__ unsigned int shi[kMaxCodebook];
    __shared__ unsigned int scnt[kMaxCodebook];
    __shared__ float red[kWarps];
    slo[threadIdx.x] = 0u;
    shi[threadIdx.x] = 0u;
    scnt[threadIdx.x] = 0u;
    auto add = [&](int e, float x) {
        const unsigned int v = lloyd_fixed(x);
        const unsigned int old = atomicAdd(&slo[e], v);
        if (old + v < old) atomicAdd(&shi[e], 1u);
        atomicAdd(&scnt[e], 1u);
    };
    auto flush = [&]() {   // every thread of the CTA, between two __syncthreads
        if (threadIdx.x < k && scnt[threadIdx.x]) {
            const unsigned long long raw = (static_cast<unsigned long long>(shi[threadIdx.x]) << 32) | slo[threadIdx.x];
            const long long fixed = static_cast<long long>(raw) - (static_cast<long long>(scnt[threadIdx.x]) << 24);
            atomicAdd(&sums[threadIdx.x], static_cast<float>(static_cast<double>(fixed) * (1.0 / 16777216.0)));
            atomicAdd(&counts[threadIdx.x], static_cast<unsigned long long>(scnt[threadIdx.x]));
            slo[threadIdx.x] = shi[threadIdx.x] = scnt[threadIdx.x] = 0u;
        }
    };
    const LloydTables t = stage_lloyd_tables(ws, tables);
    const int lane = threadIdx.x & 31;
    const int tig = GROUP == 32 ? lane : static_cast<int>(threadIdx.x);
    const long long group0 = GROUP == 32 ? static_cast<long long>(blockIdx.x) * kWarps + (threadIdx.x >> 5)
                                         : static_cast<long long>(blockIdx.x);
    const long long stride = GROUP == 32 ? static_cast<long long>(gridDim.x) * kWarps : static_cast<long long>(gridDim.x);
    unsigned long long since_flush = 0;
    for (long long b = group0; b < num_blocks; b += stride) {
        const S* gb = g + b * period;
        if (VEC) {
            const int nchunks = static_cast<int>(period >> 3);
            float m = 0.0f;
            for (int c = lane; c < nchunks; c += 32) {
                float f[8];
                load8<S>(gb + 8 * c, f);
#pragma unroll
                for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(f[i]));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            const BlockDivider divide(m);
            auto second_look = [&](auto quotient) {
                for (int c = lane; c < nchunks; c += 32) {
                    float f[8];
                    load8<S>(gb + 8 * c, f);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float x = quotient(f[i]);
                        add(t.entry(x), x);
                    }
                }
            };
            if (divide.fast) second_look([&](float v) { return divide.quick(v); });
            else second_look([&](float v) { return divide.careful(v); });
        } else {
            const float absmax = block_absmax<S, GROUP>(gb, period, tig, red);
            for (long long i = tig; i < period; i += GROUP) {
                const float v = ScalarIO<S>::load(gb + i);
                float x = 0.0f;
                if (absmax > 0.0f) x = v / absmax;
                add(t.entry(x), x);
            }
        }
        since_flush += static_cast<unsigned long long>(period);
        if (GROUP > 32 && since_flush > 0x7fffffffull) {   // keep the 32-bit counts from wrapping
            __syncthreads();
            flush();
            __syncthreads();
            since_flush = 0;
        }
    }
    __syncthreads();
    flush();
}

// Logging MSE of assigning with the old codebook and reconstructing with the new one
// (reference: lloyd_max_fused_kernel.cu:120-195).
template <typename S, int GROUP, bool VEC>
__global__ void __launch_bounds__(kThreads) lloyd_mse_kernel(const S* __restrict__ g, long long period,
                                                             long long num_blocks, const unsigned char* old_ws,
                                                             const float* __restrict__ new_codebook, int k,
                                                             float* __restrict__ mse_norm, float* __restrict__ mse_orig) {
    __shared__ __align__(16) unsigned char tables[GEFEN_B200_CODEBOOK_WS_BYTES];
    __shared__ float ncb[kMaxCodebook];
    __shared__ float red[kWarps];
    __shared__ float red2[2][kWarps];
    ncb[threadIdx.x] = new_codebook[threadIdx.x < k ? threadIdx.x : k - 1];
    const LloydTables t = stage_lloyd_tables(old_ws, tables);
    const int lane = threadIdx.x & 31;
    const int tig = GROUP == 32 ? lane : static_cast<int>(threadIdx.x);
    const long long group0 = GROUP == 32 ? static_cast<long long>(blockIdx.x) * kWarps + (threadIdx.x >> 5)
                                         : static_cast<long long>(blockIdx.x);
    const long long stride = GROUP == 32 ? static_cast<long long>(gridDim.x) * kWarps : static_cast<long long>(gridDim.x);
    float en = 0.0f, eo = 0.0f;
    for (long long b = group0; b < num_blocks; b += stride) {
        const S* gb = g + b * period;
        if (VEC) {
            const int nchunks = static_cast<int>(period >> 3);
            float m = 0.0f;
            for (int c = lane; c < nchunks; c += 32) {
                float f[8];
                load8<S>(gb + 8 * c, f);
#pragma unroll
                for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(f[i]));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            const BlockDivider divide(m);
            auto second_look = [&](auto quotient) {
                for (int c = lane; c < nchunks; c += 32) {
                    float f[8];
                    load8<S>(gb + 8 * c, f);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float x = quotient(f[i]);
                        const float err = x - ncb[t.entry(x)];
                        en = fmaf(err, err, en);
                        const float oe = err * m;
                        eo = fmaf(oe, oe, eo);
                    }
                }
            };
            if (divide.fast) second_look([&](float v) { return divide.quick(v); });
            else second_look([&](float v) { return divide.careful(v); });
        } else {
            const float absmax = block_absmax<S, GROUP>(gb, period, tig, red);
            for (long long i = tig; i < period; i += GROUP) {
                const float v = ScalarIO<S>::load(gb + i);
                float x = 0.0f;
                if (absmax > 0.0f) x = v / absmax;
                const float err = x - ncb[t.entry(x)];
                en = fmaf(err, err, en);
                const float oe = err * absmax;
                eo = fmaf(oe, oe, eo);
            }
        }
    }
    en = warp_sum(en);
    eo = warp_sum(eo);
    if (lane == 0) { red2[0][threadIdx.x >> 5] = en; red2[1][threadIdx.x >> 5] = eo; }
    __syncthreads();
    if (threadIdx.x == 0) {
        float a = 0.0f, c = 0.0f;
        for (int w = 0; w < kWarps; ++w) { a += red2[0][w]; c += red2[1][w]; }
        atomicAdd(mse_norm, a);
        atomicAdd(mse_orig, c);
    }
}

// ------------------------------------------------------------------------------- host side
static int check_flat(const void* values, int dtype, int64_t numel, int64_t period) {
    GEFEN_CHECK_ARG(values != nullptr || numel == 0, "Expected a non-null tensor.");
    GEFEN_CHECK_ARG(is_float_dtype(dtype), "Expected a floating-point tensor.");
    GEFEN_CHECK_ARG(period > 0, "Expected a positive period.");
    GEFEN_CHECK_ARG(numel >= 0 && numel % period == 0, "Expected tensor length to be divisible by period.");
    return GEFEN_B200_OK;
}

#define GEFEN_DISPATCH_S(dtype, ...)                                                       \
    switch (dtype) {                                                                       \
        case GEFEN_B200_F32: { using S = float; __VA_ARGS__; } break;                      \
        case GEFEN_B200_F16: { using S = __half; __VA_ARGS__; } break;                     \
        case GEFEN_B200_BF16: { using S = __nv_bfloat16; __VA_ARGS__; } break;             \
        default: { using S = double; __VA_ARGS__; } break;                                 \
    }

constexpr int kMaxPartials = 1024;
static int partials_for(int64_t pairs) {
    int n_partial = static_cast<int>((pairs + 4095) / 4096);
    if (n_partial > kMaxPartials) n_partial = kMaxPartials;
    if (n_partial < 1) n_partial = 1;
    return n_partial;
}

static int launch_block_logsums(const void* values, int dtype, int64_t numel, int64_t period, bool squared, double eps,
                                double* sums, unsigned long long* invalid, cudaStream_t stream) {
    const int64_t nb = numel / period;
    const int grid = period >= 64 ? persistent_grid(nb, kWarps, 8) : persistent_grid(nb, kThreads, 8);
    GEFEN_DISPATCH_S(dtype, {
        if (squared)
            block_logsum_kernel<S, true><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(values), period, nb, eps, sums, invalid);
        else
            block_logsum_kernel<S, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(values), period, nb, eps, sums, invalid);
    });
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

// score = mean over adjacent pairs of |S[j+1]/P - S[j]/P|; `partial` holds kMaxPartials doubles.
static int launch_adjacent_score(const double* sums, int64_t nb, int64_t period, const unsigned long long* invalid,
                                 double* partial, double* stats, cudaStream_t stream) {
    const int64_t pairs = nb - 1;
    const int n_partial = partials_for(pairs);
    adjacent_diff_partial_kernel<<<n_partial, kThreads, 0, stream>>>(sums, pairs, static_cast<double>(period), partial);
    GEFEN_CHECK_CUDA(cudaGetLastError());
    adjacent_diff_final_kernel<<<1, 32, 0, stream>>>(partial, n_partial, static_cast<double>(pairs), invalid, stats);
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

static int adjacent_score(const void* values, int dtype, int64_t numel, int64_t period, bool squared, double eps,
                          double* stats, double* block_sums, cudaStream_t stream) {
    const int64_t nb = numel / period;
    unsigned long long* invalid = reinterpret_cast<unsigned long long*>(block_sums + nb);
    double* partial = block_sums + nb + 1;
    GEFEN_CHECK_CUDA(cudaMemsetAsync(invalid, 0, sizeof(unsigned long long), stream));
    int rc = launch_block_logsums(values, dtype, numel, period, squared, eps, block_sums, invalid, stream);
    if (rc != GEFEN_B200_OK) return rc;
    return launch_adjacent_score(block_sums, nb, period, invalid, partial, stats, stream);
}

// Plan of a scan: for every tensor the bases, and for every other candidate its parent. Offsets index one scratch
// array: [invalid counts | sums | partial sums | tables].
struct ScanPlan {
    std::vector<ScanBase> bases;
    std::vector<ScanCandidate> candidates;   // by level, bases first
    std::vector<int> place;                  // index of each in the caller's order
    std::vector<int> level_begin;            // first candidate of each level, and the end
    std::vector<int64_t> level_units;
    int64_t base_units = 0, partials = 0;
    int64_t partial_offset = 0, bases_offset = 0, candidates_offset = 0, place_offset = 0, total = 0;   // doubles
};

static int64_t doubles_for(size_t bytes) { return static_cast<int64_t>((bytes + 7) / 8); }

static ScanPlan make_scan_plan(int n_tensors, const uint64_t* values, const int32_t* dtypes, const int64_t* numels,
                               const int32_t* offsets, const int64_t* periods) {
    struct Item { int tensor, index, parent, level; int64_t period; };
    ScanPlan plan;
    std::vector<Item> items;
    int levels = 1;
    for (int t = 0; t < n_tensors; ++t) {
        const int first = static_cast<int>(items.size());
        for (int i = offsets[t]; i < offsets[t + 1]; ++i) items.push_back({t, i, -1, 0, periods[i]});
        std::stable_sort(items.begin() + first, items.end(), [](const Item& x, const Item& y) { return x.period < y.period; });
        for (int i = first; i < static_cast<int>(items.size()); ++i) {
            // the parent: a divisor of at least a sixteenth with the shortest way to the tensor, else the largest divisor
            int best = -1, largest = -1;
            for (int j = i - 1; j >= first; --j) {
                if (items[j].period == items[i].period || items[i].period % items[j].period != 0) continue;
                if (largest < 0) largest = j;
                if (items[i].period / items[j].period <= 16 && (best < 0 || items[j].level < items[best].level)) best = j;
            }
            items[i].parent = best >= 0 ? best : largest;
            items[i].level = items[i].parent < 0 ? 0 : items[items[i].parent].level + 1;
            levels = std::max(levels, items[i].level + 1);
        }
    }
    const int n = static_cast<int>(items.size());
    int64_t cursor = n_tensors;
    std::vector<int64_t> dst(n);
    for (int i = 0; i < n; ++i) { dst[i] = cursor; cursor += numels[items[i].tensor] / items[i].period; }
    std::vector<bool> counted(n_tensors, false);
    for (int level = 0; level < levels; ++level) {
        plan.level_begin.push_back(static_cast<int>(plan.candidates.size()));
        int64_t units = 0;
        for (int i = 0; i < n; ++i) {
            const Item& it = items[i];
            if (it.level != level) continue;
            ScanCandidate c = {};
            c.nb = numels[it.tensor] / it.period;
            c.dst = dst[i];
            c.period = static_cast<double>(it.period);
            c.tensor = it.tensor;
            c.n_partial = partials_for(c.nb - 1);
            c.first_partial = plan.partials;
            plan.partials += c.n_partial;
            if (level == 0) {
                ScanBase b = {};
                b.values = reinterpret_cast<const void*>(static_cast<uintptr_t>(values[it.tensor]));
                b.dst = c.dst;
                b.period = it.period;
                b.nb = c.nb;
                b.first_unit = plan.base_units;
                b.dtype = dtypes[it.tensor];
                b.tensor = it.tensor;
                b.count_invalid = counted[it.tensor] ? 0 : 1;
                counted[it.tensor] = true;
                b.vec = it.period % 8 == 0 && aligned16(b.values) && b.dtype != GEFEN_B200_F64;
                plan.base_units += (b.nb + base_unit_blocks(b.period) - 1) / base_unit_blocks(b.period);
                plan.bases.push_back(b);
            } else {
                c.src = dst[it.parent];
                c.ratio = it.period / items[it.parent].period;
                c.first_unit = units;
                units += regroup_units(c.ratio, c.nb);
            }
            plan.candidates.push_back(c);
            plan.place.push_back(it.index);
        }
        plan.level_units.push_back(units);
    }
    plan.level_begin.push_back(n);
    plan.partial_offset = cursor;
    cursor += plan.partials;
    plan.bases_offset = cursor;
    cursor += doubles_for(plan.bases.size() * sizeof(ScanBase));
    plan.candidates_offset = cursor;
    cursor += doubles_for(plan.candidates.size() * sizeof(ScanCandidate));
    plan.place_offset = cursor;
    cursor += doubles_for(plan.place.size() * sizeof(int));
    plan.total = cursor;
    return plan;
}

}  // namespace gefen

using namespace gefen;

extern "C" {

int gefen_b200_exact_histogram(const void* grad_flat, int grad_dtype, int64_t numel, int64_t period,
                               int64_t* bin_counts, int histogram_bins, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(bin_counts != nullptr, "Expected a non-null bin_counts.");
    GEFEN_CHECK_ARG(histogram_bins >= 1 && histogram_bins <= 4096, "Expected histogram size in [1, 4096].");
    GEFEN_CHECK_ARG(period > 0, "Expected period to be positive.");
    GEFEN_CHECK_ARG(grad_flat != nullptr || numel == 0, "Expected a non-null grad_flat.");
    GEFEN_CHECK_ARG(is_float_dtype(grad_dtype), "Unsupported gradient dtype tag %d.", grad_dtype);
    GEFEN_CHECK_ARG(numel >= 0 && numel % period == 0, "Expected grad_flat.numel() to be divisible by period.");
    const int64_t nb = numel / period;
    if (nb == 0) return GEFEN_B200_OK;
    unsigned long long* counts = reinterpret_cast<unsigned long long*>(bin_counts);
    // a warp's 32-bit counters cannot wrap: a CTA of the warp-per-block form sees at most 2^31 elements
    if (period <= 8192) {
        const int grid = persistent_grid(nb, kWarps, 6);
        const bool vec = period % 8 == 0 && aligned16(grad_flat) && grad_dtype != GEFEN_B200_F64 &&
                         numel / grid < 0x7fffffffll;
        const bool pow2 = (histogram_bins & (histogram_bins - 1)) == 0 && histogram_bins >= 2;
        if (vec && pow2) {
            GEFEN_DISPATCH_S(grad_dtype, histogram_kernel<S, 32, true, true><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, histogram_bins, counts));
        } else if (vec) {
            GEFEN_DISPATCH_S(grad_dtype, histogram_kernel<S, 32, true, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, histogram_bins, counts));
        } else {
            GEFEN_DISPATCH_S(grad_dtype, histogram_kernel<S, 32, false, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, histogram_bins, counts));
        }
    } else {
        const int grid = persistent_grid(nb, 1, 6);
        GEFEN_DISPATCH_S(grad_dtype, histogram_kernel<S, 256, false, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, histogram_bins, counts));
    }
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

int64_t gefen_b200_exact_histogram_many_table_bytes(int n_tensors) {
    return n_tensors > 0 ? static_cast<int64_t>(n_tensors) * static_cast<int64_t>(sizeof(HistEntry)) : 0;
}

int gefen_b200_exact_histogram_many(int n_tensors, const uint64_t* values, const int32_t* dtypes, const int64_t* numels,
                                    const int64_t* periods, int64_t* rows, float* total, int histogram_bins, void* device_table,
                                    void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(n_tensors >= 1 && values && dtypes && numels && periods && rows && total && device_table, "Expected non-null arguments.");
    GEFEN_CHECK_ARG(histogram_bins >= 1 && histogram_bins <= 4096, "Expected histogram size in [1, 4096].");
    GEFEN_CHECK_ARG(aligned16(device_table), "Expected a 16-byte aligned table.");
    try {
        std::vector<HistEntry> table(n_tensors);
        int64_t units = 0;
        for (int t = 0; t < n_tensors; ++t) {
            HistEntry& e = table[t];
            e.values = reinterpret_cast<const void*>(static_cast<uintptr_t>(values[t]));
            const int rc = check_flat(e.values, dtypes[t], numels[t], periods[t]);
            if (rc != GEFEN_B200_OK) return rc;
            e.period = periods[t];
            e.nb = numels[t] / periods[t];
            e.dtype = dtypes[t];
            e.vec = e.period % 8 == 0 && aligned16(e.values) && e.dtype != GEFEN_B200_F64;
            e.first_unit = units;
            units += (e.nb + hist_unit_blocks(e.period) - 1) / hist_unit_blocks(e.period);
            GEFEN_CHECK_ARG(e.period <= 0x7fffffffll, "Period %lld is too large.", static_cast<long long>(e.period));
        }
        GEFEN_CHECK_CUDA(cudaMemsetAsync(rows, 0, sizeof(int64_t) * histogram_bins * n_tensors, stream));
        GEFEN_CHECK_CUDA(cudaMemcpyAsync(device_table, table.data(), sizeof(HistEntry) * n_tensors, cudaMemcpyHostToDevice, stream));
        if (units > 0) {
            const int grid = static_cast<int>(std::min<int64_t>(units, static_cast<int64_t>(sm_count()) * 6));
            histogram_many_kernel<<<grid, kThreads, 0, stream>>>(static_cast<const HistEntry*>(device_table), n_tensors, units, histogram_bins,
                                                                 reinterpret_cast<unsigned long long*>(rows));
            GEFEN_CHECK_CUDA(cudaGetLastError());
        }
        histogram_total_kernel<<<(histogram_bins + kThreads - 1) / kThreads, kThreads, 0, stream>>>(
            reinterpret_cast<const long long*>(rows), n_tensors, histogram_bins, total);
        GEFEN_CHECK_CUDA(cudaGetLastError());
        return GEFEN_B200_OK;
    } catch (const std::bad_alloc&) {
        return fail(GEFEN_B200_ERUNTIME, "Out of host memory for the histogram table.");
    }
}

int gefen_b200_average_within_block_variance(const void* values, int dtype, int64_t numel, int64_t period,
                                             int input_is_squared, double* stats, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_flat(values, dtype, numel, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(stats != nullptr, "Expected a non-null stats buffer.");
    GEFEN_CHECK_CUDA(cudaMemsetAsync(stats, 0, sizeof(double), stream));
    const int64_t nb = numel / period;
    if (nb == 0) return GEFEN_B200_OK;
    const int grid = persistent_grid(nb, kWarps, 8);
    GEFEN_DISPATCH_S(dtype, {
        if (input_is_squared) block_moment_kernel<S, true, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(values), period, nb, stats);
        else block_moment_kernel<S, false, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(values), period, nb, stats);
    });
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

int gefen_b200_average_within_block_coefficient_of_variation(const void* values, int dtype, int64_t numel,
                                                             int64_t period, int input_is_squared, double* stats,
                                                             void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_flat(values, dtype, numel, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(stats != nullptr, "Expected a non-null stats buffer.");
    GEFEN_CHECK_CUDA(cudaMemsetAsync(stats, 0, 3 * sizeof(double), stream));
    const int64_t nb = numel / period;
    if (nb == 0) return GEFEN_B200_OK;
    const int grid = persistent_grid(nb, kWarps, 8);
    GEFEN_DISPATCH_S(dtype, {
        if (input_is_squared) block_moment_kernel<S, true, true><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(values), period, nb, stats);
        else block_moment_kernel<S, false, true><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(values), period, nb, stats);
    });
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

int64_t gefen_b200_period_scratch_doubles(int64_t numel, int64_t period) {
    if (period <= 0 || numel < 0) return 0;
    return numel / period + 1 + kMaxPartials;
}

int gefen_b200_average_adjacent_log_block_mean_difference(const void* values, int dtype, int64_t numel,
                                                          int64_t period, int input_is_squared, double epsilon,
                                                          double* stats, double* block_sums, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_flat(values, dtype, numel, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(epsilon > 0.0, "Expected a positive epsilon.");
    GEFEN_CHECK_ARG(numel / period >= 2, "Expected at least two blocks to compare adjacent block means.");
    GEFEN_CHECK_ARG(stats != nullptr && block_sums != nullptr, "Expected non-null stats and block_sums.");
    return adjacent_score(values, dtype, numel, period, input_is_squared != 0, epsilon, stats, block_sums, stream);
}

int64_t gefen_b200_period_scan_many_scratch_doubles(int n_tensors, const int64_t* numels, const int32_t* offsets,
                                                    const int64_t* periods) {
    if (n_tensors <= 0 || numels == nullptr || offsets == nullptr || periods == nullptr) return 0;
    for (int t = 0; t < n_tensors; ++t) {
        if (numels[t] <= 0 || offsets[t + 1] < offsets[t]) return 0;
        for (int i = offsets[t]; i < offsets[t + 1]; ++i)
            if (periods[i] <= 0 || numels[t] % periods[i] != 0) return 0;
    }
    try {
        const std::vector<uint64_t> values(n_tensors, 0);
        const std::vector<int32_t> dtypes(n_tensors, GEFEN_B200_F32);
        return make_scan_plan(n_tensors, values.data(), dtypes.data(), numels, offsets, periods).total;
    } catch (const std::bad_alloc&) {
        return 0;
    }
}

int64_t gefen_b200_period_scan_scratch_doubles(int64_t numel, const int64_t* host_periods, int n_periods) {
    if (n_periods <= 0) return 0;
    const int32_t offsets[2] = {0, n_periods};
    return gefen_b200_period_scan_many_scratch_doubles(1, &numel, offsets, host_periods);
}

int gefen_b200_period_scan_many(int n_tensors, const uint64_t* values, const int32_t* dtypes, const int64_t* numels,
                                const int32_t* offsets, const int64_t* periods, int input_is_squared, double epsilon,
                                double* stats, double* scratch, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(n_tensors >= 0, "Expected a non-negative number of tensors.");
    if (n_tensors == 0) return GEFEN_B200_OK;
    GEFEN_CHECK_ARG(values && dtypes && numels && offsets && periods && stats && scratch, "Expected non-null arguments.");
    GEFEN_CHECK_ARG(epsilon > 0.0, "Expected a positive epsilon.");
    for (int t = 0; t < n_tensors; ++t) {
        GEFEN_CHECK_ARG(offsets[t + 1] >= offsets[t], "Expected ascending offsets.");
        for (int i = offsets[t]; i < offsets[t + 1]; ++i) {
            const int rc = check_flat(reinterpret_cast<const void*>(static_cast<uintptr_t>(values[t])), dtypes[t], numels[t], periods[i]);
            if (rc != GEFEN_B200_OK) return rc;
            GEFEN_CHECK_ARG(numels[t] / periods[i] >= 2, "Expected at least two blocks for period %lld.", static_cast<long long>(periods[i]));
        }
    }
    try {
        const ScanPlan plan = make_scan_plan(n_tensors, values, dtypes, numels, offsets, periods);
        const int n = static_cast<int>(plan.candidates.size());
        if (n == 0) return GEFEN_B200_OK;
        unsigned long long* invalid = reinterpret_cast<unsigned long long*>(scratch);
        ScanBase* bases = reinterpret_cast<ScanBase*>(scratch + plan.bases_offset);
        ScanCandidate* table = reinterpret_cast<ScanCandidate*>(scratch + plan.candidates_offset);
        int* place = reinterpret_cast<int*>(scratch + plan.place_offset);
        // one copy for the three tables, which lie one after the other
        std::vector<double> image(static_cast<size_t>(plan.total - plan.bases_offset), 0.0);
        memcpy(image.data(), plan.bases.data(), plan.bases.size() * sizeof(ScanBase));
        memcpy(image.data() + (plan.candidates_offset - plan.bases_offset), plan.candidates.data(), plan.candidates.size() * sizeof(ScanCandidate));
        memcpy(image.data() + (plan.place_offset - plan.bases_offset), plan.place.data(), plan.place.size() * sizeof(int));
        GEFEN_CHECK_CUDA(cudaMemsetAsync(invalid, 0, sizeof(unsigned long long) * n_tensors, stream));
        GEFEN_CHECK_CUDA(cudaMemcpyAsync(bases, image.data(), image.size() * 8, cudaMemcpyHostToDevice, stream));
        const int64_t cap = static_cast<int64_t>(sm_count()) * 8;
        const int n_bases = static_cast<int>(plan.bases.size());
        const int grid = static_cast<int>(std::min(plan.base_units, 4 * cap));
        if (input_is_squared) scan_base_kernel<true><<<grid, kThreads, 0, stream>>>(scratch, bases, n_bases, plan.base_units, epsilon, invalid);
        else scan_base_kernel<false><<<grid, kThreads, 0, stream>>>(scratch, bases, n_bases, plan.base_units, epsilon, invalid);
        GEFEN_CHECK_CUDA(cudaGetLastError());
        for (size_t level = 1; level + 1 < plan.level_begin.size(); ++level) {
            const int64_t units = plan.level_units[level];
            scan_regroup_kernel<<<static_cast<int>(std::min(units, 4 * cap)), kThreads, 0, stream>>>(
                scratch, table + plan.level_begin[level], plan.level_begin[level + 1] - plan.level_begin[level], units);
            GEFEN_CHECK_CUDA(cudaGetLastError());
        }
        double* partials = scratch + plan.partial_offset;
        scan_partial_kernel<<<static_cast<unsigned>(plan.partials), kThreads, 0, stream>>>(scratch, table, n, partials);
        GEFEN_CHECK_CUDA(cudaGetLastError());
        scan_final_kernel<<<(n + kWarps - 1) / kWarps, kThreads, 0, stream>>>(partials, table, place, n, invalid, stats);
        GEFEN_CHECK_CUDA(cudaGetLastError());
        return GEFEN_B200_OK;
    } catch (const std::bad_alloc&) {
        return fail(GEFEN_B200_ERUNTIME, "Out of host memory for the plan of the period scan.");
    }
}

int gefen_b200_period_scan(const void* values, int dtype, int64_t numel, int input_is_squared, double epsilon,
                           const int64_t* host_periods, int n_periods, double* stats, double* scratch,
                           void* stream) {
    GEFEN_CHECK_ARG(n_periods >= 0, "Expected a non-negative number of periods.");
    if (n_periods == 0) return GEFEN_B200_OK;
    GEFEN_CHECK_ARG(host_periods != nullptr && stats != nullptr && scratch != nullptr,
                    "Expected non-null periods, stats and scratch.");
    const uint64_t pointer = static_cast<uint64_t>(reinterpret_cast<uintptr_t>(values));
    const int32_t offsets[2] = {0, n_periods}, tag = dtype;
    return gefen_b200_period_scan_many(1, &pointer, &tag, &numel, offsets, host_periods, input_is_squared, epsilon, stats, scratch, stream);
}

int gefen_b200_divisors(int64_t n, int64_t* out, int capacity) {
    if (n <= 0 || (out == nullptr && capacity > 0)) return 0;
    int count = 0;   // ascending: the small divisors, then their cofactors backwards
    int64_t root = 0;
    for (int64_t i = 1; i * i <= n; ++i) {
        if (n % i != 0) continue;
        if (count < capacity) out[count] = i;
        ++count;
        root = i;
    }
    const int small = count;
    for (int s = small - 1; s >= 0; --s) {
        if (s >= capacity) return -1;
        if (s == small - 1 && root * root == n) continue;
        if (count < capacity) out[count] = n / out[s];
        ++count;
    }
    return count;
}

int gefen_b200_lloyd_accumulate(const void* grad_flat, int grad_dtype, int64_t numel, int64_t period,
                                const float* codebook, int codebook_size, const void* codebook_ws, float* sums,
                                int64_t* counts, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_flat(grad_flat, grad_dtype, numel, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(sums != nullptr && counts != nullptr, "Expected non-null sums and counts.");
    const void* ws = nullptr;
    rc = resolve_codebook_ws(codebook, codebook_size, codebook_ws, stream, &ws);
    if (rc != GEFEN_B200_OK) return rc;
    const int64_t nb = numel / period;
    if (nb == 0) return GEFEN_B200_OK;
    unsigned long long* cnt = reinterpret_cast<unsigned long long*>(counts);
    const unsigned char* wsb = static_cast<const unsigned char*>(ws);
    GEFEN_CHECK_ARG(aligned16(ws), "Expected a 16-byte aligned codebook workspace.");
    if (period <= 8192) {
        const int grid = persistent_grid(nb, kWarps, 4);
        if (period % 8 == 0 && aligned16(grad_flat) && grad_dtype != GEFEN_B200_F64) {
            GEFEN_DISPATCH_S(grad_dtype, lloyd_accumulate_kernel<S, 32, true><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, wsb, codebook_size, sums, cnt));
        } else {
            GEFEN_DISPATCH_S(grad_dtype, lloyd_accumulate_kernel<S, 32, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, wsb, codebook_size, sums, cnt));
        }
    } else {
        const int grid = persistent_grid(nb, 1, 4);
        GEFEN_DISPATCH_S(grad_dtype, lloyd_accumulate_kernel<S, 256, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, wsb, codebook_size, sums, cnt));
    }
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

int gefen_b200_lloyd_mse(const void* grad_flat, int grad_dtype, int64_t numel, int64_t period,
                         const float* old_codebook, const float* new_codebook, int codebook_size,
                         const void* old_codebook_ws, float* mse_normalized_sum, float* mse_original_sum,
                         void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_flat(grad_flat, grad_dtype, numel, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(new_codebook != nullptr && mse_normalized_sum != nullptr && mse_original_sum != nullptr,
                    "Expected non-null new_codebook and outputs.");
    const void* ws = nullptr;
    rc = resolve_codebook_ws(old_codebook, codebook_size, old_codebook_ws, stream, &ws);
    if (rc != GEFEN_B200_OK) return rc;
    const int64_t nb = numel / period;
    if (nb == 0) return GEFEN_B200_OK;
    const unsigned char* wsb = static_cast<const unsigned char*>(ws);
    GEFEN_CHECK_ARG(aligned16(ws), "Expected a 16-byte aligned codebook workspace.");
    if (period <= 8192) {
        const int grid = persistent_grid(nb, kWarps, 4);
        if (period % 8 == 0 && aligned16(grad_flat) && grad_dtype != GEFEN_B200_F64) {
            GEFEN_DISPATCH_S(grad_dtype, lloyd_mse_kernel<S, 32, true><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, wsb, new_codebook, codebook_size, mse_normalized_sum, mse_original_sum));
        } else {
            GEFEN_DISPATCH_S(grad_dtype, lloyd_mse_kernel<S, 32, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, wsb, new_codebook, codebook_size, mse_normalized_sum, mse_original_sum));
        }
    } else {
        const int grid = persistent_grid(nb, 1, 4);
        GEFEN_DISPATCH_S(grad_dtype, lloyd_mse_kernel<S, 256, false><<<grid, kThreads, 0, stream>>>(static_cast<const S*>(grad_flat), period, nb, wsb, new_codebook, codebook_size, mse_normalized_sum, mse_original_sum));
    }
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

}  // extern "C"
