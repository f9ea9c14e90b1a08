// Exact 1-D k-means by dynamic programming, stage-parallel on the device in fp64.
//
// Same recurrence, same fp64 expressions and the same tie rule as the reference's numba kernel
// (quantization.py:92-145): dp[e][c] = min over s in [c, e] of dp[s-1][c-1] + cost(s, e), the FIRST
// minimum in ascending s winning (strict `<`). Every candidate is an independent expression, so
// evaluating the candidates of one stage in parallel and reducing with "smaller value, then
// smaller s" gives bit-identical tables. Arithmetic uses the _rn intrinsics so that nothing is
// contracted into FMAs (numba does not contract either).
#include "common.cuh"

namespace gefen {

constexpr int kDpThreads = 256;

__device__ __forceinline__ double segment_cost(const double* pw, const double* pwx, const double* pwx2, int s, int e,
                                               int mode) {
    const double sw = __dsub_rn(pw[e], pw[s - 1]);
    const double swx = __dsub_rn(pwx[e], pwx[s - 1]);
    const double swx2 = __dsub_rn(pwx2[e], pwx2[s - 1]);
    if (mode != 0) {
        // forced centre fc = -1 (mode 1) or +1 (mode 2):
        // (swx2 - (2.0*fc)*swx) + (fc*fc)*sw, evaluated left to right as in the reference.
        const double fc = mode == 1 ? -1.0 : 1.0;
        const double a = __dsub_rn(swx2, __dmul_rn(__dmul_rn(2.0, fc), swx));
        return __dadd_rn(a, __dmul_rn(__dmul_rn(fc, fc), sw));
    }
    return __dsub_rn(swx2, __ddiv_rn(__dmul_rn(swx, swx), sw));
}

// One warp per end index e. dp_prev = dp[.][c-1], dp_cur = dp[.][c], starts_prev = the best starts of stage c - 1.
//
// Only the starts that can be the minimum are evaluated (a stage of 4096 points has 8.4 M candidates otherwise, each
// with a double-precision division; the 256 stages took 5.6 ms). With U the candidate at the previous stage's best
// start, a start s is out if dp_prev[s-1] > U + margin (the segment's cost is not negative) and all larger starts with
// it (dp_prev grows with s), or if cost(s, e) > U + margin (dp_prev is not negative) and all smaller starts with it
// (a segment's cost grows as it is extended). These hold exactly for exact costs; computed ones differ by rounding:
// a prefix sum carries at most n 2^-53 of the total T = sum w + sum w x^2 (by Cauchy-Schwarz no other
// sum is larger) where errors do not cancel, typically sqrt(n) 2^-53 T, a cost a few of those, and dp_prev a
// cost's error per stage. The differences that matter are those between prefixes that all candidates read from the same
// arrays; the functions above are evaluated on these arrays as they are, so what is left is the rounding of the
// differences, product, quotient and sums: at most 8 * 2^-53 T per cost and K times that in dp_prev, 2.3e-13 T for 256
// stages. margin = 1e-10 T (clusters are 1e-8 T and more) covers it, and the accumulated error of the prefixes
// (4096 * 2^-53 T = 4.5e-13 T per element at the very worst), several hundred times over. Every start whose value is U
// or less is therefore evaluated, with the expressions and the tie rule as before: the tables are the same bits.
constexpr double kMargin = 1e-10;

__global__ void __launch_bounds__(kDpThreads) dp_stage_kernel(const double* __restrict__ pw, const double* __restrict__ pwx,
                                                              const double* __restrict__ pwx2, int num_points, int c,
                                                              int mode, const double* __restrict__ dp_prev,
                                                              const int* __restrict__ starts_prev,
                                                              double* __restrict__ dp_cur, int* __restrict__ backtrack,
                                                              int first_end) {
    const int lane = threadIdx.x & 31;
    const int e = first_end + static_cast<int>(blockIdx.x) * (kDpThreads / 32) + (threadIdx.x >> 5);
    if (e > num_points) return;
    if (e < c) {
        if (lane == 0) { dp_cur[e] = INFINITY; backtrack[e] = -1; }
        return;
    }
    int lo = c, hi = e;      // candidates [lo, hi]
    if (c == 1) {
        hi = 1;              // dp[s - 1][0] is infinite for every other start
    } else {
        const int guess = starts_prev[e] > c ? starts_prev[e] : c;
        const double bound = dp_prev[guess - 1] + segment_cost(pw, pwx, pwx2, guess, e, mode) +
                             kMargin * (pw[num_points] + pwx2[num_points]);
        if (isfinite(bound)) {
            // starts below `lo` cost too much: 32 probes over [lo, guess], twice
            for (int round = 0; round < 2; ++round) {
                const int step = (guess - lo) / 32 + 1;
                const int probe = lo + lane * step;
                const bool out = probe < guess && segment_cost(pw, pwx, pwx2, probe, e, mode) > bound;
                const unsigned votes = __ballot_sync(0xffffffffu, out);
                if (votes != 0u) lo = lo + (31 - __clz(votes)) * step + 1;
                if (step == 1) break;
            }
            // starts above `hi` have too much before them
            int low = guess;
            for (int round = 0; round < 2; ++round) {
                const int step = (hi - low) / 32 + 1;
                const int probe = low + (lane + 1) * step;
                const bool out = probe <= hi && dp_prev[probe - 1] > bound;
                const unsigned votes = __ballot_sync(0xffffffffu, out);
                if (votes != 0u) {
                    const int first = __ffs(votes) - 1;
                    hi = low + (first + 1) * step - 1;
                    low = low + first * step;
                } else {
                    low = low + 31 * step < hi ? low + 31 * step : hi;
                }
                if (step == 1) break;
            }
        }
    }
    double best = INFINITY;
    int best_s = -1;
    for (int s = lo + lane; s <= hi; s += 32) {
        const double cand = __dadd_rn(dp_prev[s - 1], segment_cost(pw, pwx, pwx2, s, e, mode));
        if (cand < best) { best = cand; best_s = s; }
    }
    // reduce: smaller value wins, on equal values the smaller start index (-1 = no candidate)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int os = __shfl_xor_sync(0xffffffffu, best_s, o);
        if (os >= 0 && (best_s < 0 || ov < best || (ov == best && os < best_s))) { best = ov; best_s = os; }
    }
    if (lane == 0) {
        dp_cur[e] = best;
        backtrack[e] = best_s;
    }
}

__global__ void dp_init_kernel(double* dp0, int num_points) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= num_points) dp0[i] = (i == 0) ? 0.0 : INFINITY;
}

// Walks the backtrack table from (num_points, K) and emits the centres (reference :132-145).
__global__ void dp_backtrack_kernel(const double* __restrict__ pw, const double* __restrict__ pwx, int num_points,
                                    int num_codebooks, int force, const int* __restrict__ backtrack,
                                    float* __restrict__ codebook, int* __restrict__ status) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int e = num_points;
    for (int c = num_codebooks; c >= 1; --c) {
        const int s = backtrack[static_cast<long long>(c) * (num_points + 1) + e];
        if (s < 1) { *status = 1; return; }
        if (force && c == 1) codebook[c - 1] = -1.0f;
        else if (force && c == num_codebooks) codebook[c - 1] = 1.0f;
        else {
            const double sw = __dsub_rn(pw[e], pw[s - 1]);
            const double swx = __dsub_rn(pwx[e], pwx[s - 1]);
            codebook[c - 1] = static_cast<float>(__ddiv_rn(swx, sw));
        }
        e = s - 1;
    }
    *status = 0;
}

}  // namespace gefen

using namespace gefen;

extern "C" {

int64_t gefen_b200_exact_dp_scratch_bytes(int num_points, int num_codebooks) {
    if (num_points < 1 || num_codebooks < 1) return 0;
    const int64_t n1 = static_cast<int64_t>(num_points) + 1;
    // two dp columns, the backtrack table, one status word (padded)
    return 2 * n1 * 8 + (static_cast<int64_t>(num_codebooks) + 1) * n1 * 4 + 16;
}

int gefen_b200_exact_dp(const double* prefix_w, const double* prefix_wx, const double* prefix_wx2, int num_points,
                        int num_codebooks, int force_endpoints, void* dp_scratch, float* codebook_out, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(prefix_w && prefix_wx && prefix_wx2 && dp_scratch && codebook_out, "Expected non-null arguments.");
    GEFEN_CHECK_ARG(num_points >= 1, "Cannot run exact DP on an empty histogram.");
    GEFEN_CHECK_ARG(num_codebooks >= 1 && num_codebooks <= num_points,
                    "Expected 1 <= num_codebooks <= num_points (the padded path is handled by the caller).");
    GEFEN_CHECK_ARG((reinterpret_cast<uintptr_t>(dp_scratch) & 7u) == 0, "Expected 8-byte aligned scratch.");
    const int64_t n1 = static_cast<int64_t>(num_points) + 1;
    double* dp_a = static_cast<double*>(dp_scratch);
    double* dp_b = dp_a + n1;
    int* backtrack = reinterpret_cast<int*>(dp_b + n1);
    int* status = backtrack + (static_cast<int64_t>(num_codebooks) + 1) * n1;
    dp_init_kernel<<<static_cast<int>((n1 + 255) / 256), 256, 0, stream>>>(dp_a, num_points);
    GEFEN_CHECK_CUDA(cudaGetLastError());
    double* prev = dp_a;
    double* cur = dp_b;
    for (int c = 1; c <= num_codebooks; ++c) {
        int mode = 0;
        if (force_endpoints && c == 1) mode = 1;
        else if (force_endpoints && c == num_codebooks) mode = 2;
        // only dp[num_points][K] is read from the last stage
        const int first_end = (c == num_codebooks) ? num_points : 0;
        const int n_ends = num_points - first_end + 1;
        dp_stage_kernel<<<(n_ends + kDpThreads / 32 - 1) / (kDpThreads / 32), kDpThreads, 0, stream>>>(
            prefix_w, prefix_wx, prefix_wx2, num_points, c, mode, prev, backtrack + static_cast<int64_t>(c - 1) * n1, cur,
            backtrack + static_cast<int64_t>(c) * n1, first_end);
        GEFEN_CHECK_CUDA(cudaGetLastError());
        double* t = prev; prev = cur; cur = t;
    }
    dp_backtrack_kernel<<<1, 32, 0, stream>>>(prefix_w, prefix_wx, num_points, num_codebooks, force_endpoints ? 1 : 0,
                                              backtrack, codebook_out, status);
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

}  // extern "C"
