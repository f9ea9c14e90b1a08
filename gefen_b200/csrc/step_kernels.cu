// The steady-state Gefen step on sm_100a.
//
// What one block (`period` consecutive elements sharing a magnitude and a second moment) goes
// through, in the reference's arithmetic (kernels/automatic_gefen_fused_kernel.cu:239-318 for the
// AdamW form, :320-407 for period 1, :169-237 for GefenMuon; kernels/automatic_vmean_kernel.cu:12-51
// for the second moment; gefen.py:1280-1281 for the decoupled weight decay):
//
//   m_i   = beta1 * (mag * cb[code_i]) + (1 - beta1) * g_i              (fp32)
//   mag'  = max_i |m_i|            stored rounded to the state dtype
//   code' = nearest codebook entry of m_i / mag'   (IEEE divide by the un-rounded fp32 mag')
//   p_i  -= cb[code'_i] * mag' * step * lr,   step = (1/bc1) / (sqrt(v/bc2) + eps)
//
// Four kernels:
//  * step_ring_kernel - what every usual tensor takes: one warp owns one block, or several blocks when they are not longer
//    than 1024 elements (see lanes_shift). Codes and gradients come through shared memory by bulk (TMA) copies one unit
//    ahead, in chunks of eight elements (four, two or one where the block length or a pointer is a multiple of no more);
//    the updated momenta wait in tensor memory while the block's absmax is reduced with shuffles, then they are re-encoded
//    and the parameters updated: codes, gradients and parameters cross HBM exactly once (8 B/element in bf16, 14 in fp32).
//    The codebook arrives by one bulk copy per CTA, which turns it into tables with a copy per lane (see LaneTables). No
//    __syncthreads after set-up; the loops are short so the code stays in the instruction cache. What bounds it and what it
//    measured stands at the kernel.
//  * step_vec_kernel - the same without the ring: gradients averaged over ranks, chunks below eight with peer stores or
//    whose reads of the buffers would conflict, blocks too long for the buffers (see route), fp32 launches that make one
//    round of it and two of the ring kernel (see launch_ring); momenta in shared memory or formed twice (see Momenta).
//  * step_vector_kernel - period-1 tensors, one warp per magnitude, everything in registers.
//  * step_generic_kernel - blocks of more than 8192 elements, fp64, 4-bit packed codes, and vectors of ranks with peers:
//    two passes with scalar accesses, the second pass re-reading from L1/L2.
// All take their tensors from a descriptor table (one launch for many tensors); a single-tensor
// call passes a one-row table inside the kernel parameters. For data-parallel ranks whose buffers
// are mapped into each other's address space the kernels can also store every updated parameter
// to the peers' copies (the all-gather) and average the gradients over the peers' copies while
// reading them (the reduce-scatter): see StepLaunch.
#include "common.cuh"

#include <mutex>
#include <stdlib.h>
#include <string.h>

namespace gefen {

// fp32 contraction choices. They reproduce what nvcc emits for the reference source when it is
// compiled with its own flags (-O3, fmad on): a*b + c*d becomes fma(a, b, c*d) and p - a*b becomes
// fma(-a, b, p); checked on a B200 against the reference's own kernels. The CPU oracle makes the
// same choices explicitly.
__device__ __forceinline__ float ema_update(float beta, float cur, float omb, float g) {
    return fmaf(beta, cur, omb * g);
}
// In the reference's period-1 kernel (automatic_gefen_fused_kernel.cu:360, :392) nvcc fuses the other
// product of the same expression; measured against the reference build, bit-identical with this form.
__device__ __forceinline__ float ema_update_period1(float beta, float cur, float omb, float g) {
    return fmaf(omb, g, beta * cur);
}

struct StepLaunch {
    const gefen_b200_step_tensor_t* table;  // device table, or nullptr: the rows in the kernel params
    int n_tensors;
    int stage_floats;                       // staged kernel: floats of staging per warp (>= max period)
    int ring_g, ring_codes;                 // ring kernel: bytes of a warp's buffers for one unit's gradients and codes
    int hold_columns, tmem_columns;         // ring kernel: tensor-memory columns of a warp and of the CTA
    long long total_blocks;
    const unsigned char* ws;                // codebook workspace
    const float* stepsize;                  // optional precomputed per-block step (single tensor only)
    // ZeRO-1 with the all-gather fused in: every updated parameter is also stored into the same
    // place of n_peers other GPUs' parameter buffers (byte distance from this GPU's buffer to
    // theirs in this process's address space; plain peer stores over NVLink, no loads).
    int n_peers;
    long long peer_delta[GEFEN_B200_MAX_PEERS];
    // ... and with the reduce-scatter fused in: the gradient of an element is grad_scale times the
    // sum over n_grad_srcs buffers (byte distances from this GPU's gradient buffer, rank order, 0
    // for this rank itself), rounded to the gradient dtype. 0 sources: gradients are used as they are.
    int n_grad_srcs;
    float grad_scale;
    long long grad_delta[GEFEN_B200_MAX_PEERS + 1];
    // NVLink multicast (NVSwitch) mappings of the ranks' buffers, as byte distances from this GPU's own
    // buffer; 0 = not used. grad_mc_delta: the staged kernel reads every gradient chunk with one
    // multimem.ld_reduce (the switch adds the ranks' copies, fp32 accumulation) instead of n_grad_srcs
    // peer loads. param_mc_delta: every updated parameter chunk leaves with one multimem.st that the
    // switch delivers to all ranks' copies, this GPU's included, instead of a local store plus n_peers
    // peer stores.
    long long grad_mc_delta;
    long long param_mc_delta;
    // iteration limits of the waits for the staged tables and the ring's inputs (g_stage_spin_limit, g_input_spin_limit)
    unsigned int spin_limit, input_limit;
    // the launch before this one (host only) and the one after it belong to the same step (see let_successor_in)
    int follows, leads;
};

// Descriptors that travel with the launch itself: a call of up to this many tensors needs no copy of its table to the
// device (kernel parameters hold 4 KB; the copy costs the host about 5 us and the GPU a launch gap).
constexpr int kParamRows = 24;
struct StepRows {
    gefen_b200_step_tensor_t row[kParamRows];
};
static_assert(sizeof(StepRows) + sizeof(StepLaunch) <= 4096, "kernel parameter space");
// Buffers that a chunk of averaged gradients is read from; the multicast mapping is one.
__host__ __device__ __forceinline__ int chunk_sources(const StepLaunch& L) { return L.grad_mc_delta != 0 ? 1 : L.n_grad_srcs; }

// Set (never cleared by a kernel) when a bounded wait ran out and the CTA left without doing its
// share of the step: bit 0 = the table staging or the inputs of a step kernel, bit 1 = its shared-memory layout does not fit. Read and cleared by
// gefen_b200_step_status on the host.
__device__ int g_step_status;

// Two fp32 operations in one instruction (sm_100: each half is the IEEE operation of its own, so the results
// are those of the scalar forms). The step kernels are bound by instruction issue; their arithmetic runs on pairs.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpair(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

template <typename T> __device__ __forceinline__ T* peer_ptr(T* p, long long delta) {
    return reinterpret_cast<T*>(reinterpret_cast<uintptr_t>(p) + delta);
}

// Every step kernel stages the head of the codebook workspace: codebook, thresholds, size.
constexpr int kSmemWs = kWsLutOff;
static_assert(kSmemWs % 16 == 0, "bulk copies move multiples of 16 bytes");
constexpr int kMaxSmem = 227 * 1024;

struct SmemView {
    const float* cb;             // 256, padded with the last entry
    const float* thr;            // 256, padded with +inf
    int k;                       // true codebook size
};

// Stages the tables with one bulk copy. Returns false (uniformly for the CTA) if the copy did
// not land within `spin_limit` polls of its barrier; the status word is raised then, and the CTA
// still gives the copy a second, long bounded wait before it returns, so that it does not leave
// while a copy into its shared memory is in flight.
constexpr unsigned int kStageDrainLimit = 4000000u;
__device__ __forceinline__ bool stage_tables(const unsigned char* ws, unsigned char* smem, SmemView& view,
                                             unsigned int spin_limit) {
    __shared__ uint64_t bar;
    __shared__ int ok;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar, kSmemWs);
        bulk_copy_g2s(smem, ws, kSmemWs, &bar);
        ok = mbar_wait_bounded(&bar, 0, spin_limit) ? 1 : 0;
        if (!ok) {
            atomicOr(&g_step_status, 1);
            mbar_wait_bounded(&bar, 0, kStageDrainLimit);
        }
    }
    __syncthreads();
    view.cb = reinterpret_cast<const float*>(smem + kWsCodebookOff);
    view.thr = reinterpret_cast<const float*>(smem + kWsThresholdOff);
    view.k = 1;
    if (!ok) return false;
    view.k = reinterpret_cast<const int*>(smem + kWsMetaOff)[0];
    return true;
}

__device__ __forceinline__ float adam_step_size(float v, float bc1, float bc2, float eps) {
    const float corrected = v / bc2;
    return (1.0f / bc1) / (sqrtf(corrected) + eps);
}

// Finds the row that owns global block `gb` (rows sorted by first_block).
__device__ __forceinline__ int find_tensor(const gefen_b200_step_tensor_t* table, int n, long long gb) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (table[mid].first_block <= gb) lo = mid; else hi = mid - 1;
    }
    return lo;
}
// The same by a whole warp for one gb: 32 probes at a time, so that a table of 148 rows takes two dependent loads
// instead of eight.
__device__ __forceinline__ int find_tensor_warp(const gefen_b200_step_tensor_t* table, int n, long long gb) {
    int lo = 0, count = n;   // the row lies in [lo, lo + count)
    while (count > 1) {
        const int step = (count + 31) >> 5;
        const int probe = static_cast<int>(threadIdx.x & 31) * step;
        const unsigned votes = __ballot_sync(0xffffffffu, probe < count && table[lo + probe].first_block <= gb);
        const int last = 31 - __clz(votes);   // (lane 0 always votes: the rows before lo are out)
        lo += last * step;
        count = count - last * step < step ? count - last * step : step;
    }
    return lo;
}

// The launches of one step follow each other without waiting (programmatic dependent launch): they work on different
// tensors. A kernel lets its successor in at its start, and waits for its predecessor at its end, so that whatever
// follows the last of them follows all of them.
// The last one lets nobody in: what follows may be any kernel of the program that was launched programmatically, and one
// that holds tensor memory while it waits for this one to end would keep a CTA of step_ring_kernel on its SM from ever
// getting its columns. (A launch of this step gives its columns back before it waits for the one before it.)
__device__ __forceinline__ void let_successor_in(const StepLaunch& L) {
    if (L.leads) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// --------------------------------------------------------------------------- vector IO
// A "chunk" is 8 consecutive elements: 8 code bytes, 16 B of bf16/f16 or 32 B of fp32. Everything is
// read once per step: the loads carry the streaming (evict-first) hint.
// 16-byte accesses to a multicast address: the store reaches every GPU's copy, the load returns the
// element-wise sum of all copies (added in the switch, fp32 accumulation for the 2-byte types).
__device__ __forceinline__ void multimem_store16(void* mc_addr, uint4 v) {
    asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(mc_addr), "r"(v.x), "r"(v.y), "r"(v.z),
                 "r"(v.w)
                 : "memory");
}
template <typename S> __device__ __forceinline__ uint4 multimem_load_sum16(const void* mc_addr);
template <> __device__ __forceinline__ uint4 multimem_load_sum16<__nv_bfloat16>(const void* mc_addr) {
    uint4 v;
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.bf16x2 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(mc_addr)
                 : "memory");
    return v;
}
template <> __device__ __forceinline__ uint4 multimem_load_sum16<__half>(const void* mc_addr) {
    uint4 v;
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.f16x2 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(mc_addr)
                 : "memory");
    return v;
}
template <> __device__ __forceinline__ uint4 multimem_load_sum16<float>(const void* mc_addr) {
    uint4 v;
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(mc_addr)
                 : "memory");
    return v;
}

// Storage form of one element: widening to fp32 and rounding back, two at a time.
template <typename S> struct Packed;
template <> struct Packed<__nv_bfloat16> {
    static __device__ __forceinline__ void unpack(uint32_t w, float& lo, float& hi) {
        lo = __uint_as_float(w << 16);
        hi = __uint_as_float(w & 0xFFFF0000u);
    }
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
};
template <> struct Packed<__half> {
    static __device__ __forceinline__ void unpack(uint32_t w, float& lo, float& hi) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w));
        lo = v.x;
        hi = v.y;
    }
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        const __half2 h = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
};

// V consecutive elements of a tensor: V code bytes and V * sizeof(S) bytes of gradients or parameters, aligned to
// the smaller of that and 16. V = 8 is the usual chunk; 4, 2 and 1 serve blocks and pointers that are multiples of
// no more than that.
template <typename S, int V> struct Chunk {
    static constexpr int kBytes = V * static_cast<int>(sizeof(S));
    static constexpr int kWords = kBytes < 4 ? 1 : kBytes / 4;
    uint32_t w[kWords];
    __device__ __forceinline__ void load(const void* base, long long chunk) {
        const char* p = static_cast<const char*>(base) + chunk * kBytes;
        if constexpr (kBytes >= 16) {
#pragma unroll
            for (int q = 0; q < kBytes / 16; ++q) {
                const uint4 v = __ldcs(reinterpret_cast<const uint4*>(p) + q);
                w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
            }
        } else if constexpr (kBytes == 8) {
            const uint2 v = __ldcs(reinterpret_cast<const uint2*>(p));
            w[0] = v.x; w[1] = v.y;
        } else if constexpr (kBytes == 4) {
            w[0] = __ldcs(reinterpret_cast<const unsigned int*>(p));
        } else {
            w[0] = __ldcs(reinterpret_cast<const unsigned short*>(p));
        }
    }
    __device__ __forceinline__ void load_again_later(const void* base, long long chunk) {   // (V = 8; no streaming hint)
        const uint4* p = reinterpret_cast<const uint4*>(static_cast<const char*>(base) + chunk * kBytes);
#pragma unroll
        for (int q = 0; q < kBytes / 16; ++q) {
            const uint4 v = p[q];
            w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
        }
    }
    __device__ __forceinline__ void load_shared(uint32_t at) {
        if constexpr (kBytes >= 16) {
#pragma unroll
            for (int q = 0; q < kBytes / 16; ++q)
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(w[4 * q]), "=r"(w[4 * q + 1]), "=r"(w[4 * q + 2]), "=r"(w[4 * q + 3]) : "r"(at + 16 * q));
        } else if constexpr (kBytes == 8) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(at));
        else if constexpr (kBytes == 4) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[0]) : "r"(at));
        else asm volatile("ld.shared.u16 %0, [%1];" : "=r"(w[0]) : "r"(at));
    }
    __device__ __forceinline__ void store(void* base, long long chunk) const {
        char* p = static_cast<char*>(base) + chunk * kBytes;
        if constexpr (kBytes >= 16) {
#pragma unroll
            for (int q = 0; q < kBytes / 16; ++q) {
                const uint4 v = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
                if constexpr (sizeof(S) == 4) __stcs(reinterpret_cast<uint4*>(p) + q, v);   // measured: streaming stores pay for fp32 only
                else reinterpret_cast<uint4*>(p)[q] = v;
            }
        } else if constexpr (kBytes == 8) {
            *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
        } else if constexpr (kBytes == 4) {
            *reinterpret_cast<unsigned int*>(p) = w[0];
        } else {
            *reinterpret_cast<unsigned short*>(p) = static_cast<unsigned short>(w[0]);
        }
    }
    // the element-wise sum over a multicast address; a store that reaches every GPU's copy (V = 8)
    __device__ __forceinline__ void load_sum(const void* mc_base, long long chunk) {
#pragma unroll
        for (int q = 0; q < kBytes / 16; ++q) {
            const uint4 v = multimem_load_sum16<S>(reinterpret_cast<const uint4*>(mc_base) + chunk * (kBytes / 16) + q);
            w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
        }
    }
    __device__ __forceinline__ void store_all(void* mc_base, long long chunk) const {
#pragma unroll
        for (int q = 0; q < kBytes / 16; ++q)
            multimem_store16(reinterpret_cast<uint4*>(mc_base) + chunk * (kBytes / 16) + q,
                             make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]));
    }
    __device__ __forceinline__ void unpack(float (&f)[V]) const {
        if constexpr (sizeof(S) == 4) {
#pragma unroll
            for (int i = 0; i < V; ++i) f[i] = __uint_as_float(w[i]);
        } else if constexpr (V == 1) {
            float unused;
            Packed<S>::unpack(w[0], f[0], unused);
        } else {
#pragma unroll
            for (int i = 0; i < V; i += 2) Packed<S>::unpack(w[i / 2], f[i], f[i + 1]);
        }
    }
    __device__ __forceinline__ void pack(const float (&f)[V]) {
        if constexpr (sizeof(S) == 4) {
#pragma unroll
            for (int i = 0; i < V; ++i) w[i] = __float_as_uint(f[i]);
        } else if constexpr (V == 1) {
            w[0] = Packed<S>::pack(f[0], 0.0f);
        } else {
#pragma unroll
            for (int i = 0; i < V; i += 2) w[i / 2] = Packed<S>::pack(f[i], f[i + 1]);
        }
    }
};

// The V code bytes of a chunk, in one or two words.
template <int V> struct CodeChunk {
    uint32_t w[V == 8 ? 2 : 1];
    __device__ __forceinline__ void load(const uint8_t* base, long long chunk) {
        if constexpr (V == 8) {
            const uint2 v = __ldcs(reinterpret_cast<const uint2*>(base) + chunk);
            w[0] = v.x; w[1] = v.y;
        } else if constexpr (V == 4) w[0] = __ldcs(reinterpret_cast<const unsigned int*>(base) + chunk);
        else if constexpr (V == 2) w[0] = __ldcs(reinterpret_cast<const unsigned short*>(base) + chunk);
        else w[0] = __ldcs(base + chunk);
    }
    __device__ __forceinline__ void load_again_later(const uint8_t* base, long long chunk) {   // (V = 8; no streaming hint)
        const uint2 v = reinterpret_cast<const uint2*>(base)[chunk];
        w[0] = v.x; w[1] = v.y;
    }
    __device__ __forceinline__ void load_shared(uint32_t at) {
        if constexpr (V == 8) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(at));
        else if constexpr (V == 4) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[0]) : "r"(at));
        else if constexpr (V == 2) asm volatile("ld.shared.u16 %0, [%1];" : "=r"(w[0]) : "r"(at));
        else asm volatile("ld.shared.u8 %0, [%1];" : "=r"(w[0]) : "r"(at));
    }
    __device__ __forceinline__ void store(uint8_t* base, long long chunk) const {
        if constexpr (V == 8) reinterpret_cast<uint2*>(base)[chunk] = make_uint2(w[0], w[1]);
        else if constexpr (V == 4) reinterpret_cast<uint32_t*>(base)[chunk] = w[0];
        else if constexpr (V == 2) reinterpret_cast<unsigned short*>(base)[chunk] = static_cast<unsigned short>(w[0]);
        else base[chunk] = static_cast<uint8_t>(w[0]);
    }
};

// Pulls the lines of this warp's NEXT block towards L2 while the current block is being worked on, so that its
// loads later pay an L2 hit instead of a DRAM round trip: one instruction of one lane for a whole range (widened
// to 16-byte boundaries).
__device__ __forceinline__ void prefetch_l2_range(const void* base, long long bytes) {
    const uintptr_t first = reinterpret_cast<uintptr_t>(base) & ~static_cast<uintptr_t>(15);
    const uintptr_t last = (reinterpret_cast<uintptr_t>(base) + bytes + 15) & ~static_cast<uintptr_t>(15);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(first), "r"(static_cast<uint32_t>(last - first)) : "memory");
}

// A block's updated momenta in the warp's staging slice: chunks of V floats; for V = 8 the first halves of all
// chunks, then the second halves (`half` floats further on), so that the 128-bit accesses of a full warp are
// conflict-free.
template <int V> __device__ __forceinline__ void stage_store(float* stage, int half, int c, const float (&m)[V]) {
    if constexpr (V == 8) {
        *reinterpret_cast<float4*>(stage + 4 * c) = make_float4(m[0], m[1], m[2], m[3]);
        *reinterpret_cast<float4*>(stage + half + 4 * c) = make_float4(m[4], m[5], m[6], m[7]);
    } else if constexpr (V == 4) *reinterpret_cast<float4*>(stage + 4 * c) = make_float4(m[0], m[1], m[2], m[3]);
    else if constexpr (V == 2) *reinterpret_cast<float2*>(stage + 2 * c) = make_float2(m[0], m[1]);
    else stage[c] = m[0];
}
template <int V> __device__ __forceinline__ void stage_load(const float* stage, int half, int c, float (&m)[V]) {
    if constexpr (V >= 4) {
        const float4 a = *reinterpret_cast<const float4*>(stage + 4 * c);
        m[0] = a.x; m[1] = a.y; m[2] = a.z; m[3] = a.w;
        if constexpr (V == 8) {
            const float4 b = *reinterpret_cast<const float4*>(stage + half + 4 * c);
            m[4] = b.x; m[5] = b.y; m[6] = b.z; m[7] = b.w;
        }
    } else if constexpr (V == 2) {
        const float2 a = *reinterpret_cast<const float2*>(stage + 2 * c);
        m[0] = a.x; m[1] = a.y;
    } else m[0] = stage[c];
}

// The same in tensor memory: each lane keeps V floats of its own per round, in V consecutive columns. Both are
// executed by the whole warp.
template <int V> __device__ __forceinline__ void hold_store(uint32_t at, const float (&m)[V]) {
    if constexpr (V == 8)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(at), "f"(m[0]), "f"(m[1]),
                     "f"(m[2]), "f"(m[3]), "f"(m[4]), "f"(m[5]), "f"(m[6]), "f"(m[7]) : "memory");
    else if constexpr (V == 4)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(m[0]), "f"(m[1]), "f"(m[2]), "f"(m[3]) : "memory");
    else if constexpr (V == 2)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(at), "f"(m[0]), "f"(m[1]) : "memory");
    else
        asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(at), "f"(m[0]) : "memory");
}
__device__ __forceinline__ void hold_stores_done() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
template <int V> __device__ __forceinline__ void hold_load(uint32_t at, float (&m)[V]) {
    if constexpr (V == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
                     : "=f"(m[0]), "=f"(m[1]), "=f"(m[2]), "=f"(m[3]), "=f"(m[4]), "=f"(m[5]), "=f"(m[6]), "=f"(m[7]) : "r"(at) : "memory");
    else if constexpr (V == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n\ttcgen05.wait::ld.sync.aligned;"
                     : "=f"(m[0]), "=f"(m[1]), "=f"(m[2]), "=f"(m[3]) : "r"(at) : "memory");
    else if constexpr (V == 2)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];\n\ttcgen05.wait::ld.sync.aligned;" : "=f"(m[0]), "=f"(m[1]) : "r"(at) : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\ttcgen05.wait::ld.sync.aligned;" : "=f"(m[0]) : "r"(at) : "memory");
}

// --------------------------------------------------------------------------- fast path
// The quantiser of the fast path. Data-dependent shared-memory reads are what it would be bound by (the data pipe
// serves one 128-byte row per cycle; a single table answers 32 random lanes in 3.5 to 6.6 rows), so every lane has
// copies of its own, on its own bank, and every read is one row:
//   rows   256 rows of 256 bytes: thr[e] of all 32 lanes, then cb[e] of all 32 lanes. A lane's address of entry e is
//          (e << 8) + 4 * lane, one byte permute from a code byte.
//   cells  256 words per lane; byte j of word r counts the thresholds below cell (j << 8) + r of 1024 uniform
//          cells over [-1, 1].
// x lies in cell N >> 7 with N = round(65472 x) + 65536 (the low mantissa bits of one FMA; 64 <= N <= 131008),
// a map that is monotone in x, so its entry is the count of its cell plus the thresholds of the same cell below
// x: `rounds` comparisons with the threshold of the entry so far, where rounds is the most thresholds that share a
// cell (one or two for codebooks of the fit; a comparison too many is always false). Codebooks that put more than
// kMaxRounds into a cell, or end below 1 (where the rule is not monotone), go through the binary search of exact_row.
constexpr int kRowBytes = 256;
constexpr int kSmemRows = kMaxCodebook * kRowBytes;
constexpr int kCells = 1024;
constexpr int kSmemCells = kCells * 32;
constexpr int kMaxRounds = 6;
// The tables lie at fixed shared-memory addresses, so that a read needs no address arithmetic beyond the row itself:
// the offsets are immediates of the loads. Dynamic shared memory starts behind the 1024 bytes that the system keeps
// and the kernels' static variables (at most 256 bytes; checked at run time, see fast_smem).
constexpr int kFixed = 1024 + 256;
constexpr int kRowsAt = kFixed, kCellsAt = kRowsAt + kSmemRows, kWsAt = kCellsAt + kSmemCells;
constexpr int kStageAt = kWsAt + kSmemWs;       // the warps' staging slices follow
constexpr int kSmemTables = kStageAt - 1024;    // dynamic shared memory up to the slices
static_assert(kFixed % 128 == 0 && kStageAt % 16 == 0, "a lane's words lie on its own bank, the staging slices hold float4");

extern __shared__ __align__(128) unsigned char g_smem[];
// The generic pointer of a fixed shared-memory address.
__device__ __forceinline__ unsigned char* fast_smem(int address) { return g_smem + (address - static_cast<int>(smem_u32(g_smem))); }

__device__ __forceinline__ float cell_position(float x) { return fmaf(x, 65472.0f, 8388608.0f + 65536.0f); }
__device__ __forceinline__ int threshold_cell(float t) {   // -1: below every x; kCells: above or equal to every x
    if (t < -1.0f) return -1;
    if (!(t < 1.0f)) return kCells;
    return static_cast<int>((__float_as_uint(cell_position(t)) & 0x1FFFFu) >> 7);
}

// This lane's view of the tables.
struct LaneTables {
    uint32_t lane4;       // 4 * lane
    int rounds;           // 0: no fast answer, exact_row
    int k;                // true codebook size
    // row address of the entry in byte `i` of w
    __device__ __forceinline__ uint32_t row_of_byte(uint32_t w, int i) const { return __byte_perm(w, lane4, 0x6504u | (i << 4)); }
    __device__ __forceinline__ uint32_t row_of_entry(uint32_t e) const { return row_of_byte(e, 0); }
    __device__ __forceinline__ float value(uint32_t row) const {
        float f;
        asm("ld.shared.f32 %0, [%1 + %2];" : "=f"(f) : "r"(row), "n"(kRowsAt + 128));
        return f;
    }
    __device__ __forceinline__ float threshold(uint32_t row) const {
        float f;
        asm("ld.shared.f32 %0, [%1 + %2];" : "=f"(f) : "r"(row), "n"(kRowsAt));
        return f;
    }
    // y = cell_position(x): the row of the count of thresholds in lower cells (the exponent bits of y come off in
    // the load's offset)
    __device__ __forceinline__ uint32_t cell_row(float y) const {
        const uint32_t bits = __float_as_uint(y);
        const uint32_t at = ((bits & 0x7F80u) | lane4) + (bits >> 15);
        uint32_t below;
        asm("ld.shared.u8 %0, [%1 + %2];" : "=r"(below) : "r"(at), "n"(kCellsAt - (0x4B000000 >> 15)));
        return row_of_byte(below, 0);
    }
    __device__ __forceinline__ uint32_t refine(float x, uint32_t row) const { return row + (x > threshold(row) ? kRowBytes : 0u); }
    // entry_exact (any codebook, NaN and values above the last entry included), reading this lane's copies
    __device__ __forceinline__ uint32_t exact_row(float x) const {
        const uint32_t last = row_of_entry(k - 1);
        if (x > value(last)) {
            const uint32_t left = k >= 2 ? last - kRowBytes : last;
            return fabsf(x - value(left)) <= fabsf(x - value(last)) ? left : last;
        }
        uint32_t row = lane4;
#pragma unroll
        for (uint32_t step = 128; step > 0; step >>= 1) {
            if (threshold(row + (step - 1) * kRowBytes) < x) row += step * kRowBytes;
        }
        return row;
    }
};

// Fills rows and cells from the staged codebook and thresholds; every thread of the CTA. `scratch`: kTableScratch bytes
// of shared memory that are free until the next __syncthreads after the call.
constexpr int kTableScratch = kCells + 16;
__device__ __forceinline__ LaneTables build_lane_tables(const SmemView& s, unsigned char* scratch) {
    unsigned char* below = scratch;
    int* most = reinterpret_cast<int*>(scratch + kCells);
    if (threadIdx.x == 0) *most = 1;
    __syncthreads();
    for (int i = threadIdx.x; i < kMaxCodebook; i += blockDim.x) {
        const int c = threshold_cell(s.thr[i]);
        const int before = i == 0 ? -1 : threshold_cell(s.thr[i - 1]);
        for (int cell = before + 1; cell <= c && cell < kCells; ++cell) below[cell] = static_cast<unsigned char>(i);
        if (c >= 0 && c < kCells) {
            int run = 1;
            while (run <= kMaxRounds && i + run < kMaxCodebook && threshold_cell(s.thr[i + run]) == c) ++run;
            if (run > 1) atomicMax(most, run);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSmemRows / 16; i += blockDim.x) {
        const float v = (i & 8) ? s.cb[i >> 4] : s.thr[i >> 4];
        reinterpret_cast<float4*>(fast_smem(kRowsAt))[i] = make_float4(v, v, v, v);
    }
    for (int i = threadIdx.x; i < kSmemCells / 16; i += blockDim.x) {
        const int r = i >> 3;
        const uint32_t w = below[r] | (below[256 + r] << 8) | (below[512 + r] << 16) | (static_cast<uint32_t>(below[768 + r]) << 24);
        reinterpret_cast<uint4*>(fast_smem(kCellsAt))[i] = make_uint4(w, w, w, w);
    }
    LaneTables t;
    t.lane4 = (threadIdx.x & 31u) * 4u;
    t.k = s.k;
    t.rounds = __shfl_sync(0xffffffffu, (*most > kMaxRounds || s.cb[s.k - 1] < 1.0f) ? 0 : *most, 0);
    __syncthreads();
    asm volatile("" : "+r"(t.lane4)::"memory");   // every read of the tables depends on lane4: none before this point
    return t;
}

// The same two-operation form for the last element of an odd chunk: the second half is not used.
template <int V> __device__ __forceinline__ f32x2 pair_at(const float (&f)[V], int i) { return pair(f[i], f[i + 1 < V ? i + 1 : i]); }
template <int V> __device__ __forceinline__ void unpair_at(f32x2 v, float (&f)[V], int i) {
    float spare;
    if (i + 1 < V) unpair(v, f[i], f[i + 1]); else unpair(v, f[i], spare);
}

// Row addresses of the entries of a chunk of momenta (quotients m / absmax through the block's reciprocal, see
// div_by_block_constant). ONE: t.rounds == 1, the usual codebook.
template <int V, bool ONE>
__device__ __forceinline__ void encode(const float (&m)[V], f32x2 neg_absmax2, f32x2 rinv2, const LaneTables& t,
                                       uint32_t (&row)[V]) {
    float x[V];
#pragma unroll
    for (int i = 0; i < V; i += 2) {
        const f32x2 m2 = pair_at(m, i);
        const f32x2 q0 = mul2(m2, rinv2);
        unpair_at(fma2(fma2(q0, neg_absmax2, m2), rinv2, q0), x, i);
    }
#pragma unroll
    for (int i = 0; i < V; ++i) row[i] = t.cell_row(cell_position(x[i]));
#pragma unroll
    for (int i = 0; i < V; ++i) row[i] = t.refine(x[i], row[i]);
    if constexpr (!ONE) {
        if (t.rounds == 0) {
#pragma unroll
            for (int i = 0; i < V; ++i) row[i] = t.exact_row(x[i]);
        } else {
            for (int r = 1; r < t.rounds; ++r) {
#pragma unroll
                for (int i = 0; i < V; ++i) row[i] = t.refine(x[i], row[i]);
            }
        }
    }
}
// The code bytes of a chunk's row addresses.
template <int V> __device__ __forceinline__ CodeChunk<V> row_codes(const uint32_t (&row)[V]) {
    CodeChunk<V> c;
    if constexpr (V >= 4) {
#pragma unroll
        for (int i = 0; i < V; i += 4)
            c.w[i / 4] = __byte_perm(__byte_perm(row[i], row[i + 1], 0x0051), __byte_perm(row[i + 2], row[i + 3], 0x0051), 0x5410);
    } else if constexpr (V == 2) c.w[0] = __byte_perm(row[0], row[1], 0x0051);
    else c.w[0] = row[0] >> 8;
    return c;
}

// Lanes that share one block, a power of two, so that a warp works on 32 / lanes blocks at once. A lane takes
// several chunks of its block, which keeps as many loads in flight and shares the per-block work (reductions,
// step size, reciprocal) between more elements: about eight chunks of eight elements per lane for blocks of more
// than 256 elements, as in a 2048-element block (8 lanes for 512 elements, 16 for 1024, all 32 from 1032 on), up to
// four down to blocks of 72 elements, two below that (the blocks of a warp lie side by side in its buffer, so lanes with
// four chunks of their own would read the same banks: 134 M bf16 elements in blocks of 64 / 32 0.60 / 0.58 ms with four,
// 0.342 / 0.336 with two; before the buffers 0.350 / 0.351). Averaged gradients differ, see deep_lanes.
__host__ __device__ __forceinline__ int lanes_shift(long long nchunks, int v) {   // log2 of the lanes; chunks of v elements
    if (v < 8) {   // smaller chunks: about sixteen per lane, eight of them in flight
        int shift = 0;
        while (shift < 5 && (16 << shift) < nchunks) ++shift;
        return shift;
    }
    const long long want = nchunks > 32 ? (nchunks + 7) >> 3 : (nchunks <= 8 ? (nchunks + 1) >> 1 : (nchunks + 3) >> 2);
    int shift = 0;
    while (shift < 5 && (1 << shift) < want) ++shift;
    return shift;
}
// Averaged gradients of two-byte types in blocks of 24, 40, 48 and 64 elements: half as many lanes with up to four chunks
// each where the sources are few. The staged slices have no conflicts (slice_stride), and a lane's loads are what is in
// flight; many sources read better with more lanes on one line. 67 M bf16 elements, ms, two / four chunks per lane: two
// sources, blocks of 24 0.339 / 0.271, 40 0.406 / 0.280, 48 0.346 / 0.244, 64 0.263 / 0.232 (32 0.264 / 0.336, 56 0.304 / 0.357);
// three, blocks of 24 0.363 / 0.380, 40 0.433 / 0.329, 48 0.380 / 0.310; four, 40 0.406 / 0.372, 48 0.359 / 0.364; eight, 64
// 0.469 / 0.747. The second moments stay a single process's: each half of a lane's chunks has a sum of its own, and they
// are added as the first step over twice the lanes adds them. (Kernels of their own, GSRC == 3: the second sum cost those
// of eight sources 6 to 9 %, those of four up to 3 %.)
// `sources`: buffers that a chunk is read from (1: the switch's sum), 0 = this GPU's gradients.
constexpr int kFewSources = 3;
__host__ __device__ __forceinline__ bool deep_lanes(long long nchunks, int v, int es, int sources) {
    if (v != 8 || es != 2 || sources < 1) return false;
    return ((nchunks == 5 || nchunks == 6) && sources <= kFewSources) || ((nchunks == 3 || nchunks == 8) && sources <= 2);
}
__host__ __device__ __forceinline__ int lanes_shift(long long nchunks, int v, int es, int sources) {
    return lanes_shift(nchunks, v) - (deep_lanes(nchunks, v, es, sources) ? 1 : 0);
}
// Elements of one work unit of a tensor (what a warp works on at a time), blocks of nchunks chunks of v elements.
__host__ __device__ __forceinline__ long long unit_elements(long long period, int v) { return period << (5 - lanes_shift(period / v, v)); }
// Floats from one block's staged momenta to the next one's in a warp's slice. Eight lanes make one 128-byte access;
// where they belong to several blocks (fewer than eight lanes per block), the blocks' slices start on different banks.
__host__ __device__ __forceinline__ int slice_stride(int period, int shift, int v) {
    return v < 8 || shift >= 3 ? period : ((period + 31) & ~31) + (4 << shift);
}
// Floats that a warp stages for one unit.
__host__ __device__ __forceinline__ long long unit_floats(long long period, int v, int es, int sources) {
    const int shift = lanes_shift(period / v, v, es, sources);
    return static_cast<long long>(slice_stride(static_cast<int>(period), shift, v)) << (5 - shift);
}
// Work units (one warp pass each) of a tensor on the fast path.
__host__ __device__ __forceinline__ long long vec_units(long long num_blocks, long long period, int v, int es, int sources) {
    const int shift = 5 - lanes_shift(period / v, v, es, sources);
    return (num_blocks + (1 << shift) - 1) >> shift;
}

// Reductions over aligned groups of `lanes` lanes (a power of two); every lane of the warp calls them.
__device__ __forceinline__ float group_max_nan(float v, int lanes) {
    for (int o = lanes >> 1; o > 0; o >>= 1) {
        const float other = __shfl_xor_sync(0xffffffffu, v, o);
        asm("max.NaN.f32 %0, %1, %2;" : "=f"(v) : "f"(v), "f"(other));
    }
    return v;
}
__device__ __forceinline__ float group_max(float v, int lanes) {
    for (int o = lanes >> 1; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float group_sum(float v, int lanes) {
    for (int o = lanes >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// What the passes need of a tensor, in a shared-memory slot of the warp: its descriptor lives in global memory, where
// the passes' stores might alias it as far as the compiler can tell, and is read again only when the warp comes to
// another tensor. (In registers it would cost some 25 of them for values that are used once per block.)
template <typename S> struct alignas(8) TensorSlot {
    const S* g;
    S* p;
    uint8_t* codes;
    void* mag;
    void* v;
    long long first, units, num_blocks;   // in the launch's work units; blocks
    int period, mag_dtype, v_dtype;
    uint32_t flags;
    float beta1, beta2, inv_bc1, bc2, eps, lr, wd_mul;
    __device__ __forceinline__ void load(const gefen_b200_step_tensor_t* t, int v_elems, int sources) {
        g = static_cast<const S*>(t->g);
        p = static_cast<S*>(t->p);
        codes = t->codes;
        mag = t->mag;
        v = t->v;
        first = t->first_block;
        num_blocks = t->num_blocks;
        period = static_cast<int>(t->period);   // at most kFastMaxPeriod
        flags = t->flags;
        units = vec_units(num_blocks, period, v_elems, sizeof(S), sources);
        mag_dtype = t->mag_dtype;
        v_dtype = t->v_dtype;
        beta1 = t->beta1;
        beta2 = t->beta2;
        inv_bc1 = 1.0f / t->bc1;
        bc2 = t->bc2;
        eps = t->eps;
        lr = t->lr;
        wd_mul = t->wd_mul;
    }
};

// The sum of squares of a lane's other chunks (see deep_lanes): the two change places after every chunk.
struct OtherHalf {
    bool used;
    f32x2 sum;
    __device__ __forceinline__ void turn(f32x2& mine) {
        const f32x2 was = mine;
        mine = used ? sum : was;
        sum = used ? was : sum;
    }
};

// First pass over U chunks of one lane (chunks c0, c0 + LANES, ...): all loads first, then the
// moment update, the running absmax and sum of squares, and the staging of the updated momenta.
// SUMMED: g_blk is the multicast address of the block's gradients; a load returns the sum over the ranks,
// which is scaled by `scale` and rounded to the gradient dtype as a reduce-scatter into it would leave it.
template <typename S, int V, int U, bool GUARD, bool SUMMED, bool STAGED = true>
__device__ __forceinline__ void first_pass_group(const S* g_blk, const uint8_t* codes_in, float* stage, int half,
                                                 const LaneTables& t, int c0, int LANES, int nchunks, f32x2 mag2,
                                                 f32x2 beta2_, f32x2 omb2_, float scale, float& absmax, f32x2& sumsq2, OtherHalf& other) {
    CodeChunk<V> craw[U];
    Chunk<S, V> graw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int c = c0 + LANES * u;
        if (!GUARD || c < nchunks) {
            if constexpr (STAGED) craw[u].load(codes_in, c);
            else craw[u].load_again_later(codes_in, c);
            if (SUMMED) graw[u].load_sum(g_blk, c);
            else if constexpr (STAGED) graw[u].load(g_blk, c);
            else graw[u].load_again_later(g_blk, c);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int c = c0 + LANES * u;
        if (!GUARD || c < nchunks) {
            float g[V], m[V];
            graw[u].unpack(g);
            if (SUMMED) {
#pragma unroll
                for (int i = 0; i < V; ++i) g[i] *= scale;
                Chunk<S, V> rounded;
                rounded.pack(g);
                rounded.unpack(g);
            }
            if constexpr (V == 1) {
                const float cur = t.value(t.row_of_byte(craw[u].w[0], 0));
                float lo, spare;
                unpair(fma2(beta2_, mul2(mag2, pair(cur, cur)), mul2(omb2_, pair(g[0], g[0]))), lo, spare);
                m[0] = lo;
                absmax = max_abs_nan(absmax, lo);
                sumsq2 = fma2(pair(g[0], 0.0f), pair(g[0], 0.0f), sumsq2);
            } else {
#pragma unroll
                for (int i = 0; i < V; i += 2) {
                    const f32x2 g2 = pair(g[i], g[i + 1]);
                    const f32x2 cur = mul2(mag2, pair(t.value(t.row_of_byte(craw[u].w[i >> 2], i & 3)),
                                                      t.value(t.row_of_byte(craw[u].w[i >> 2], (i & 3) + 1))));
                    unpair(fma2(beta2_, cur, mul2(omb2_, g2)), m[i], m[i + 1]);   // ema_update
                    absmax = max_abs_nan(max_abs_nan(absmax, m[i]), m[i + 1]);
                    sumsq2 = fma2(g2, g2, sumsq2);
                }
            }
            if (SUMMED) other.turn(sumsq2);
            if (STAGED) stage_store<V>(stage, half, c, m);
        }
    }
}

// The same over U chunks of a unit whose inputs a bulk copy has brought to shared memory (g_at, codes_at: the lane's
// block); the updated momenta go to tensor memory, V columns per round. The whole warp calls it.
template <typename S, int V, int U, bool GUARD>
__device__ __forceinline__ void first_pass_ring(uint32_t g_at, uint32_t codes_at, uint32_t hold, const LaneTables& t, int c0, int LANES,
                                                int nchunks, f32x2 mag2, f32x2 beta2_, f32x2 omb2_, float& absmax, f32x2& sumsq2) {
    CodeChunk<V> craw[U];
    Chunk<S, V> graw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int c = c0 + LANES * u;
        if (!GUARD || c < nchunks) {
            craw[u].load_shared(codes_at + c * V);
            graw[u].load_shared(g_at + c * Chunk<S, V>::kBytes);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        float m[V];
#pragma unroll
        for (int i = 0; i < V; ++i) m[i] = 0.0f;
        if (!GUARD || c0 + LANES * u < nchunks) {
            float g[V];
            graw[u].unpack(g);
            if constexpr (V == 1) {
                const float cur = t.value(t.row_of_byte(craw[u].w[0], 0));
                float spare;
                unpair(fma2(beta2_, mul2(mag2, pair(cur, cur)), mul2(omb2_, pair(g[0], g[0]))), m[0], spare);
                absmax = max_abs_nan(absmax, m[0]);
                sumsq2 = fma2(pair(g[0], 0.0f), pair(g[0], 0.0f), sumsq2);
            } else {
#pragma unroll
                for (int i = 0; i < V; i += 2) {
                    const f32x2 g2 = pair(g[i], g[i + 1]);
                    const f32x2 cur = mul2(mag2, pair(t.value(t.row_of_byte(craw[u].w[i >> 2], i & 3)),
                                                      t.value(t.row_of_byte(craw[u].w[i >> 2], (i & 3) + 1))));
                    unpair(fma2(beta2_, cur, mul2(omb2_, g2)), m[i], m[i + 1]);   // ema_update
                    absmax = max_abs_nan(max_abs_nan(absmax, m[i]), m[i + 1]);
                    sumsq2 = fma2(g2, g2, sumsq2);
                }
            }
        }
        if (GUARD) __syncwarp();
        hold_store<V>(hold + u * V, m);
    }
}

// First pass of a block whose gradient is averaged over up to NSRC buffers. kSlots 16-byte (fp32:
// 32-byte) loads per lane are in flight at a time: U chunks x a batch of BS sources; the sources of
// a chunk are added batch after batch, in the order given.
// EXACT: there are exactly NSRC sources (no test per source). TURNS: the blocks may be those of deep_lanes.
template <typename S, bool TURNS, int NSRC, bool EXACT = false>
__device__ __forceinline__ void reduce_pass(const StepLaunch& L, const S* g_blk, const uint8_t* codes_in, float* stage, int half,
                                            const LaneTables& t, int lane, int LANES, int nchunks,
                                            float old_mag, float beta1, float omb1, float& absmax, f32x2& sumsq2, OtherHalf& other) {
    constexpr int kSlots = sizeof(S) == 2 ? 4 : 2;
    constexpr int BS = NSRC < kSlots ? NSRC : kSlots;
    constexpr int U = kSlots / BS;
    const int n_src = EXACT ? NSRC : L.n_grad_srcs;
    const float scale = L.grad_scale;
    for (int c0 = lane; c0 < nchunks; c0 += LANES * U) {
        float acc[U][8];
        CodeChunk<8> craw[U];   // the codes travel with the first batch of gradient loads
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[u][i] = 0.0f;
            if (c0 + LANES * u < nchunks) craw[u].load(codes_in, c0 + LANES * u);
        }
#pragma unroll
        for (int r0 = 0; r0 < NSRC; r0 += BS) {
            if (r0 < n_src) {
                Chunk<S, 8> src[U * BS];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int c = c0 + LANES * u;
#pragma unroll
                    for (int r = 0; r < BS; ++r)
                        if (c < nchunks && r0 + r < n_src) src[u * BS + r].load(peer_ptr(g_blk, L.grad_delta[r0 + r]), c);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int c = c0 + LANES * u;
#pragma unroll
                    for (int r = 0; r < BS; ++r) {
                        if (c < nchunks && r0 + r < n_src) {
                            float part[8];
                            src[u * BS + r].unpack(part);
#pragma unroll
                            for (int i = 0; i < 8; ++i) acc[u][i] += part[i];
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + LANES * u;
            if (c < nchunks) {
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[u][i] *= scale;
                Chunk<S, 8> rounded;
                rounded.pack(acc[u]);
                float g[8], m[8];
                rounded.unpack(g);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float cur = old_mag * t.value(t.row_of_byte(craw[u].w[i >> 2], i & 3));
                    m[i] = ema_update(beta1, cur, omb1, g[i]);
                    absmax = max_abs_nan(absmax, m[i]);
                }
#pragma unroll
                for (int i = 0; i < 8; i += 2) sumsq2 = fma2(pair(g[i], g[i + 1]), pair(g[i], g[i + 1]), sumsq2);   // as first_pass_group
                if constexpr (TURNS) other.turn(sumsq2);
                stage_store<8>(stage, half, c, m);
            }
        }
    }
}

// The same in chunks of V < 8 elements, for any number of sources (none: this GPU's buffer). Four chunks per lane are in
// flight for one source at a time; the sums are formed in the order of first_pass_group.
template <typename S, int V>
__device__ __forceinline__ void reduce_pass_small(const StepLaunch& L, const S* g_blk, const uint8_t* codes_in, float* stage, int half,
                                                  const LaneTables& t, int lane, int LANES, int nchunks, float old_mag, float beta1,
                                                  float omb1, float& absmax, f32x2& sumsq2) {
    constexpr int U = 4;
    const int n_src = L.n_grad_srcs;
    for (int c0 = lane; c0 < nchunks; c0 += LANES * U) {
        CodeChunk<V> craw[U];
        Chunk<S, V> graw[U];
        float acc[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int i = 0; i < V; ++i) acc[u][i] = 0.0f;
            if (c0 + LANES * u < nchunks) {
                craw[u].load(codes_in, c0 + LANES * u);
                if (n_src == 0) graw[u].load(g_blk, c0 + LANES * u);
            }
        }
        for (int r = 0; r < n_src; ++r) {
            const S* const src = peer_ptr(g_blk, L.grad_delta[r]);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (c0 + LANES * u < nchunks) graw[u].load(src, c0 + LANES * u);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (c0 + LANES * u < nchunks) {
                    float part[V];
                    graw[u].unpack(part);
#pragma unroll
                    for (int i = 0; i < V; ++i) acc[u][i] += part[i];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + LANES * u;
            if (c < nchunks) {
                if (n_src > 0) {
#pragma unroll
                    for (int i = 0; i < V; ++i) acc[u][i] *= L.grad_scale;
                    graw[u].pack(acc[u]);
                }
                float g[V], m[V];
                graw[u].unpack(g);
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const float cur = old_mag * t.value(t.row_of_byte(craw[u].w[0], i));
                    m[i] = ema_update(beta1, cur, omb1, g[i]);
                    absmax = max_abs_nan(absmax, m[i]);
                }
#pragma unroll
                for (int i = 0; i < V; i += 2) {
                    const f32x2 g2 = V == 1 ? pair(g[0], 0.0f) : pair_at(g, i);
                    sumsq2 = fma2(g2, g2, sumsq2);
                }
                stage_store<V>(stage, half, c, m);
            }
        }
    }
}

// Where the second pass takes a chunk's updated momenta from:
//   kShared  the warp's slice of shared memory (gradients of several ranks, what route() and launch_ring leave);
//   kTwice   computed once more from codes and gradients, which L2 still holds (blocks too long for the other two, see
//            route); the next chunk's are requested while this one is worked on;
//   kTensor  the warp's columns of tensor memory (step_ring_kernel).
// All walk the chunks of a lane in order; the whole warp calls take() (round `it`, chunk c of the lane; ALL: every lane
// has one).
enum Hold { kShared, kTwice, kTensor };
template <typename S, int V, int HOLD> struct Momenta {   // kShared
    const float* const stage;
    const int half;
    __device__ __forceinline__ Momenta(const float* s, int h, uint32_t, const uint8_t*, const S*, const LaneTables&, float, float, float)
        : stage(s), half(h) {}
    __device__ __forceinline__ void start(int, int, int) {}
    template <bool ALL> __device__ __forceinline__ void take(int, int c, int, int nchunks, float (&m)[V]) {
        if (ALL || c < nchunks) stage_load<V>(stage, half, c, m);
    }
};
template <typename S, int V> struct Momenta<S, V, kTensor> {
    const uint32_t hold;
    __device__ __forceinline__ Momenta(const float*, int, uint32_t h, const uint8_t*, const S*, const LaneTables&, float, float, float)
        : hold(h) {}
    __device__ __forceinline__ void start(int, int, int) {}
    // (The work on the chunk before branches by lane: requests of the last rounds, the search of exact_row. tcgen05.ld
    // wants the whole warp together.)
    template <bool ALL> __device__ __forceinline__ void take(int it, int, int, int, float (&m)[V]) {
        __syncwarp();
        hold_load<V>(hold + it * V, m);
    }
};
template <typename S, int V> struct Momenta<S, V, kTwice> {
    const uint8_t* const codes;
    const S* const g;
    const LaneTables& t;
    const f32x2 mag2, beta2_, omb2_;
    CodeChunk<V> craw;
    Chunk<S, V> graw;
    __device__ __forceinline__ Momenta(const float*, int, uint32_t, const uint8_t* c, const S* gradients, const LaneTables& tables,
                                       float old_mag, float beta1, float omb1)
        : codes(c), g(gradients), t(tables), mag2(pair(old_mag, old_mag)), beta2_(pair(beta1, beta1)), omb2_(pair(omb1, omb1)) {}
    __device__ __forceinline__ void start(int lane, int, int nchunks) {
        if (lane < nchunks) { craw.load(codes, lane); graw.load(g, lane); }
    }
    template <bool ALL> __device__ __forceinline__ void take(int, int c, int LANES, int nchunks, float (&m)[V]) {
        if (!ALL && c >= nchunks) return;
        const CodeChunk<V> code = craw;
        float gv[V];
        graw.unpack(gv);
        if (c + LANES < nchunks) { craw.load(codes, c + LANES); graw.load(g, c + LANES); }
#pragma unroll
        for (int i = 0; i < V; i += 2) {
            const f32x2 cur = mul2(mag2, pair(t.value(t.row_of_byte(code.w[i >> 2], i & 3)), t.value(t.row_of_byte(code.w[i >> 2], (i & 3) + 1))));
            unpair(fma2(beta2_, cur, mul2(omb2_, pair(gv[i], gv[i + 1]))), m[i], m[i + 1]);   // as first_pass_group
        }
    }
};

// One chunk of the re-encode and update of the common case (finite block, Gefen update of the parameters) with
// everything that is fixed per launch or per tensor decided at compile time: WD = the decoupled weight decay of the
// reference's separate multiply, STORE = 0 this GPU's copy only, 1 peer stores as well, 2 one multicast store, ONE =
// see encode.
struct BlockScalars {
    f32x2 neg_absmax2, rinv2, step2, lr2, wd2;
};
template <typename S, int V, bool WD, int STORE, bool ONE>
__device__ __forceinline__ void update_chunk(const StepLaunch& L, const LaneTables& t, const float (&m)[V], uint8_t* codes, S* p_blk,
                                             Chunk<S, V> praw, int c, const BlockScalars& b) {
    uint32_t row[V];
    encode<V, ONE>(m, b.neg_absmax2, b.rinv2, t, row);
    row_codes<V>(row).store(codes, c);
    float pv[V];
    praw.unpack(pv);
    if (WD) {
#pragma unroll
        for (int i = 0; i < V; i += 2) unpair_at(mul2(pair_at(pv, i), b.wd2), pv, i);
        Chunk<S, V> rounded;       // the separate multiply of the reference rounds to the parameter dtype
        rounded.pack(pv);
        rounded.unpack(pv);
    }
#pragma unroll
    for (int i = 0; i < V; i += 2) {
        const f32x2 neg_q = mul2(pair(t.value(row[i]), t.value(row[i + 1 < V ? i + 1 : i])), b.neg_absmax2);
        unpair_at(fma2(mul2(neg_q, b.step2), b.lr2, pair_at(pv, i)), pv, i);   // fma(-(q * step), lr, p)
    }
    praw.pack(pv);
    if (STORE == 2) {
        praw.store_all(peer_ptr(p_blk, L.param_mc_delta), c);   // every rank's copy, this one included
    } else {
        praw.store(p_blk, c);
        if (STORE == 1) {
            const int n_peers = L.n_peers;
            for (int r = 0; r < n_peers; ++r) praw.store(peer_ptr(p_blk, L.peer_delta[r]), c);
        }
    }
}
// Parameters (GefenMuon: gradients) of a lane's chunks that are requested ahead of the re-encoding: the next chunk of
// eight elements (two in the ring kernel, which has the registers for them: 134 M bf16 elements in blocks of 1120 0.322 ->
// 0.227 ms, of 2048 0.208 -> 0.197), the next four to eight of the smaller chunks, whose work is too short to cover the
// latency of a load.
template <typename S, int V, int HOLD> struct Ahead {
    static constexpr int kDepth = V < 8 ? (V * sizeof(S) > 8 || (V == 4 && HOLD == kTensor) ? 4 : 8) : (HOLD == kTensor ? 2 : 1);
    Chunk<S, V> slot[kDepth];
    __device__ __forceinline__ void start(const S* blk, int lane, int LANES, int nchunks) {
#pragma unroll
        for (int u = 0; u < kDepth; ++u)
            if (lane + u * LANES < nchunks) slot[u].load(blk, lane + u * LANES);
    }
    // hands out slot u (chunk c) and requests the chunk that comes to it next
    __device__ __forceinline__ Chunk<S, V> take(int u, const S* blk, int c, int LANES, int nchunks) {
        const Chunk<S, V> now = slot[u];
        if (c + kDepth * LANES < nchunks) slot[u].load(blk, c + kDepth * LANES);
        return now;
    }
};
// The chunks of one block: `full` rounds in which every lane of the warp has one, then the guarded rest. The
// parameters of the next chunks are fetched while this one is encoded.
template <typename S, int V, int HOLD, bool WD, int STORE, bool ONE>
__device__ __forceinline__ void second_pass_common(const StepLaunch& L, const LaneTables& t, Momenta<S, V, HOLD>& momenta, uint8_t* codes, S* p_blk,
                                                   Ahead<S, V, HOLD>& ahead, int lane, int LANES, int nchunks, int full, int rounds_all,
                                                   const BlockScalars& b) {
    constexpr int D = Ahead<S, V, HOLD>::kDepth;
    int c = lane;
    int it = 0;
    if constexpr (V == 8) {
        for (; it + D <= full; it += D) {
#pragma unroll
            for (int u = 0; u < D; ++u, c += LANES) {
                float m[V];
                momenta.template take<true>(it + u, c, LANES, nchunks, m);
                const Chunk<S, V> praw = ahead.take(u, p_blk, c, LANES, nchunks);
                update_chunk<S, V, WD, STORE, ONE>(L, t, m, codes, p_blk, praw, c, b);
            }
        }
    }
    for (; it < rounds_all; it += D) {
#pragma unroll
        for (int u = 0; u < D; ++u, c += LANES) {
            if (it + u < rounds_all) {
                float m[V];
                momenta.template take<false>(it + u, c, LANES, nchunks, m);
                if (c < nchunks) {
                    const Chunk<S, V> praw = ahead.take(u, p_blk, c, LANES, nchunks);
                    update_chunk<S, V, WD, STORE, ONE>(L, t, m, codes, p_blk, praw, c, b);
                }
            }
        }
    }
}

// The same loop for GefenMuon's momentum step (finite block): the dequantised new momentum, Nesterov-blended
// with the gradient when asked (torch: m.mul_(momentum).add_(g, alpha=1-momentum) on the rounded momentum,
// reference gefen_muon.py:312-314; alpha travels in the descriptor's beta2), goes where the Gefen step keeps
// the parameters. The gradient chunk of the next iteration is requested while this one is encoded.
template <typename S, int V, int HOLD, bool NESTEROV, bool ONE>
__device__ __forceinline__ void second_pass_muon(const LaneTables& t, Momenta<S, V, HOLD>& momenta, uint8_t* codes, const S* g_blk, S* out_blk,
                                                 int lane, int LANES, int nchunks, int rounds_all, float absmax, f32x2 neg_absmax2, f32x2 rinv2,
                                                 float beta1, float alpha) {
    constexpr int D = Ahead<S, V, HOLD>::kDepth;
    Ahead<S, V, HOLD> ahead;
    if (NESTEROV) ahead.start(g_blk, lane, LANES, nchunks);
    int c = lane;
    for (int it = 0; it < rounds_all; it += D) {
#pragma unroll
        for (int u = 0; u < D; ++u, c += LANES) {
            if (it + u >= rounds_all) break;
            float m[V];
            momenta.template take<false>(it + u, c, LANES, nchunks, m);
            if (c >= nchunks) continue;
            Chunk<S, V> graw;
            if (NESTEROV) graw = ahead.take(u, g_blk, c, LANES, nchunks);
            uint32_t row[V];
            encode<V, ONE>(m, neg_absmax2, rinv2, t, row);
            row_codes<V>(row).store(codes, c);
            float q[V];
#pragma unroll
            for (int i = 0; i < V; ++i) q[i] = t.value(row[i]) * absmax;
            Chunk<S, V> out;
            if (NESTEROV) {
                float g[V];
                graw.unpack(g);
                out.pack(q);
                out.unpack(q);
#pragma unroll
                for (int i = 0; i < V; ++i) q[i] *= beta1;
                out.pack(q);
                out.unpack(q);
#pragma unroll
                for (int i = 0; i < V; ++i) q[i] = fmaf(alpha, g[i], q[i]);
            }
            out.pack(q);
            out.store(out_blk, c);
        }
    }
}

// One warp, one unit: 32 / LANES consecutive blocks of t.period = V * chunks elements, LANES lanes
// each (a power of two, uniform over the warp; FULL fixes it to 32 at compile
// time, for blocks of more than 1024 elements). A block's slice of `stage` holds period floats (see stage_store).
// GSRC: where the gradients come from: 0 = this GPU's buffer, 1 = averaged over the ranks' buffers with peer
// loads, 2 = summed by the switch through the multicast mapping (StepLaunch::grad_mc_delta), 3 = as 1, over at most
// kFewSources buffers and with the lanes of deep_lanes (blocks that share a warp, two-byte types). Chunks below eight elements
// know 0 and 1 only: 1 is every launch with peers, gradients of this GPU's buffer (no sources) included.
// In: how the unit's inputs arrive (RingInputs; DirectInputs: they are loaded here). False: a bounded wait for the inputs
// ran out and nothing was done.
template <typename S, int V, int GSRC, bool FULL, int HOLD, typename In>
__device__ __forceinline__ bool warp_block_step(const TensorSlot<S>& t, long long unit, const StepLaunch& L, const LaneTables& tables,
                                                float* stage, In& in, int warp_lane) {
    constexpr bool STAGED = HOLD == kShared;
    const float* const stepsize = L.stepsize;
    const int n_peers = GSRC == 0 && V < 8 ? 0 : L.n_peers;            // (chunks below 8: GSRC == 1 wherever there are peers)
    const long long param_mc = V < 8 ? 0 : L.param_mc_delta;           // (a multicast access moves 16 bytes)
    // (the shuffle tells the compiler that the period is the same in all lanes, which the loops' bounds profit from)
    const int period = __shfl_sync(0xffffffffu, t.period, 0);
    const int chunks = period / V;                     // of a block
    constexpr bool kMayBeDeep = (GSRC == 2 || GSRC == 3) && !FULL && sizeof(S) == 2;
    const int shift = FULL ? 5 : (kMayBeDeep ? lanes_shift(chunks, V, sizeof(S), chunk_sources(L)) : lanes_shift(chunks, V));
    const int LANES = 1 << shift;
    const int lane = warp_lane & (LANES - 1);          // lane within the block's group
    const int member = warp_lane >> shift;             // which block of the unit
    const long long b = (unit << (5 - shift)) + member;
    const bool all_valid = FULL || ((unit + 1) << (5 - shift)) <= t.num_blocks;   // the last unit of a tensor may be short
    const bool valid = FULL || b < t.num_blocks;
    const int nchunks = valid ? chunks : 0;
    stage += member * slice_stride(period, shift, V);
    const int half = period >> 1;
    const long long elem0 = b * static_cast<long long>(period);
    uint8_t* const codes = t.codes + elem0;
    const S* const g_blk = t.g + elem0;   // chunk c of the block = V elements at g_blk + V c
    S* const p_blk = t.p + elem0;
    const uint32_t flags = t.flags;
    const bool muon = (flags & GEFEN_B200_STEP_MUON) != 0;

    const float beta1 = t.beta1;
    const float omb1 = 1.0f - beta1;
    float old_mag = 0.0f;
    if constexpr (HOLD == kTensor) old_mag = in.mag;
    else if (valid) old_mag = load_state(t.mag, b, t.mag_dtype);

    // Everything the block needs from HBM besides codes and gradients is requested now, so that its
    // latency overlaps the first pass: the second moment (the ring kernel has it already) and, where the registers
    // allow it (2-byte types, ring kernel), the first chunks of parameters.
    constexpr bool kEarlyParams = sizeof(S) == 2 || HOLD == kTensor;
    const float lr = t.lr;
    const bool do_update = muon || lr != 0.0f;
    const bool load_p = !muon && do_update;
    float v_in = 1.0f;
    if constexpr (HOLD == kTensor) v_in = in.v;
    else if (!muon && valid) v_in = stepsize != nullptr ? stepsize[b] : load_state(t.v, b, t.v_dtype);
    Ahead<S, V, HOLD> ahead;
    if (kEarlyParams && load_p) ahead.start(p_blk, lane, LANES, nchunks);

    const int rounds_all = (chunks + LANES - 1) >> shift, full = all_valid ? chunks >> shift : 0;
    // ---- pass over codes and gradients (the only read of both)
    float absmax = 0.0f;
    float sumsq = 0.0f;
    f32x2 sumsq2 = pair(0.0f, 0.0f);
    OtherHalf other = {kMayBeDeep && deep_lanes(chunks, V, sizeof(S), chunk_sources(L)), pair(0.0f, 0.0f)};
    if (GSRC == 1 || GSRC == 3) {
        // The gradient of this block is the average over the ranks' buffers (this GPU's and the
        // peers', read over NVLink), summed in fp32 in rank order and rounded to the gradient dtype,
        // as a reduce-scatter into that dtype would leave it.
        if constexpr (GSRC == 1 && V < 8) {
            reduce_pass_small<S, V>(L, g_blk, codes, stage, half, tables, lane, LANES, nchunks, old_mag, beta1, omb1, absmax, sumsq2);
        } else if constexpr (GSRC == 1 || GSRC == 3) {
            const int n_src = L.n_grad_srcs;
#define GEFEN_REDUCE_PASS(...) reduce_pass<S, GSRC == 3, __VA_ARGS__>(L, g_blk, codes, stage, half, tables, lane, LANES, nchunks, old_mag, beta1, omb1, absmax, sumsq2, other)
            if (n_src == 2) GEFEN_REDUCE_PASS(2, true);
            else if (n_src < 2) GEFEN_REDUCE_PASS(2);
            else if (GSRC == 1 && n_src == 4) GEFEN_REDUCE_PASS(4, true);
            else if (GSRC == 3 || n_src < 4) GEFEN_REDUCE_PASS(4);
            else GEFEN_REDUCE_PASS(8);
#undef GEFEN_REDUCE_PASS
        }
    } else if constexpr (HOLD == kTensor) {
        constexpr int U = 2;
        const long long unit0 = (unit << (5 - shift)) * period;
        const uint32_t g_at = in.g_at(t.g + unit0) + static_cast<uint32_t>(member * period) * static_cast<uint32_t>(sizeof(S));
        const uint32_t codes_at = in.codes_at(t.codes + unit0) + static_cast<uint32_t>(member * period);
        const f32x2 mag2 = pair(old_mag, old_mag), beta2_ = pair(beta1, beta1), omb2_ = pair(omb1, omb1);
        if (!in.arrived(L.input_limit)) return false;
        __syncwarp();   // (the lanes leave the wait one by one, tcgen05.st wants them together)
        int it = 0;
        for (; it + U <= full; it += U)
            first_pass_ring<S, V, U, false>(g_at, codes_at, in.hold + it * V, tables, lane + it * LANES, LANES, nchunks, mag2, beta2_, omb2_,
                                            absmax, sumsq2);
        for (; it < rounds_all; ++it)
            first_pass_ring<S, V, 1, true>(g_at, codes_at, in.hold + it * V, tables, lane + it * LANES, LANES, nchunks, mag2, beta2_, omb2_,
                                           absmax, sumsq2);
        hold_stores_done();
        __syncwarp();   // the whole warp has read the buffers
        in.request_next();
    } else {
        // Up to four chunks in flight per lane; complete groups of four in every lane without bounds tests, which
        // cost four instructions each and sit on the one path that every element takes.
        constexpr int U = V < 8 ? 8 : 4;
        constexpr bool SUMMED = GSRC == 2;
        const S* const g_src = SUMMED ? peer_ptr(g_blk, L.grad_mc_delta) : g_blk;
        const float scale = SUMMED ? L.grad_scale : 1.0f;
        const f32x2 mag2 = pair(old_mag, old_mag), beta2_ = pair(beta1, beta1), omb2_ = pair(omb1, omb1);
        int c0 = 0;
        if (all_valid && sizeof(S) == 2) {   // (fp32: the second copy of the loop costs registers; measured slower)
            for (; c0 + LANES * U <= chunks; c0 += LANES * U)
                first_pass_group<S, V, U, false, SUMMED, STAGED>(g_src, codes, stage, half, tables, c0 + lane, LANES, nchunks, mag2, beta2_, omb2_,
                                                         scale, absmax, sumsq2, other);
        }
        for (; c0 < chunks; c0 += LANES * U)
            first_pass_group<S, V, U, true, SUMMED, STAGED>(g_src, codes, stage, half, tables, c0 + lane, LANES, nchunks, mag2, beta2_, omb2_,
                                                    scale, absmax, sumsq2, other);
    }
    {   // (the same partial sums wherever the gradients come from: a rank's second moments are a single process's)
        float even, odd;
        unpair(sumsq2, even, odd);
        sumsq = even + odd;
        if (other.used) {
            unpair(other.sum, even, odd);
            sumsq += even + odd;
        }
    }
    absmax = group_max_nan(absmax, LANES);

    // ---- second moment (optionally fused) and the step size
    float step = 0.0f;
    if (!muon) {
        if (stepsize != nullptr) {
            step = v_in;
        } else {
            float v = v_in;
            if (flags & GEFEN_B200_STEP_FUSE_VMEAN) {
                const float mean_sq = group_sum(sumsq, LANES) / static_cast<float>(period);
                const float nv = fmaf(t.beta2, v_in, (1.0f - t.beta2) * mean_sq);
                v = 0.0f;
                if (lane == 0 && valid) v = store_state(t.v, b, t.v_dtype, nv);
                v = __shfl_sync(0xffffffffu, v, warp_lane & ~(LANES - 1));
            }
            step = t.inv_bc1 / (sqrtf(v / t.bc2) + t.eps);   // adam_step_size
        }
    }
    __syncwarp();  // staged momenta are visible to the whole warp; every lane has read the old magnitude
    uint32_t hold = 0;
    if constexpr (HOLD == kTensor) hold = in.hold;
    Momenta<S, V, HOLD> momenta(stage, half, hold, codes, g_blk, tables, old_mag, beta1, omb1);

    // ---- rare: a NaN or Inf in the block. The reference's max ignores NaN; redo it that way and
    // let the exact (threshold) quantiser handle non-finite quotients.
    bool exact_path = false;
    if (__any_sync(0xffffffffu, !(absmax <= 3.0e38f))) {   // warp-uniform: the reduction below shuffles
        float mx = 0.0f;
        momenta.start(lane, LANES, nchunks);
        for (int it = 0, c = lane; it < rounds_all; ++it, c += LANES) {
            float m[V];
            momenta.template take<false>(it, c, LANES, nchunks, m);
            if (c >= nchunks) continue;
#pragma unroll
            for (int i = 0; i < V; ++i) mx = fmaxf(mx, fabsf(m[i]));
        }
        absmax = group_max(mx, LANES);
        exact_path = true;
    }
    if (lane == 0 && valid) store_state(t.mag, b, t.mag_dtype, absmax);

    const bool nonzero = absmax > 0.0f;
    const bool fastdiv = !exact_path && div_range_ok(absmax);
    const float rinv = fastdiv ? 1.0f / absmax : 0.0f;
    const bool wd = (flags & GEFEN_B200_STEP_WEIGHT_DECAY) != 0;
    const bool nesterov = (flags & GEFEN_B200_STEP_NESTEROV) != 0;
    const float wd_mul = t.wd_mul;
    const BlockScalars bs = {pair(-absmax, -absmax), pair(rinv, rinv), pair(step, step), pair(lr, lr), pair(wd_mul, wd_mul)};

    // ---- re-encode and update; the parameters of the next chunk are fetched while this one is encoded
    if (!kEarlyParams && load_p) ahead.start(p_blk, lane, LANES, nchunks);
    momenta.start(lane, LANES, nchunks);
    // The common case takes the loop that was compiled for it (the conditions are uniform over the warp: they
    // come from the launch and the tensor's descriptor, and a warp's blocks go one way together).
    if (__all_sync(0xffffffffu, fastdiv || !valid) && !muon && do_update) {
#define GEFEN_SECOND_PASS(WD_, STORE_, ONE_)                                                                                       \
    second_pass_common<S, V, HOLD, WD_, STORE_, ONE_>(L, tables, momenta, codes, p_blk, ahead, lane, LANES, nchunks, full,             \
                                                rounds_all, bs)
        if constexpr (V == 8) {
            const int store = param_mc != 0 ? 2 : (n_peers > 0 ? 1 : 0);
            if (store == 0) {
                if (tables.rounds == 1) { if (wd) GEFEN_SECOND_PASS(true, 0, true); else GEFEN_SECOND_PASS(false, 0, true); }
                else { if (wd) GEFEN_SECOND_PASS(true, 0, false); else GEFEN_SECOND_PASS(false, 0, false); }
            } else if (store == 1) { if (wd) GEFEN_SECOND_PASS(true, 1, false); else GEFEN_SECOND_PASS(false, 1, false); }
            else { if (wd) GEFEN_SECOND_PASS(true, 2, false); else GEFEN_SECOND_PASS(false, 2, false); }
        } else {
            constexpr int kStore = GSRC == 0 ? 0 : 1;
            if (wd) GEFEN_SECOND_PASS(true, kStore, false); else GEFEN_SECOND_PASS(false, kStore, false);
        }
#undef GEFEN_SECOND_PASS
        __syncwarp();  // the staging slice is free for this warp's next block
        return true;
    }
    if (GSRC == 0 && muon && __all_sync(0xffffffffu, fastdiv || !valid)) {
#define GEFEN_SECOND_PASS(NESTEROV_, ONE_)                                                                                         \
    second_pass_muon<S, V, HOLD, NESTEROV_, ONE_>(tables, momenta, codes, g_blk, p_blk, lane, LANES, nchunks, rounds_all, absmax,   \
                                                  bs.neg_absmax2, bs.rinv2, beta1, t.beta2)
        if (nesterov && tables.rounds == 1) GEFEN_SECOND_PASS(true, true);
        else if (nesterov) GEFEN_SECOND_PASS(true, false);
        else GEFEN_SECOND_PASS(false, false);
#undef GEFEN_SECOND_PASS
        __syncwarp();  // the staging slice is free for this warp's next block
        return true;
    }
    // Everything else (lr == 0, blocks that are all zero or hold NaN or Inf, magnitudes outside the range of the
    // reciprocal, GefenMuon's momentum over averaged gradients): the general loop.
    for (int it = 0, c = lane; it < rounds_all; ++it, c += LANES) {
        float m[V];
        momenta.template take<false>(it, c, LANES, nchunks, m);
        if (c >= nchunks) continue;
        Chunk<S, V> praw;
        if (load_p) praw.load(p_blk, c);
        uint32_t row[V];
        float q[V];
        if (fastdiv) {
            encode<V, false>(m, bs.neg_absmax2, bs.rinv2, tables, row);
        } else {
#pragma unroll
            for (int i = 0; i < V; ++i) {
                float x = 0.0f;
                if (nonzero) x = m[i] / absmax;
                row[i] = tables.exact_row(x);
            }
        }
#pragma unroll
        for (int i = 0; i < V; ++i) q[i] = tables.value(row[i]) * absmax;
        row_codes<V>(row).store(codes, c);
        if (muon) {
            if (nesterov) {
                // torch: m.mul_(momentum).add_(g, alpha=1-momentum) on the rounded momentum
                // (reference: gefen_muon.py:312-314); alpha travels in t.beta2.
                Chunk<S, V> g2;
                g2.load(g_blk, c);
                float g[V];
                g2.unpack(g);
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const float m1 = ScalarIO<S>::round(ScalarIO<S>::round(q[i]) * beta1);
                    q[i] = fmaf(t.beta2, g[i], m1);
                }
            }
            Chunk<S, V> out;
            out.pack(q);
            out.store(p_blk, c);
        } else if (do_update) {
            float pv[V];
            praw.unpack(pv);
            if (wd) {
#pragma unroll
                for (int i = 0; i < V; ++i) pv[i] *= wd_mul;
                Chunk<S, V> rounded;       // the separate multiply of the reference rounds to the parameter dtype
                rounded.pack(pv);
                rounded.unpack(pv);
            }
#pragma unroll
            for (int i = 0; i < V; ++i) pv[i] = fmaf(-(q[i] * step), lr, pv[i]);
            praw.pack(pv);
            if (V == 8 && param_mc != 0) {
                if constexpr (V == 8) praw.store_all(peer_ptr(p_blk, param_mc), c);   // every rank's copy, this one included
            } else {
                praw.store(p_blk, c);
                for (int r = 0; r < n_peers; ++r) praw.store(peer_ptr(p_blk, L.peer_delta[r]), c);
            }
        }
    }
    __syncwarp();  // the staging slice is free for this warp's next block
    return true;
}

// Threads per CTA: sixteen warps of 128 registers; the tables leave room for sixteen staging slices of 2048 elements.
constexpr int kVecThreads = 512;
struct DirectInputs {};

// GSRC: see warp_block_step. FULL: every tensor of the launch has whole-warp blocks (32 lanes per block);
// otherwise none has. The kinds are separate kernels so that each is compiled (registers, code size) for
// its own loop structure. HOLD: see Momenta.
template <typename S, int V, int GSRC, bool FULL, int HOLD = kShared>
__global__ void __launch_bounds__(kVecThreads, 1) step_vec_kernel(const __grid_constant__ StepLaunch L,
                                                                  const __grid_constant__ StepRows rows) {
    SmemView s;
    let_successor_in(L);
    if (smem_u32(g_smem) > kFixed) {   // (static variables have outgrown their share: nothing is done, the status says so)
        if (threadIdx.x == 0) atomicOr(&g_step_status, 2);
        wait_for_predecessor();
        return;
    }
    if (!stage_tables(L.ws, fast_smem(kWsAt), s, L.spin_limit)) { wait_for_predecessor(); return; }
    const gefen_b200_step_tensor_t* table = L.table != nullptr ? L.table : rows.row;

    const int lane = threadIdx.x & 31;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int warps = blockDim.x >> 5;
    const LaneTables tables = build_lane_tables(s, fast_smem(kStageAt));
    float* stage = reinterpret_cast<float*>(fast_smem(kStageAt)) + static_cast<size_t>(warp) * L.stage_floats;
    const long long warp_global = static_cast<long long>(blockIdx.x) * warps + warp;
    const long long warp_stride = static_cast<long long>(gridDim.x) * warps;
    // On this path first_block and total_blocks count work units (see vec_units), not blocks.
    // the warp's slot lies where the codebook was staged (build_lane_tables has consumed it)
    TensorSlot<S>& t = reinterpret_cast<TensorSlot<S>*>(fast_smem(kWsAt))[warp];
    static_assert(sizeof(TensorSlot<S>) * (kVecThreads / 32) <= kSmemWs, "a slot per warp");
    DirectInputs in;
    long long t_first = 0, t_units = 0;
    for (long long gb = warp_global; gb < L.total_blocks; gb += warp_stride) {
        if (gb < t_first || gb >= t_first + t_units) {
            const gefen_b200_step_tensor_t* found = table + find_tensor_warp(table, L.n_tensors, gb);
            if (lane == 0) t.load(found, V, chunk_sources(L));
            __syncwarp();
            t_first = t.first;
            t_units = t.units;
        }
        const long long unit = gb - t_first;
        const long long next = unit + warp_stride;
        // same tensor: hint the next block of this warp
        if (GSRC == 0 && lane == 0 && next + 1 < t_units) {   // (not a ragged last unit)
            const long long unit_elems = unit_elements(t.period, V);
            const long long elem0 = next * unit_elems;
            prefetch_l2_range(t.codes + elem0, unit_elems);
            prefetch_l2_range(t.g + elem0, unit_elems * sizeof(S));
            if (!(t.flags & GEFEN_B200_STEP_MUON) && unit_elems * static_cast<int>(sizeof(S)) < 8192) prefetch_l2_range(t.p + elem0, unit_elems * sizeof(S));
        }
        warp_block_step<S, V, GSRC, FULL, HOLD>(t, unit, L, tables, stage, in, lane);
    }
    wait_for_predecessor();
}

// --------------------------------------------------------------------------- ring kernel
// The same step for every usual tensor: gradients in this GPU's buffer, units of up to kRingBytes of codes and gradients.
// What is different:
//  * The codes and gradients of a warp's next unit are on their way to shared memory (two bulk copies and one mbarrier
//    per warp) from the moment that the first pass over the current unit is over, its magnitude and second moment to
//    registers, its parameters to L2. The first pass waits for nothing.
//  * The updated momenta of the unit wait in tensor memory (tcgen05.st / tcgen05.ld, four bytes exactly as they are),
//    which leaves shared memory to those buffers and takes a quarter of the traffic off its data pipe.
// Twenty warps of 96 registers (fp32: sixteen of 128) instead of sixteen of 128. Before, sixteen warps could not cover the
// loads of the first pass (long scoreboard 2.06 of 7 cycles per issue, 56 % of the issue slots); now 70 % are used. 134 M
// bf16 elements (67 M fp32) with second moment and decay, ms before and now: blocks of 2048 0.230 -> 0.198, 1664 0.244 ->
// 0.191, 1120 0.297 -> 0.224, 512 0.240 -> 0.195, 128 0.335 -> 0.239; fp32 768 0.193 -> 0.165, 1152 0.179 -> 0.164; GefenMuon's
// momentum, blocks of 2048, 0.244 -> 0.174; rows that are multiples of four only, 300 0.378 -> 0.256 (120 M), 1500 0.295 -> 0.223.
template <typename S> constexpr int ring_threads() { return sizeof(S) == 2 ? 640 : 512; }
// The warps' descriptors and buffers start behind the scratch of the tables: what the CTA has written there with ordinary
// stores is not ordered before the bulk copies.
constexpr int kRingAt = kStageAt + kTableScratch;
constexpr int kSmemRing = kRingAt - 1024;       // dynamic shared memory up to them

// A warp's descriptors (the current unit's and the next one's) and the barrier of its buffers.
template <typename S> struct alignas(16) RingWarp {
    TensorSlot<S> slot[2];
    uint64_t bar;
};

template <typename S, int V, bool FULL> struct RingInputs {
    const StepLaunch& L;
    const gefen_b200_step_tensor_t* const table;
    RingWarp<S>& w;
    const uint32_t buffer, hold;      // shared-memory address of the buffers, tensor-memory address of the warp's columns
    const int lane;
    const long long stride;
    long long unit;                   // the unit that the buffers hold or wait for
    long long first = 0, units = 0;   // of its tensor
    int slot = 0;
    uint32_t parity = 0;
    float mag = 0.0f, v = 0.0f;       // of its blocks
    __device__ __forceinline__ RingInputs(const StepLaunch& l, const gefen_b200_step_tensor_t* rows, RingWarp<S>& own, uint32_t buffers, uint32_t columns,
                                          int lane_, long long unit0, long long stride_)
        : L(l), table(rows), w(own), buffer(buffers), hold(columns), lane(lane_), stride(stride_), unit(unit0) {}
    // the copies start on 16 bytes: where the unit's first byte lies in a buffer
    __device__ __forceinline__ uint32_t g_at(const S* g) const { return buffer + (static_cast<uint32_t>(reinterpret_cast<uintptr_t>(g)) & 15u); }
    __device__ __forceinline__ uint32_t codes_at(const uint8_t* codes) const {
        return buffer + L.ring_g + (static_cast<uint32_t>(reinterpret_cast<uintptr_t>(codes)) & 15u);
    }
    // [p, p + bytes) widened to 16-byte boundaries: the bytes beside it lie in the same 16 bytes as bytes of the range, and
    // nothing reads their copies.
    static __device__ __forceinline__ uint32_t widened(const void* p, uint32_t bytes) {
        return ((static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p)) & 15u) + bytes + 15u) & ~15u;
    }
    static __device__ __forceinline__ void copy(uint32_t dst, const void* p, uint32_t bytes, uint64_t* bar) {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                     "l"(reinterpret_cast<uintptr_t>(p) & ~static_cast<uintptr_t>(15)), "r"(bytes), "r"(smem_u32(bar)) : "memory");
    }
    __device__ __forceinline__ void request() {
        if (unit >= L.total_blocks) return;
        if (unit < first || unit >= first + units) {
            const gefen_b200_step_tensor_t* found = table + find_tensor_warp(table, L.n_tensors, unit);
            slot ^= 1;
            if (lane == 0) w.slot[slot].load(found, V, 0);
            __syncwarp();
            first = w.slot[slot].first;
            units = w.slot[slot].units;
        }
        const TensorSlot<S>& t = w.slot[slot];
        const int period = t.period, shift = FULL ? 5 : lanes_shift(period / V, V);
        const long long b0 = (unit - first) << (5 - shift), left = t.num_blocks - b0;
        const int blocks = FULL ? 1 : (left < (1 << (5 - shift)) ? static_cast<int>(left) : 1 << (5 - shift));
        const bool muon = (t.flags & GEFEN_B200_STEP_MUON) != 0;
        if (lane == 0) {
            const uint32_t elems = static_cast<uint32_t>(blocks * period);
            const S* const g = t.g + b0 * period;
            const uint8_t* const codes = t.codes + b0 * period;
            const uint32_t g_bytes = widened(g, elems * static_cast<uint32_t>(sizeof(S))), code_bytes = widened(codes, elems);
            mbar_expect_tx(&w.bar, g_bytes + code_bytes);
            copy(buffer, g, g_bytes, &w.bar);
            copy(buffer + L.ring_g, codes, code_bytes, &w.bar);
            if (!muon) prefetch_l2_range(t.p + b0 * period, elems * static_cast<uint32_t>(sizeof(S)));
        }
        const long long b = b0 + (lane >> shift);
        const bool valid = (lane >> shift) < blocks;
        mag = valid ? load_state(t.mag, b, t.mag_dtype) : 0.0f;
        v = valid && !muon ? (L.stepsize != nullptr ? L.stepsize[b] : load_state(t.v, b, t.v_dtype)) : 1.0f;
    }
    __device__ __forceinline__ void request_next() {
        unit += stride;
        request();
    }
    __device__ __forceinline__ bool arrived(uint32_t limit) {
        const bool ok = mbar_wait_bounded(&w.bar, parity, limit);
        parity ^= 1u;
        return __all_sync(0xffffffffu, ok);
    }
};

template <typename S, int V, bool FULL>
__global__ void __launch_bounds__(ring_threads<S>(), 1) step_ring_kernel(const __grid_constant__ StepLaunch L,
                                                                         const __grid_constant__ StepRows rows) {
    __shared__ uint32_t tmem_base;
    SmemView s;
    let_successor_in(L);
    if (smem_u32(g_smem) > kFixed) {   // (as in step_vec_kernel)
        if (threadIdx.x == 0) atomicOr(&g_step_status, 2);
        wait_for_predecessor();
        return;
    }
    if (!stage_tables(L.ws, fast_smem(kWsAt), s, L.spin_limit)) { wait_for_predecessor(); return; }
    const int lane = threadIdx.x & 31;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int warps = blockDim.x >> 5;
    const LaneTables tables = build_lane_tables(s, fast_smem(kStageAt));
    RingWarp<S>& own = reinterpret_cast<RingWarp<S>*>(fast_smem(kRingAt))[warp];
    if (warp == 0) {   // (waits while another CTA of this SM holds the columns; that one does not wait for this launch, see let_successor_in)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(L.tmem_columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (lane == 0) {
        mbar_init(&own.bar, 1);
        fence_mbar_init();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // a warp reaches the 32 lanes of tensor memory that its place in its group of four gives it
    const uint32_t hold = tmem_base + (static_cast<uint32_t>(warp & 3) << 21) + static_cast<uint32_t>((warp >> 2) * L.hold_columns);
    const uint32_t buffer = kRingAt + static_cast<uint32_t>(sizeof(RingWarp<S>)) * warps + static_cast<uint32_t>(warp * (L.ring_g + L.ring_codes));
    // Neighbouring units go to different SMs; where they share lines of memory (small chunks) and there are many, to
    // the warps of one SM. (134 M bf16 elements in blocks of 1664 0.203 against 0.188 ms, of 128 0.256 / 0.236; with
    // chunks of four, blocks of 2500, 0.234 / 0.261; chunks of one, blocks of 27, 0.540 / 0.612.)
    const long long warp_stride = static_cast<long long>(gridDim.x) * warps;
    const bool spread = V == 8 || L.total_blocks <= warp_stride;
    const long long warp_global = spread ? static_cast<long long>(warp) * gridDim.x + blockIdx.x : static_cast<long long>(blockIdx.x) * warps + warp;
    RingInputs<S, V, FULL> in(L, L.table != nullptr ? L.table : rows.row, own, buffer, hold, lane, warp_global, warp_stride);
    in.request();
    for (long long gb = warp_global; gb < L.total_blocks; gb += warp_stride) {
        if (!warp_block_step<S, V, 0, FULL, kTensor>(own.slot[in.slot], gb - in.first, L, tables, nullptr, in, lane)) {
            // the wait for the inputs ran out: this warp leaves its blocks as they are, but not before the copies have ended
            if (lane == 0) atomicOr(&g_step_status, 1);
            mbar_wait_bounded(&own.bar, in.parity ^ 1u, kStageDrainLimit);
            break;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(L.tmem_columns) : "memory");
    wait_for_predecessor();
}

// One gradient element as the step sees it: the local value, or the rounded average over the
// ranks' buffers (see StepLaunch::grad_delta).
template <typename S>
__device__ __forceinline__ float gradient_element(const S* g, const StepLaunch& L) {
    if (L.n_grad_srcs == 0) return ScalarIO<S>::load(g);
    float acc = 0.0f;
    for (int r = 0; r < L.n_grad_srcs; ++r) acc += ScalarIO<S>::load(peer_ptr(g, L.grad_delta[r]));
    return ScalarIO<S>::round(acc * L.grad_scale);
}

// --------------------------------------------------------------------------- generic path
// GROUP = 32: one warp per block; GROUP = 256: one CTA per block. Two passes, scalar accesses.
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

template <typename S, int GROUP>
__global__ void __launch_bounds__(kThreads) step_generic_kernel(const __grid_constant__ StepLaunch L,
                                                                const __grid_constant__ StepRows rows) {
    __shared__ float red_max[kWarps];
    __shared__ float red_sum[kWarps];
    SmemView s;
    let_successor_in(L);
    if (!stage_tables(L.ws, g_smem, s, L.spin_limit)) { wait_for_predecessor(); return; }
    const gefen_b200_step_tensor_t* table = L.table != nullptr ? L.table : rows.row;

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int tig = (GROUP == 32) ? lane : static_cast<int>(threadIdx.x);
    const long long group_global = (GROUP == 32) ? static_cast<long long>(blockIdx.x) * kWarps + warp
                                                 : static_cast<long long>(blockIdx.x);
    const long long group_stride = (GROUP == 32) ? static_cast<long long>(gridDim.x) * kWarps
                                                 : static_cast<long long>(gridDim.x);

    for (long long gb = group_global; gb < L.total_blocks; gb += group_stride) {
        const gefen_b200_step_tensor_t* tp = table + find_tensor(table, L.n_tensors, gb);
        const int period = static_cast<int>(tp->period);
        const uint32_t flags = tp->flags;
        // 4-bit codes with an odd period: blocks 2k and 2k + 1 share the byte between them (and with no other
        // block), so the pair is one unit of work and its two blocks are taken one after the other by the same
        // threads; see paired_units.
        const int halves = ((flags & GEFEN_B200_STEP_PACKED) != 0 && (period & 1) != 0) ? 2 : 1;
        for (int half = 0; half < halves; ++half) {
        const long long b = (gb - tp->first_block) * halves + half;
        if (b >= tp->num_blocks) break;
        const long long start = b * period;
        const bool muon = (flags & GEFEN_B200_STEP_MUON) != 0;
        const bool period1 = (flags & GEFEN_B200_STEP_PERIOD1) != 0;
        const bool fuse_v = (flags & GEFEN_B200_STEP_FUSE_VMEAN) != 0;
        const bool wd = (flags & GEFEN_B200_STEP_WEIGHT_DECAY) != 0;
        const bool nesterov = (flags & GEFEN_B200_STEP_NESTEROV) != 0;
        const S* g = static_cast<const S*>(tp->g) + start;
        S* prm = static_cast<S*>(tp->p) + start;
        // 4-bit codes (reference: automatic_gefen_fused_kernel.cu:14-57): two per byte over the whole
        // tensor, low nibble first. A thread owns a byte and the (one or two) elements of this block in it: no
        // atomics (the reference uses atomicCAS). lead = 1: the block starts on the high nibble of its first
        // byte, whose low nibble belongs to the block before; likewise the last byte's high nibble may belong
        // to the block after. Such bytes are rewritten with the other block's nibble kept.
        const bool packed = (flags & GEFEN_B200_STEP_PACKED) != 0;
        const int per = packed ? 2 : 1;
        const int lead = packed ? static_cast<int>(start & 1) : 0;
        uint8_t* codes = tp->codes + (packed ? start / 2 : start);
        void* mag_ptr = tp->mag;
        void* v_ptr = tp->v;
        const int mag_dtype = tp->mag_dtype, v_dtype = tp->v_dtype;
        const float beta1 = tp->beta1;
        const float omb1 = 1.0f - beta1;
        const float beta2 = tp->beta2;
        const float omb2 = 1.0f - beta2;
        const float lr = tp->lr, bc1 = tp->bc1, bc2 = tp->bc2, eps = tp->eps, wd_mul = tp->wd_mul;
        const float old_mag = load_state(mag_ptr, b, mag_dtype);

        // pass 1: NaN-ignoring absmax of the updated momentum (the reference's `>` test), sum g^2;
        // period-1 tensors update their per-element second moment here
        // (reference: automatic_gefen_fused_kernel.cu:350-366).
        float absmax = 0.0f, sumsq = 0.0f;
        for (int i0 = tig * per - lead; i0 < period; i0 += GROUP * per) {
            const uint32_t byte = codes[packed ? (i0 + lead) / 2 : i0];
            for (int e = 0; e < per; ++e) {
                const int i = i0 + e;
                if (i < 0 || i >= period) continue;   // the neighbouring block's nibble
                const uint32_t old_code = packed ? ((byte >> (4 * e)) & 0xFu) : byte;
                const float gi = gradient_element(g + i, L);
                if (period1) {
                    const float prev = load_state(v_ptr, start + i, v_dtype);
                    store_state(v_ptr, start + i, v_dtype, fmaf(beta2, prev, (omb2 * gi) * gi));
                }
                const float cur = old_mag * s.cb[old_code];
                const float u = period1 ? ema_update_period1(beta1, cur, omb1, gi) : ema_update(beta1, cur, omb1, gi);
                absmax = fmaxf(absmax, fabsf(u));
                sumsq = fmaf(gi, gi, sumsq);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) absmax = fmaxf(absmax, __shfl_xor_sync(0xffffffffu, absmax, o));
        sumsq = warp_sum(sumsq);
        if (GROUP > 32) {
            __syncthreads();  // previous iteration's readers are done with red_*
            if (lane == 0) { red_max[warp] = absmax; red_sum[warp] = sumsq; }
            __syncthreads();
            absmax = red_max[0];
            sumsq = red_sum[0];
#pragma unroll
            for (int w = 1; w < kWarps; ++w) { absmax = fmaxf(absmax, red_max[w]); sumsq += red_sum[w]; }
        }

        float step = 0.0f;
        if (!muon && !period1) {
            if (L.stepsize != nullptr) {
                step = L.stepsize[b];
            } else {
                float v = load_state(v_ptr, b, v_dtype);
                float nv = 0.0f;
                if (fuse_v) {
                    nv = fmaf(beta2, v, omb2 * (sumsq / static_cast<float>(period)));
                    // every thread computes the same rounded value; one thread stores it below
                    if (v_dtype == GEFEN_B200_F32) v = nv;
                    else if (v_dtype == GEFEN_B200_BF16) v = __bfloat162float(__float2bfloat16_rn(nv));
                    else v = __half2float(__float2half_rn(nv));
                }
                step = adam_step_size(v, bc1, bc2, eps);
                if (fuse_v) {
                    if (GROUP > 32) __syncthreads(); else __syncwarp();  // everyone has read the old vmean
                    if (tig == 0) store_state(v_ptr, b, v_dtype, nv);
                }
            }
        }
        if (GROUP > 32) __syncthreads(); else __syncwarp();  // old magnitude was read by everyone
        if (tig == 0) store_state(mag_ptr, b, mag_dtype, absmax);
        const bool do_update = muon || period1 || lr != 0.0f;

        // pass 2: re-encode and update
        for (int i0 = tig * per - lead; i0 < period; i0 += GROUP * per) {
            const uint32_t byte = codes[packed ? (i0 + lead) / 2 : i0];
            uint32_t new_byte = 0u;
            for (int e = 0; e < per; ++e) {
            const int i = i0 + e;
            if (i < 0 || i >= period) {   // the neighbouring block's nibble stays
                new_byte |= byte & (0xFu << (4 * e));
                continue;
            }
            const uint32_t old_code = packed ? ((byte >> (4 * e)) & 0xFu) : byte;
            const float gi = gradient_element(g + i, L);
            const float cur = old_mag * s.cb[old_code];
            const float u = period1 ? ema_update_period1(beta1, cur, omb1, gi) : ema_update(beta1, cur, omb1, gi);
            float x = 0.0f;
            if (absmax > 0.0f) x = u / absmax;
            const uint32_t code = static_cast<uint32_t>(entry_exact(x, s.thr, s.cb, s.k));
            new_byte |= packed ? ((code & 0xFu) << (4 * e)) : code;
            const float q = s.cb[code] * absmax;
            if (muon) {
                float out = q;
                if (nesterov) out = fmaf(beta2, gi, ScalarIO<S>::round(ScalarIO<S>::round(q) * beta1));
                ScalarIO<S>::store(prm + i, out);
            } else if (do_update) {
                float st = step;
                if (period1) st = adam_step_size(load_state(v_ptr, start + i, v_dtype), bc1, bc2, eps);
                float pi = ScalarIO<S>::load(prm + i);
                if (wd) pi = ScalarIO<S>::round(pi * wd_mul);
                const float updated = fmaf(-(q * st), lr, pi);
                ScalarIO<S>::store(prm + i, updated);
                for (int r = 0; r < L.n_peers; ++r) ScalarIO<S>::store(peer_ptr(prm + i, L.peer_delta[r]), updated);
            }
            }
            codes[packed ? (i0 + lead) / 2 : i0] = static_cast<uint8_t>(new_byte);
        }
        if (halves > 1) {   // the pair's second block reads the shared byte after this block has written it
            if (GROUP > 32) __syncthreads(); else __syncwarp();
        }
        }
    }
    wait_for_predecessor();
}

// --------------------------------------------------------------------------- vectors
// Period-1 tensors (biases, norm weights): a second moment per element, one magnitude per `period` <= 256 elements
// (reference: automatic_gefen_fused_kernel.cu:320-407). One warp takes one run of that many elements, at most eight per
// lane, with all loads issued at once: such launches are a few hundred warps and take as long as their chain of
// dependent loads (98 vectors of GPT-2: 21 us with the generic kernel's loops).
constexpr int kVectorMost = 256;
constexpr int kVectorThreads = 128;
template <typename S>
__global__ void __launch_bounds__(kVectorThreads) step_vector_kernel(const __grid_constant__ StepLaunch L,
                                                                     const __grid_constant__ StepRows rows) {
    constexpr int E = kVectorMost / 32;
    let_successor_in(L);
    const gefen_b200_step_tensor_t* table = L.table != nullptr ? L.table : rows.row;
    const int lane = threadIdx.x & 31;
    const long long gb = static_cast<long long>(blockIdx.x) * (kVectorThreads / 32) + (threadIdx.x >> 5);
    const bool active = gb < L.total_blocks;
    const gefen_b200_step_tensor_t* tp = table + find_tensor_warp(table, L.n_tensors, active ? gb : 0);
    const long long b = gb - tp->first_block;
    const int period = active ? static_cast<int>(tp->period) : 0;
    const long long start = b * period;
    const S* g = static_cast<const S*>(tp->g) + start;
    S* prm = static_cast<S*>(tp->p) + start;
    uint8_t* codes = tp->codes + start;
    void* const v_ptr = tp->v;
    void* const mag_ptr = tp->mag;
    const int mag_dtype = tp->mag_dtype, v_dtype = tp->v_dtype;
    const float beta1 = tp->beta1, beta2 = tp->beta2, lr = tp->lr, bc1 = tp->bc1, bc2 = tp->bc2, eps = tp->eps, wd_mul = tp->wd_mul;
    const bool wd = (tp->flags & GEFEN_B200_STEP_WEIGHT_DECAY) != 0;
    float gi[E], vi[E], pi[E];
    uint32_t code[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = lane + 32 * e;
        if (i < period) {
            gi[e] = ScalarIO<S>::load(g + i);
            vi[e] = load_state(v_ptr, start + i, v_dtype);
            pi[e] = ScalarIO<S>::load(prm + i);
            code[e] = codes[i];
        }
    }
    const float old_mag = active ? load_state(mag_ptr, b, mag_dtype) : 0.0f;
    SmemView s;
    if (!stage_tables(L.ws, g_smem, s, L.spin_limit)) { wait_for_predecessor(); return; }
    if (active) {
        const float omb1 = 1.0f - beta1, omb2 = 1.0f - beta2;
        float u[E];
        float absmax = 0.0f;   // NaN-ignoring, as the reference's `>` test
#pragma unroll
        for (int e = 0; e < E; ++e) {
            if (lane + 32 * e < period) {
                vi[e] = store_state(v_ptr, start + lane + 32 * e, v_dtype, fmaf(beta2, vi[e], (omb2 * gi[e]) * gi[e]));
                u[e] = ema_update_period1(beta1, old_mag * s.cb[code[e]], omb1, gi[e]);
                absmax = fmaxf(absmax, fabsf(u[e]));
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) absmax = fmaxf(absmax, __shfl_xor_sync(0xffffffffu, absmax, o));
        if (lane == 0) store_state(mag_ptr, b, mag_dtype, absmax);   // (the shuffles are behind every lane's read of the old one)
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int i = lane + 32 * e;
            if (i < period) {
                const float x = absmax > 0.0f ? u[e] / absmax : 0.0f;
                const uint32_t c = static_cast<uint32_t>(entry_exact(x, s.thr, s.cb, s.k));
                codes[i] = static_cast<uint8_t>(c);
                const float p0 = wd ? ScalarIO<S>::round(pi[e] * wd_mul) : pi[e];
                ScalarIO<S>::store(prm + i, fmaf(-((s.cb[c] * absmax) * adam_step_size(vi[e], bc1, bc2, eps)), lr, p0));
            }
        }
    }
    wait_for_predecessor();
}

// --------------------------------------------------------------------------- vmean only
// vmean[b] = beta2*vmean[b] + (1-beta2)*mean(g[b,:]^2) (reference: automatic_vmean_kernel.cu:12-51).
// One warp per block, fp32 accumulation.
template <typename S>
__global__ void __launch_bounds__(kThreads) vmean_kernel(void* __restrict__ vmean, int v_dtype, const S* __restrict__ g,
                                                         long long num_blocks, long long period, float beta2) {
    const int lane = threadIdx.x & 31;
    const long long warp_global = static_cast<long long>(blockIdx.x) * kWarps + (threadIdx.x >> 5);
    const long long warp_stride = static_cast<long long>(gridDim.x) * kWarps;
    const bool vec = (sizeof(S) == 2) && (period % 8 == 0) && ((reinterpret_cast<uintptr_t>(g) & 15u) == 0);
    for (long long b = warp_global; b < num_blocks; b += warp_stride) {
        const S* gb = g + b * period;
        float sum = 0.0f;
        if (vec) {
            const uint4* g4 = reinterpret_cast<const uint4*>(gb);
            for (long long c = lane; c < period / 8; c += 32) {
                const uint4 raw = g4[c];
                const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const S* h = reinterpret_cast<const S*>(&w[i]);
                    const float a = ScalarIO<S>::load(h), c2 = ScalarIO<S>::load(h + 1);
                    sum = fmaf(a, a, sum);
                    sum = fmaf(c2, c2, sum);
                }
            }
        } else {
            for (long long i = lane; i < period; i += 32) {
                const float a = ScalarIO<S>::load(gb + i);
                sum = fmaf(a, a, sum);
            }
        }
        sum = warp_sum(sum);
        if (lane == 0) {
            const float mean_sq = sum / static_cast<float>(period);
            const float prev = load_state(vmean, b, v_dtype);
            store_state(vmean, b, v_dtype, fmaf(beta2, prev, (1.0f - beta2) * mean_sq));
        }
    }
}

// --------------------------------------------------------------------------- multicast sum
// dst[i] = round(scale * sum over the ranks of src[i]), the sum formed by the switch: the gradient the
// staged kernel sees when it reads through the multicast mapping, written out for checks.
template <typename S>
__global__ void __launch_bounds__(kThreads) multicast_sum_kernel(void* __restrict__ dst, const void* __restrict__ src_mc,
                                                                 long long chunks, float scale) {
    const long long stride = static_cast<long long>(gridDim.x) * kThreads;
    for (long long c = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x; c < chunks; c += stride) {
        Chunk<S, 8> v;
        v.load_sum(src_mc, c);
        float f[8];
        v.unpack(f);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] *= scale;
        v.pack(f);
        v.store(dst, c);
    }
}

// --------------------------------------------------------------------------- GefenMuon apply
// p <- round(p * wd_mul) ; p <- round(p + alpha * u)   (reference: gefen_muon.py:326-329, torch's mul_ and
// add_(update, alpha=-adjusted_lr): each rounds to the parameter dtype), one pass over p and u instead of
// two kernels, and - for ZeRO-1 ranks whose parameter buffers are mapped into each other - the updated
// parameters also stored to the peers' copies (the all-gather).
template <typename S>
__global__ void __launch_bounds__(kThreads) muon_apply_kernel(S* __restrict__ p, const S* __restrict__ u, long long numel,
                                                              float wd_mul, bool decay, float alpha, bool vec,
                                                              const __grid_constant__ StepLaunch L) {
    const long long stride = static_cast<long long>(gridDim.x) * kThreads;
    const long long tid = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
    const long long chunks = vec ? numel >> 3 : 0;
    for (long long c = tid; c < chunks; c += stride) {
        Chunk<S, 8> pr, ur;
        pr.load(p, c);
        ur.load(u, c);
        float pv[8], uv[8];
        pr.unpack(pv);
        ur.unpack(uv);
        if (decay) {
#pragma unroll
            for (int i = 0; i < 8; ++i) pv[i] *= wd_mul;
            pr.pack(pv);
            pr.unpack(pv);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) pv[i] = fmaf(alpha, uv[i], pv[i]);
        pr.pack(pv);
        pr.store(p, c);
        for (int r = 0; r < L.n_peers; ++r) pr.store(peer_ptr(p, L.peer_delta[r]), c);
    }
    for (long long i = chunks * 8 + tid; i < numel; i += stride) {
        float pv = ScalarIO<S>::load(p + i);
        if (decay) pv = ScalarIO<S>::round(pv * wd_mul);
        pv = fmaf(alpha, ScalarIO<S>::load(u + i), pv);
        ScalarIO<S>::store(p + i, pv);
        for (int r = 0; r < L.n_peers; ++r) ScalarIO<S>::store(peer_ptr(p + i, L.peer_delta[r]), pv);
    }
}

// --------------------------------------------------------------------------- host dispatch
static int grid_for(long long groups_needed, int groups_per_cta, int ctas_per_sm) {
    long long ctas = (groups_needed + groups_per_cta - 1) / groups_per_cta;
    const long long cap = static_cast<long long>(sm_count()) * ctas_per_sm;
    if (ctas > cap) ctas = cap;
    if (ctas < 1) ctas = 1;
    return static_cast<int>(ctas);
}

constexpr int kFastMaxPeriod = 8192;
constexpr int kStaticSmemSlack = 256;   // static __shared__ of the kernels (counted against the per-CTA limit)
constexpr int kCtaReservedSmem = 1024;  // what the hardware sets aside per resident CTA (not part of the limit)

// Per-device launch configuration (cudaFuncSetAttribute) is done once per kernel and device, under
// this lock; device ordinals beyond the table are refused with a clear error.
constexpr int kMaxDevices = 64;
static std::mutex g_config_mutex;
static int current_device(int* dev) {
    GEFEN_CHECK_CUDA(cudaGetDevice(dev));
    GEFEN_CHECK_ARG(*dev >= 0 && *dev < kMaxDevices, "Unsupported device ordinal %d (at most %d devices).", *dev, kMaxDevices);
    return GEFEN_B200_OK;
}

static int env_int(const char* name) {
    const char* e = getenv(name);
    const int v = e != nullptr ? atoi(e) : 0;
    return v < 0 ? 0 : v;
}
// GEFEN_B200_STEP_WARPS=n caps the warps per CTA of the staged and the ring kernel (for measurements; read once).
static int warps_override() {
    static const int cached = env_int("GEFEN_B200_STEP_WARPS");
    return cached;
}

// Iteration limits of the step kernels' wait for their staged tables and of a ring warp's wait for its inputs.
// gefen_b200_debug_set_stage_spin_limit and gefen_b200_debug_set_input_spin_limit lower them so that a test can watch the
// time-out paths (status word, kernel returns) without a fault.
constexpr unsigned int kDefaultSpinLimit = 4000000u;
static unsigned int g_stage_spin_limit = kDefaultSpinLimit, g_input_spin_limit = kDefaultSpinLimit;
static unsigned int spin_limit_of(int64_t limit) { return limit < 0 || limit > 0xFFFFFFFFll ? kDefaultSpinLimit : static_cast<unsigned int>(limit); }

template <typename K>
static int launch_step(K kernel, int grid, int threads, int smem, const StepLaunch& L, const StepRows& rows,
                       cudaStream_t stream) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(grid));
    config.blockDim = dim3(static_cast<unsigned>(threads));
    config.dynamicSmemBytes = static_cast<size_t>(smem);
    config.stream = stream;
    cudaLaunchAttribute overlap = {};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    if (L.follows) {
        config.attrs = &overlap;
        config.numAttrs = 1;
    }
    GEFEN_CHECK_CUDA(cudaLaunchKernelEx(&config, kernel, L, rows));
    return GEFEN_B200_OK;
}

// Bytes of a warp's slice of staged momenta (max_unit: the largest need of the launch, see unit_floats; a slice starts on 16
// bytes; 256 floats: build_lane_tables), and the slices of a CTA.
static int stage_bytes_for(long long max_unit) { return static_cast<int>(((max_unit > 256 ? max_unit : 256) * 4 + 15) / 16 * 16); }
static int staged_warps(int stage_bytes) {
    int most = kVecThreads / 32;
    if (warps_override() > 0 && warps_override() < most) most = warps_override();
    const int fit = (kMaxSmem - kStaticSmemSlack - kSmemTables) / stage_bytes;
    return fit < most ? fit : most;
}

template <typename S, int V, int GSRC, bool FULL, int HOLD = kShared>
static int launch_vec_variant(StepLaunch L, const StepRows& rows, long long max_unit, cudaStream_t stream) {
    static bool configured[kMaxDevices];
    auto kernel = step_vec_kernel<S, V, GSRC, FULL, HOLD>;
    {
        int dev = 0;
        const int rc = current_device(&dev);
        if (rc != GEFEN_B200_OK) return rc;
        std::lock_guard<std::mutex> lock(g_config_mutex);
        if (!configured[dev]) {
            GEFEN_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem - kStaticSmemSlack));
            configured[dev] = true;
        }
    }
    // a warp stages one unit: one long block, or the 32 / lanes shorter blocks that share the warp
    const int stage_bytes = stage_bytes_for(HOLD == kShared ? max_unit : 0);
    int warps = staged_warps(stage_bytes);
    if (warps < 1) return fail(GEFEN_B200_EINVAL, "internal: unit of %lld elements too large for the staged path", max_unit);
    if (L.total_blocks < warps) warps = static_cast<int>(L.total_blocks);
    const int smem = kSmemTables + stage_bytes * warps;
    int ctas_per_sm = (kMaxSmem + kCtaReservedSmem) / (smem + kStaticSmemSlack + kCtaReservedSmem);
    if (ctas_per_sm > 2) ctas_per_sm = 2;
    if (ctas_per_sm < 1) ctas_per_sm = 1;
    L.stage_floats = stage_bytes / 4;
    const int grid = grid_for(L.total_blocks, warps, ctas_per_sm);
    return launch_step(kernel, grid, warps * 32, smem, L, rows, stream);
}

// Kernels of the fast path beyond the classes of tensors: kRing + class = step_ring_kernel, kTwiceClass = long blocks
// whose momenta are formed twice; a class by itself = step_vec_kernel with staged momenta.
constexpr int kTwiceClass = 7, kRing = 16;
// The most that the ring kernel's buffers of a unit may take (codes and gradients; this much leaves six warps). Blocks of
// 4096 fp32 elements: 0.222 ms with the momenta formed twice (67 M elements), 0.194 here; bf16, 134 M: 4096 0.268 against
// 0.227, 5120 0.294 / 0.242, 8192 (24 KB) 0.300 / 0.323.
constexpr int kRingBytes = 20480;
static int route(int cls, long long period, int dtype, int n_peers, int n_grad_srcs) {
    if (cls < 1 || cls > 5 || n_grad_srcs > 0) return cls;   // (averaged gradients: the staged kernels)
    if (cls >= 3 && n_peers > 0) return cls;                 // (small chunks with peer stores: staged)
    const int v = cls <= 2 ? 8 : (cls == 3 ? 4 : (cls == 4 ? 2 : 1)), es = dtype_size(dtype);
    // Small chunks with fewer than four lanes per block read the buffers from many blocks at once, on the same banks unless
    // a block is an odd number of chunks.
    const bool conflicts = v < 8 && lanes_shift(period / v, v) < 2 && (period / v) % 2 == 0;
    if (!conflicts && unit_elements(period, v) * (es + 1) <= kRingBytes) return kRing + cls;
    return cls == 1 && n_peers == 0 ? kTwiceClass : cls;
}

template <typename S, int V, bool FULL>
static int launch_ring(StepLaunch L, const StepRows& rows, long long max_unit, cudaStream_t stream) {
    static bool configured[kMaxDevices];
    auto kernel = step_ring_kernel<S, V, FULL>;
    constexpr int kMost = kMaxSmem - kStaticSmemSlack;
    {
        int dev = 0;
        const int rc = current_device(&dev);
        if (rc != GEFEN_B200_OK) return rc;
        std::lock_guard<std::mutex> lock(g_config_mutex);
        if (!configured[dev]) {
            GEFEN_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
            configured[dev] = true;
        }
    }
    // (a copy of n bytes from any address covers at most n + 30 bytes when it is widened to 16-byte boundaries)
    L.ring_g = static_cast<int>((max_unit * static_cast<int>(sizeof(S)) + 30) / 16 * 16);
    L.ring_codes = static_cast<int>((max_unit + 30) / 16 * 16);
    const int each = L.ring_g + L.ring_codes + static_cast<int>(sizeof(RingWarp<S>));
    // a lane's momenta of one unit: whole rounds of chunks
    L.hold_columns = static_cast<int>((max_unit + 31) / 32 + 7) / 8 * 8;
    int warps = ring_threads<S>() / 32;
    if (warps_override() > 0 && warps_override() < warps) warps = warps_override();
    if (warps > (kMost - kSmemRing) / each) warps = (kMost - kSmemRing) / each;
    if (warps > 512 / L.hold_columns * 4) warps = 512 / L.hold_columns * 4;
    if (warps < 1) return fail(GEFEN_B200_EINVAL, "internal: unit of %lld elements too large for the ring", max_unit);
    if constexpr (sizeof(S) == 4 && V == 8) {
        // The buffers of long fp32 units leave fewer warps than staged momenta do (12 against 16 for units of 2048 elements).
        // Where the units make one round of those and two of these, the staged kernel takes them: 1800 to 2300 units of
        // 2048 from HBM 19.8 to 21.2 us here, 17.3 to 18.5 there, four blocks of 512 each 21.5 to 22.3 and 19.2 to 20.7;
        // 1700 units 16.8 / 17.0, 2600 22.5 / 28.0.
        if (L.total_blocks > static_cast<long long>(sm_count()) * warps &&
            L.total_blocks <= static_cast<long long>(sm_count()) * staged_warps(stage_bytes_for(max_unit)))
            return launch_vec_variant<S, V, 0, FULL>(L, rows, max_unit, stream);
    }
    L.tmem_columns = 32;
    while (L.tmem_columns < (warps + 3) / 4 * L.hold_columns) L.tmem_columns *= 2;
    const int smem = kSmemRing + each * warps;
    // Few units: one to a CTA where the launch is alone. Eight where others of the step overlap it and want SMs of their
    // own: a GefenMuon step of four small matrices (three launches) takes 219 us so, with one unit to a CTA 231.
    const int share = L.follows || L.leads ? (warps < 8 ? warps : 8) : 1;
    return launch_step(kernel, grid_for(L.total_blocks, share, 1), warps * 32, smem, L, rows, stream);
}

template <typename S>
static int launch_vec(int cls, StepLaunch L, const StepRows& rows, long long max_unit, cudaStream_t stream) {
    switch (cls) {
        case 6: {
            constexpr int kPer = kVectorThreads / 32;
            return launch_step(step_vector_kernel<S>, static_cast<int>((L.total_blocks + kPer - 1) / kPer), kVectorThreads, kSmemWs, L, rows, stream);
        }
        case kRing + 1: return launch_ring<S, 8, true>(L, rows, max_unit, stream);
        case kRing + 2: return launch_ring<S, 8, false>(L, rows, max_unit, stream);
        case kRing + 3: return launch_ring<S, 4, false>(L, rows, max_unit, stream);
        case kRing + 4: return launch_ring<S, 2, false>(L, rows, max_unit, stream);
        case kRing + 5: return launch_ring<S, 1, false>(L, rows, max_unit, stream);
        case kTwiceClass: return launch_vec_variant<S, 8, 0, true, kTwice>(L, rows, max_unit, stream);
        case 1:
            if (L.grad_mc_delta != 0) return launch_vec_variant<S, 8, 2, true>(L, rows, max_unit, stream);
            if (L.n_grad_srcs > 0) return launch_vec_variant<S, 8, 1, true>(L, rows, max_unit, stream);
            return launch_vec_variant<S, 8, 0, true>(L, rows, max_unit, stream);
        case 2:
            if (L.grad_mc_delta != 0) return launch_vec_variant<S, 8, 2, false>(L, rows, max_unit, stream);
            if constexpr (sizeof(S) == 2)
                if (L.n_grad_srcs <= kFewSources) return launch_vec_variant<S, 8, 3, false>(L, rows, max_unit, stream);
            return launch_vec_variant<S, 8, 1, false>(L, rows, max_unit, stream);
    }
    if (L.n_peers > 0 || L.n_grad_srcs > 0) {
        if (cls == 3) return launch_vec_variant<S, 4, 1, false>(L, rows, max_unit, stream);
        if (cls == 4) return launch_vec_variant<S, 2, 1, false>(L, rows, max_unit, stream);
        return launch_vec_variant<S, 1, 1, false>(L, rows, max_unit, stream);
    }
    if (cls == 3) return launch_vec_variant<S, 4, 0, false>(L, rows, max_unit, stream);
    if (cls == 4) return launch_vec_variant<S, 2, 0, false>(L, rows, max_unit, stream);
    return launch_vec_variant<S, 1, 0, false>(L, rows, max_unit, stream);
}

template <typename S>
static int launch_generic(bool cta_per_block, const StepLaunch& L, const StepRows& rows,
                          cudaStream_t stream) {
    constexpr int smem = kSmemWs;
    static bool configured[kMaxDevices];
    {
        int dev = 0;
        const int rc = current_device(&dev);
        if (rc != GEFEN_B200_OK) return rc;
        std::lock_guard<std::mutex> lock(g_config_mutex);
        if (!configured[dev]) {
            GEFEN_CHECK_CUDA(cudaFuncSetAttribute(step_generic_kernel<S, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            GEFEN_CHECK_CUDA(cudaFuncSetAttribute(step_generic_kernel<S, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            configured[dev] = true;
        }
    }
    if (cta_per_block) {
        return launch_step(step_generic_kernel<S, 256>, grid_for(L.total_blocks, 1, 3), kThreads, smem, L, rows, stream);
    }
    return launch_step(step_generic_kernel<S, 32>, grid_for(L.total_blocks, kWarps, 3), kThreads, smem, L, rows, stream);
}

// Class of a tensor: 1 = fast path in chunks of eight with whole-warp blocks, 2 = the same with several blocks
// per warp pass (blocks of up to 1024 elements), 3 / 4 / 5 = fast path in chunks of four, two, one (the most that
// divides the block length and the alignment of all pointers), 6 = vectors (period 1, runs of up to 256 elements), 0 =
// generic warp per block, -1 = generic CTA per block.
static int generic_class(const gefen_b200_step_tensor_t& t) { return t.period > 2048 ? -1 : 0; }
static int class_chunk(int cls) {
    cls &= kRing - 1;
    return cls <= 2 || cls == kTwiceClass ? 8 : (cls == 3 ? 4 : (cls == 4 ? 2 : 1));
}
static bool staged_class(int cls) { return cls >= 1 && cls != 6; }
static int tensor_class(const gefen_b200_step_tensor_t& t, int dtype) {
    const bool vec_dtype = dtype == GEFEN_B200_F32 || dtype == GEFEN_B200_BF16 || dtype == GEFEN_B200_F16;
    if (vec_dtype && (t.flags & GEFEN_B200_STEP_PERIOD1) != 0 && t.period <= kVectorMost && t.num_blocks < (1 << 28)) return 6;
    if (!vec_dtype || (t.flags & (GEFEN_B200_STEP_PERIOD1 | GEFEN_B200_STEP_PACKED)) != 0 || t.period > kFastMaxPeriod) return generic_class(t);
    const uintptr_t ptrs = reinterpret_cast<uintptr_t>(t.g) | reinterpret_cast<uintptr_t>(t.p);
    for (int cls = 2; cls <= 5; ++cls) {
        const int v = class_chunk(cls);
        const uintptr_t bytes = static_cast<uintptr_t>(v * dtype_size(dtype) < 16 ? v * dtype_size(dtype) : 16);
        if (t.period % v != 0 || ptrs % bytes != 0 || reinterpret_cast<uintptr_t>(t.codes) % v != 0) continue;
        return cls == 2 && lanes_shift(t.period / 8, 8) == 5 ? 1 : cls;
    }
    return generic_class(t);   // (a pointer that is not aligned to its own type)
}
// Units of a tensor in its launch's index space: passes of a warp on the fast path, blocks elsewhere.
// (4-bit codes with an odd period: a pair of blocks is one unit, see step_generic_kernel)
// (sources: see deep_lanes)
static long long class_units(const gefen_b200_step_tensor_t& t, int cls, int dtype, int sources) {
    if (staged_class(cls)) return vec_units(t.num_blocks, t.period, class_chunk(cls), dtype_size(dtype), sources);
    const bool paired = (t.flags & GEFEN_B200_STEP_PACKED) != 0 && (t.period & 1) != 0;
    return paired ? (t.num_blocks + 1) / 2 : t.num_blocks;
}

static int launch_class(int cls, int dtype, const StepLaunch& L, const StepRows& rows,
                        long long max_unit, cudaStream_t stream) {
    if (cls >= 1) {
        if (dtype == GEFEN_B200_BF16) return launch_vec<__nv_bfloat16>(cls, L, rows, max_unit, stream);
        if (dtype == GEFEN_B200_F16) return launch_vec<__half>(cls, L, rows, max_unit, stream);
        return launch_vec<float>(cls, L, rows, max_unit, stream);
    }
    const bool cta = cls < 0;
    switch (dtype) {
        case GEFEN_B200_F32: return launch_generic<float>(cta, L, rows, stream);
        case GEFEN_B200_F16: return launch_generic<__half>(cta, L, rows, stream);
        case GEFEN_B200_BF16: return launch_generic<__nv_bfloat16>(cta, L, rows, stream);
        case GEFEN_B200_F64: return launch_generic<double>(cta, L, rows, stream);
    }
    return fail(GEFEN_B200_EINVAL, "Unsupported parameter dtype tag %d.", dtype);
}

static int check_common(const void* g, uint8_t* codes, void* mag, int mag_dtype, int param_dtype,
                        int packed_indices, long long num_blocks, long long period) {
    GEFEN_CHECK_ARG(g != nullptr && codes != nullptr && mag != nullptr, "Expected non-null tensor pointers.");
    GEFEN_CHECK_ARG(is_float_dtype(param_dtype), "Unsupported parameter/gradient dtype tag %d.", param_dtype);
    GEFEN_CHECK_ARG(is_state_dtype(mag_dtype),
                    "Expected m_magnitude to have dtype float32, float16, or bfloat16.");
    GEFEN_CHECK_ARG(num_blocks >= 0 && period > 0, "Expected a positive period and a non-negative block count.");
    GEFEN_CHECK_ARG(period <= 0x7FFFFFFFLL, "Period %lld is too large.", period);
    (void)packed_indices;   // any period: with an odd one, pairs of blocks share a byte and are stepped together
    return GEFEN_B200_OK;
}

static int run_single(gefen_b200_step_tensor_t& t, int param_dtype, const float* stepsize, const float* codebook,
                      int codebook_size, const void* codebook_ws, cudaStream_t stream) {
    if (t.num_blocks == 0) return GEFEN_B200_OK;
    const void* ws = nullptr;
    const int rc = resolve_codebook_ws(codebook, codebook_size, codebook_ws, stream, &ws);
    if (rc != GEFEN_B200_OK) return rc;
    t.first_block = 0;
    StepLaunch L;
    L.table = nullptr;
    L.n_tensors = 1;
    L.stage_floats = 0;
    const int cls = route(tensor_class(t, param_dtype), t.period, param_dtype, 0, 0);
    L.total_blocks = class_units(t, cls, param_dtype, 0);
    L.ws = static_cast<const unsigned char*>(ws);
    L.stepsize = stepsize;
    L.n_peers = 0;
    L.n_grad_srcs = 0;
    L.grad_scale = 1.0f;
    L.grad_mc_delta = 0;
    L.param_mc_delta = 0;
    L.spin_limit = g_stage_spin_limit;
    L.input_limit = g_input_spin_limit;
    L.follows = L.leads = 0;
    StepRows rows = {};
    rows.row[0] = t;
    return launch_class(cls, param_dtype, L, rows, staged_class(cls) ? unit_floats(t.period, class_chunk(cls), dtype_size(param_dtype), 0) : t.period, stream);
}

}  // namespace gefen

using namespace gefen;

extern "C" {

int gefen_b200_automatic_vmean_update(void* vmean, int vmean_dtype, const void* grad_view, int grad_dtype,
                                      int64_t num_blocks, int64_t period, double beta2, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(vmean != nullptr && grad_view != nullptr, "Expected non-null vmean and grad_view.");
    GEFEN_CHECK_ARG(is_state_dtype(vmean_dtype), "Expected vmean to have dtype float32, float16, or bfloat16.");
    GEFEN_CHECK_ARG(is_float_dtype(grad_dtype), "Unsupported gradient dtype tag %d.", grad_dtype);
    GEFEN_CHECK_ARG(period > 0, "Expected grad_view to have a positive period.");
    GEFEN_CHECK_ARG(num_blocks >= 0, "Expected a non-negative block count.");
    if (num_blocks == 0) return GEFEN_B200_OK;
    const int grid = grid_for(num_blocks, kWarps, 8);
    const float b2 = static_cast<float>(beta2);
    switch (grad_dtype) {
        case GEFEN_B200_F32:
            vmean_kernel<float><<<grid, kThreads, 0, stream>>>(vmean, vmean_dtype, static_cast<const float*>(grad_view), num_blocks, period, b2);
            break;
        case GEFEN_B200_F16:
            vmean_kernel<__half><<<grid, kThreads, 0, stream>>>(vmean, vmean_dtype, static_cast<const __half*>(grad_view), num_blocks, period, b2);
            break;
        case GEFEN_B200_BF16:
            vmean_kernel<__nv_bfloat16><<<grid, kThreads, 0, stream>>>(vmean, vmean_dtype, static_cast<const __nv_bfloat16*>(grad_view), num_blocks, period, b2);
            break;
        default:
            vmean_kernel<double><<<grid, kThreads, 0, stream>>>(vmean, vmean_dtype, static_cast<const double*>(grad_view), num_blocks, period, b2);
            break;
    }
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

int gefen_b200_automatic_gefen_fused_update_from_vmean(
    void* p, const void* grad_view, int param_dtype, uint8_t* m_sign, void* m_magnitude, int magnitude_dtype,
    const void* vmean, int vmean_dtype, const float* codebook, int codebook_size, const void* codebook_ws,
    int packed_indices, int64_t num_blocks, int64_t period, double beta1, double lr, double bias_correction_1,
    double bias_correction_2, double eps, void* stream) {
    int rc = check_common(grad_view, m_sign, m_magnitude, magnitude_dtype, param_dtype, packed_indices, num_blocks, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(p != nullptr && vmean != nullptr, "Expected non-null p and vmean.");
    GEFEN_CHECK_ARG(is_state_dtype(vmean_dtype), "Expected vmean to have dtype float32, float16, or bfloat16.");
    GEFEN_CHECK_ARG(bias_correction_1 > 0.0, "Expected bias_correction_1 to be positive.");
    GEFEN_CHECK_ARG(bias_correction_2 > 0.0, "Expected bias_correction_2 to be positive.");
    GEFEN_CHECK_ARG(eps >= 0.0, "Expected eps to be non-negative.");
    gefen_b200_step_tensor_t t = {};
    t.p = p; t.g = grad_view; t.codes = m_sign; t.mag = m_magnitude; t.v = const_cast<void*>(vmean);
    t.num_blocks = num_blocks; t.period = period;
    t.beta1 = static_cast<float>(beta1); t.lr = static_cast<float>(lr);
    t.bc1 = static_cast<float>(bias_correction_1); t.bc2 = static_cast<float>(bias_correction_2);
    t.eps = static_cast<float>(eps); t.wd_mul = 1.0f; t.flags = packed_indices ? GEFEN_B200_STEP_PACKED : 0u;
    t.mag_dtype = magnitude_dtype; t.v_dtype = vmean_dtype;
    return run_single(t, param_dtype, nullptr, codebook, codebook_size, codebook_ws, static_cast<cudaStream_t>(stream));
}

int gefen_b200_automatic_gefen_fused_update(
    void* p, const void* grad_view, int param_dtype, uint8_t* m_sign, void* m_magnitude, int magnitude_dtype,
    const float* stepsize, const float* codebook, int codebook_size, const void* codebook_ws, int packed_indices,
    int64_t num_blocks, int64_t period, double beta1, double lr, void* stream) {
    int rc = check_common(grad_view, m_sign, m_magnitude, magnitude_dtype, param_dtype, packed_indices, num_blocks, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(p != nullptr && stepsize != nullptr, "Expected non-null p and stepsize.");
    gefen_b200_step_tensor_t t = {};
    t.p = p; t.g = grad_view; t.codes = m_sign; t.mag = m_magnitude; t.v = nullptr;
    t.num_blocks = num_blocks; t.period = period;
    t.beta1 = static_cast<float>(beta1); t.lr = static_cast<float>(lr);
    t.bc1 = 1.0f; t.bc2 = 1.0f; t.eps = 0.0f; t.wd_mul = 1.0f; t.flags = packed_indices ? GEFEN_B200_STEP_PACKED : 0u;
    t.mag_dtype = magnitude_dtype; t.v_dtype = GEFEN_B200_F32;
    return run_single(t, param_dtype, stepsize, codebook, codebook_size, codebook_ws, static_cast<cudaStream_t>(stream));
}

int gefen_b200_automatic_gefen_period1_update(
    void* p, const void* grad_flat, int param_dtype, uint8_t* m_sign, void* m_magnitude, int magnitude_dtype,
    void* vmean, int vmean_dtype, const float* codebook, int codebook_size, const void* codebook_ws,
    int64_t total_numel, int64_t period_one_divisor, double beta1, double beta2, double lr,
    double bias_correction_1, double bias_correction_2, double eps, void* stream) {
    GEFEN_CHECK_ARG(period_one_divisor > 0, "Expected period_one_divisor to be positive.");
    GEFEN_CHECK_ARG(total_numel >= 0 && total_numel % period_one_divisor == 0,
                    "Expected period_one_divisor to divide total_numel.");
    const int64_t num_blocks = total_numel / period_one_divisor;
    int rc = check_common(grad_flat, m_sign, m_magnitude, magnitude_dtype, param_dtype, 0, num_blocks, period_one_divisor);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(p != nullptr && vmean != nullptr, "Expected non-null p and vmean.");
    GEFEN_CHECK_ARG(is_state_dtype(vmean_dtype), "Expected vmean to have dtype float32, float16, or bfloat16.");
    GEFEN_CHECK_ARG(bias_correction_1 > 0.0, "Expected bias_correction_1 to be positive.");
    GEFEN_CHECK_ARG(bias_correction_2 > 0.0, "Expected bias_correction_2 to be positive.");
    GEFEN_CHECK_ARG(eps >= 0.0, "Expected eps to be non-negative.");
    gefen_b200_step_tensor_t t = {};
    t.p = p; t.g = grad_flat; t.codes = m_sign; t.mag = m_magnitude; t.v = vmean;
    t.num_blocks = num_blocks; t.period = period_one_divisor;
    t.beta1 = static_cast<float>(beta1); t.beta2 = static_cast<float>(beta2); t.lr = static_cast<float>(lr);
    t.bc1 = static_cast<float>(bias_correction_1); t.bc2 = static_cast<float>(bias_correction_2);
    t.eps = static_cast<float>(eps); t.wd_mul = 1.0f; t.flags = GEFEN_B200_STEP_PERIOD1;
    t.mag_dtype = magnitude_dtype; t.v_dtype = vmean_dtype;
    return run_single(t, param_dtype, nullptr, codebook, codebook_size, codebook_ws, static_cast<cudaStream_t>(stream));
}

int gefen_b200_automatic_gefen_step(
    void* p, const void* grad, int param_dtype, uint8_t* m_sign, void* m_magnitude, int magnitude_dtype, void* vmean,
    int vmean_dtype, const float* codebook, int codebook_size, const void* codebook_ws, int64_t num_blocks, int64_t period,
    int period_one, double beta1, double beta2, double lr, double weight_decay_mul, double bias_correction_1,
    double bias_correction_2, double eps, void* stream) {
    int rc = check_common(grad, m_sign, m_magnitude, magnitude_dtype, param_dtype, 0, num_blocks, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(p != nullptr && vmean != nullptr, "Expected non-null p and vmean.");
    GEFEN_CHECK_ARG(is_state_dtype(vmean_dtype), "Expected vmean to have dtype float32, float16, or bfloat16.");
    GEFEN_CHECK_ARG(bias_correction_1 > 0.0, "Expected bias_correction_1 to be positive.");
    GEFEN_CHECK_ARG(bias_correction_2 > 0.0, "Expected bias_correction_2 to be positive.");
    GEFEN_CHECK_ARG(eps >= 0.0, "Expected eps to be non-negative.");
    gefen_b200_step_tensor_t t = {};
    t.p = p; t.g = grad; t.codes = m_sign; t.mag = m_magnitude; t.v = vmean;
    t.num_blocks = num_blocks; t.period = period;
    t.beta1 = static_cast<float>(beta1); t.beta2 = static_cast<float>(beta2); t.lr = static_cast<float>(lr);
    t.bc1 = static_cast<float>(bias_correction_1); t.bc2 = static_cast<float>(bias_correction_2);
    t.eps = static_cast<float>(eps); t.wd_mul = static_cast<float>(weight_decay_mul);
    t.flags = (period_one ? GEFEN_B200_STEP_PERIOD1 : GEFEN_B200_STEP_FUSE_VMEAN) | (weight_decay_mul != 1.0 ? GEFEN_B200_STEP_WEIGHT_DECAY : 0u);
    t.mag_dtype = magnitude_dtype; t.v_dtype = vmean_dtype;
    return run_single(t, param_dtype, nullptr, codebook, codebook_size, codebook_ws, static_cast<cudaStream_t>(stream));
}

int gefen_b200_automatic_gefen_muon_momentum(
    const void* grad_view, int grad_dtype, uint8_t* m_sign, void* m_magnitude, int magnitude_dtype,
    const float* codebook, int codebook_size, const void* codebook_ws, void* momentum_update, int packed_indices,
    int64_t num_blocks, int64_t period, double beta1, void* stream) {
    int rc = check_common(grad_view, m_sign, m_magnitude, magnitude_dtype, grad_dtype, packed_indices, num_blocks, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(momentum_update != nullptr, "Expected a non-null momentum_update.");
    gefen_b200_step_tensor_t t = {};
    t.p = momentum_update; t.g = grad_view; t.codes = m_sign; t.mag = m_magnitude; t.v = nullptr;
    t.num_blocks = num_blocks; t.period = period;
    t.beta1 = static_cast<float>(beta1); t.lr = 0.0f; t.bc1 = 1.0f; t.bc2 = 1.0f; t.wd_mul = 1.0f;
    t.flags = GEFEN_B200_STEP_MUON | (packed_indices ? GEFEN_B200_STEP_PACKED : 0u);
    t.mag_dtype = magnitude_dtype; t.v_dtype = GEFEN_B200_F32;
    return run_single(t, grad_dtype, nullptr, codebook, codebook_size, codebook_ws, static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------------------------
// The same step for callers that must not allocate device memory.
//
// Who needs it: code that runs after all device memory has been handed to another owner (a
// framework's caching allocator holding the whole card, a fixed memory plan of an inference or
// training runtime), and code on paths where an allocation is simply not allowed to happen
// (latency-critical loops, library hooks that promise not to touch the allocator). The regular
// entry point, when it is given no codebook workspace, allocates one per device with cudaMalloc on
// first use; this one keeps that workspace in a fixed array inside the library image instead.
//
// The array costs GEFEN_B200_CODEBOOK_WS_BYTES (34 848 bytes) of device memory on every GPU that
// loads the library, until the process exits. It is sized for the largest codebook the kernels
// accept, 256 entries; a larger codebook is rejected. Every call rewrites the whole array from the
// codebook it is given, on the caller's stream, before the step kernel reads it, so nothing has to
// be cleared and consecutive calls on one stream are independent; calls that may run concurrently
// on the same GPU (different streams) share the array and would race on it.
static __device__ __align__(256) unsigned char g_static_codebook_ws[GEFEN_B200_CODEBOOK_WS_BYTES];

// In host code the array's name is only a handle: the device address comes from the runtime, once
// per device, with that device current.
static std::mutex g_static_ws_mutex;
static void* g_static_ws_address[kMaxDevices];

static int static_codebook_ws(void** out) {
    int dev = 0;
    const int rc_dev = current_device(&dev);
    if (rc_dev != GEFEN_B200_OK) return rc_dev;
    std::lock_guard<std::mutex> lock(g_static_ws_mutex);
    if (g_static_ws_address[dev] == nullptr) {
        void* address = nullptr;
        GEFEN_CHECK_CUDA(cudaGetSymbolAddress(&address, g_static_codebook_ws));
        g_static_ws_address[dev] = address;
    }
    *out = g_static_ws_address[dev];
    return GEFEN_B200_OK;
}

int gefen_b200_automatic_gefen_fused_update_from_vmean_static_ws(
    void* p, const void* grad_view, int param_dtype, uint8_t* m_sign, void* m_magnitude, int magnitude_dtype,
    const void* vmean, int vmean_dtype, const float* codebook, int codebook_size, int packed_indices,
    int64_t num_blocks, int64_t period, double beta1, double lr, double bias_correction_1,
    double bias_correction_2, double eps, void* stream) {
    GEFEN_CHECK_ARG(codebook != nullptr, "Expected a codebook pointer.");
    GEFEN_CHECK_ARG(codebook_size >= 1 && codebook_size <= kMaxCodebook,
                    "The built-in workspace holds tables for at most 256 codebook entries, got %d.", codebook_size);
    // every argument is checked before the shared array is touched: a refused call leaves it as it was
    int rc = check_common(grad_view, m_sign, m_magnitude, magnitude_dtype, param_dtype, packed_indices, num_blocks, period);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(p != nullptr && vmean != nullptr, "Expected non-null p and vmean.");
    GEFEN_CHECK_ARG(is_state_dtype(vmean_dtype), "Expected vmean to have dtype float32, float16, or bfloat16.");
    GEFEN_CHECK_ARG(bias_correction_1 > 0.0, "Expected bias_correction_1 to be positive.");
    GEFEN_CHECK_ARG(bias_correction_2 > 0.0, "Expected bias_correction_2 to be positive.");
    GEFEN_CHECK_ARG(eps >= 0.0, "Expected eps to be non-negative.");
    if (num_blocks == 0) return GEFEN_B200_OK;
    void* ws = nullptr;
    rc = static_codebook_ws(&ws);
    if (rc != GEFEN_B200_OK) return rc;
    rc = launch_codebook_prepare(codebook, codebook_size, ws, static_cast<cudaStream_t>(stream));
    if (rc != GEFEN_B200_OK) return rc;
    return gefen_b200_automatic_gefen_fused_update_from_vmean(
        p, grad_view, param_dtype, m_sign, m_magnitude, magnitude_dtype, vmean, vmean_dtype, codebook, codebook_size,
        ws, packed_indices, num_blocks, period, beta1, lr, bias_correction_1, bias_correction_2, eps, stream);
}

int gefen_b200_step_tensor_size(void) { return static_cast<int>(sizeof(gefen_b200_step_tensor_t)); }

int gefen_b200_step_tensor_class(const gefen_b200_step_tensor_t* host_entry, int param_dtype) {
    if (host_entry == nullptr) return -2;
    const int cls = tensor_class(*host_entry, param_dtype);
    return cls >= 3 ? generic_class(*host_entry) : cls;
}

int gefen_b200_step_launch_class(const gefen_b200_step_tensor_t* host_entry, int param_dtype) {
    if (host_entry == nullptr) return -2;
    return tensor_class(*host_entry, param_dtype);
}

int gefen_b200_step_classes(const gefen_b200_step_tensor_t* host_table, int n_tensors, int param_dtype, int32_t* tensor_classes,
                            int32_t* launch_classes) {
    GEFEN_CHECK_ARG(n_tensors >= 0 && (n_tensors == 0 || host_table != nullptr), "Expected a table of %d rows.", n_tensors);
    for (int i = 0; i < n_tensors; ++i) {
        const int cls = tensor_class(host_table[i], param_dtype);
        if (launch_classes != nullptr) launch_classes[i] = cls;
        if (tensor_classes != nullptr) tensor_classes[i] = cls >= 3 ? generic_class(host_table[i]) : cls;
    }
    return GEFEN_B200_OK;
}

int gefen_b200_multicast_sum(void* dst, const void* src_multicast, int dtype, int64_t numel, double scale, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(dst != nullptr && src_multicast != nullptr, "Expected non-null buffers.");
    GEFEN_CHECK_ARG(dtype == GEFEN_B200_F32 || dtype == GEFEN_B200_F16 || dtype == GEFEN_B200_BF16,
                    "The multicast sum supports fp32, fp16 and bf16.");
    GEFEN_CHECK_ARG(numel >= 0 && numel % 8 == 0 && aligned16(dst) && aligned16(src_multicast),
                    "Expected 16-byte aligned buffers and a multiple of 8 elements.");
    if (numel == 0) return GEFEN_B200_OK;
    const long long chunks = numel / 8;
    const int grid = grid_for(chunks, kThreads, 4);
    const float sc = static_cast<float>(scale);
    if (dtype == GEFEN_B200_BF16) multicast_sum_kernel<__nv_bfloat16><<<grid, kThreads, 0, stream>>>(dst, src_multicast, chunks, sc);
    else if (dtype == GEFEN_B200_F16) multicast_sum_kernel<__half><<<grid, kThreads, 0, stream>>>(dst, src_multicast, chunks, sc);
    else multicast_sum_kernel<float><<<grid, kThreads, 0, stream>>>(dst, src_multicast, chunks, sc);
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

int gefen_b200_muon_apply(void* p, const void* update, int dtype, int64_t numel, double wd_mul, double alpha,
                          const int64_t* peer_deltas, int n_peers, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(p != nullptr && update != nullptr, "Expected non-null p and update.");
    GEFEN_CHECK_ARG(dtype == GEFEN_B200_F32 || dtype == GEFEN_B200_F16 || dtype == GEFEN_B200_BF16,
                    "The GefenMuon apply supports fp32, fp16 and bf16 parameters.");
    GEFEN_CHECK_ARG(numel >= 0, "Expected a non-negative element count.");
    GEFEN_CHECK_ARG(n_peers >= 0 && n_peers <= GEFEN_B200_MAX_PEERS, "Expected between 0 and %d peers, got %d.",
                    GEFEN_B200_MAX_PEERS, n_peers);
    GEFEN_CHECK_ARG(n_peers == 0 || peer_deltas != nullptr, "Expected peer offsets for %d peers.", n_peers);
    for (int r = 0; r < n_peers; ++r)
        GEFEN_CHECK_ARG(peer_deltas[r] % 16 == 0, "Peer offset %d is not a multiple of 16 bytes.", r);
    if (numel == 0) return GEFEN_B200_OK;
    StepLaunch L = {};
    L.n_peers = n_peers;
    for (int r = 0; r < n_peers; ++r) L.peer_delta[r] = peer_deltas[r];
    const bool vec = aligned16(p) && aligned16(update);
    const bool decay = wd_mul != 1.0;
    const int grid = grid_for((numel + 7) / 8, kThreads, 8);
    const float wm = static_cast<float>(wd_mul), a = static_cast<float>(alpha);
    if (dtype == GEFEN_B200_BF16)
        muon_apply_kernel<__nv_bfloat16><<<grid, kThreads, 0, stream>>>(static_cast<__nv_bfloat16*>(p), static_cast<const __nv_bfloat16*>(update), numel, wm, decay, a, vec, L);
    else if (dtype == GEFEN_B200_F16)
        muon_apply_kernel<__half><<<grid, kThreads, 0, stream>>>(static_cast<__half*>(p), static_cast<const __half*>(update), numel, wm, decay, a, vec, L);
    else
        muon_apply_kernel<float><<<grid, kThreads, 0, stream>>>(static_cast<float*>(p), static_cast<const float*>(update), numel, wm, decay, a, vec, L);
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

int gefen_b200_step_status(int* host_status, int clear) {
    GEFEN_CHECK_ARG(host_status != nullptr, "Expected a host pointer for the status.");
    int value = 0;
    GEFEN_CHECK_CUDA(cudaMemcpyFromSymbol(&value, g_step_status, sizeof(int)));   // synchronises the device
    if (value != 0 && clear) {
        const int zero = 0;
        GEFEN_CHECK_CUDA(cudaMemcpyToSymbol(g_step_status, &zero, sizeof(int)));
    }
    *host_status = value;
    return GEFEN_B200_OK;
}

int gefen_b200_debug_set_stage_spin_limit(int64_t limit) {
    g_stage_spin_limit = spin_limit_of(limit);
    return GEFEN_B200_OK;
}

int gefen_b200_debug_set_input_spin_limit(int64_t limit) {
    g_input_spin_limit = spin_limit_of(limit);
    return GEFEN_B200_OK;
}

int gefen_b200_multi_tensor_step(gefen_b200_step_tensor_t* host_table, void* device_table, int n_tensors,
                                 int param_dtype, const void* codebook_ws, void* stream_) {
    return gefen_b200_multi_tensor_step_peers(host_table, device_table, n_tensors, param_dtype, codebook_ws, nullptr, 0,
                                              nullptr, 0, 1.0, stream_);
}

int gefen_b200_multi_tensor_step_peers(gefen_b200_step_tensor_t* host_table, void* device_table, int n_tensors,
                                       int param_dtype, const void* codebook_ws, const int64_t* peer_deltas,
                                       int n_peers, const int64_t* grad_deltas, int n_grad_srcs, double grad_scale,
                                       void* stream_) {
    return gefen_b200_multi_tensor_step_multicast(host_table, device_table, n_tensors, param_dtype, codebook_ws, peer_deltas,
                                                  n_peers, grad_deltas, n_grad_srcs, grad_scale, 0, 0, stream_);
}

int gefen_b200_multi_tensor_step_multicast(gefen_b200_step_tensor_t* host_table, void* device_table, int n_tensors,
                                           int param_dtype, const void* codebook_ws, const int64_t* peer_deltas,
                                           int n_peers, const int64_t* grad_deltas, int n_grad_srcs, double grad_scale,
                                           int64_t param_multicast_delta, int64_t grad_multicast_delta, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(param_multicast_delta % 16 == 0 && grad_multicast_delta % 16 == 0,
                    "Multicast offsets must be multiples of 16 bytes.");
    GEFEN_CHECK_ARG(grad_multicast_delta == 0 || n_grad_srcs > 0,
                    "Summing gradients through the multicast mapping also needs the per-rank gradient offsets "
                    "(the kernels for short or odd blocks read the ranks' buffers directly).");
    GEFEN_CHECK_ARG(param_multicast_delta == 0 || n_peers > 0,
                    "Storing parameters through the multicast mapping also needs the per-rank parameter offsets.");
    GEFEN_CHECK_ARG((param_multicast_delta == 0 && grad_multicast_delta == 0) || param_dtype != GEFEN_B200_F64,
                    "The multicast paths support fp32, fp16 and bf16.");
    GEFEN_CHECK_ARG(n_grad_srcs >= 0 && n_grad_srcs <= GEFEN_B200_MAX_PEERS + 1,
                    "Expected between 0 and %d gradient buffers, got %d.", GEFEN_B200_MAX_PEERS + 1, n_grad_srcs);
    GEFEN_CHECK_ARG(n_grad_srcs == 0 || grad_deltas != nullptr, "Expected offsets for %d gradient buffers.", n_grad_srcs);
    for (int r = 0; r < n_grad_srcs; ++r)
        GEFEN_CHECK_ARG(grad_deltas[r] % 16 == 0, "Gradient buffer offset %d is not a multiple of 16 bytes.", r);
    GEFEN_CHECK_ARG(n_grad_srcs == 0 || param_dtype != GEFEN_B200_F64, "Gradient averaging supports fp32, fp16 and bf16.");
    GEFEN_CHECK_ARG(n_peers >= 0 && n_peers <= GEFEN_B200_MAX_PEERS, "Expected between 0 and %d peers, got %d.",
                    GEFEN_B200_MAX_PEERS, n_peers);
    GEFEN_CHECK_ARG(n_peers == 0 || peer_deltas != nullptr, "Expected peer offsets for %d peers.", n_peers);
    for (int r = 0; r < n_peers; ++r)
        GEFEN_CHECK_ARG(peer_deltas[r] % 16 == 0, "Peer offset %d is not a multiple of 16 bytes.", r);
    GEFEN_CHECK_ARG(n_tensors >= 0, "Expected a non-negative tensor count.");
    if (n_tensors == 0) return GEFEN_B200_OK;
    GEFEN_CHECK_ARG(host_table != nullptr && device_table != nullptr && codebook_ws != nullptr,
                    "Expected non-null tables and codebook workspace.");
    GEFEN_CHECK_ARG(aligned16(codebook_ws) && aligned16(device_table), "Expected 16-byte aligned workspace and table.");
    GEFEN_CHECK_ARG(is_float_dtype(param_dtype), "Unsupported parameter dtype tag %d.", param_dtype);
    // Tensors are launched in maximal runs of rows that share a kernel class (staged vector path,
    // generic warp, generic CTA); callers that keep equal classes adjacent get one launch per
    // class. Rows are never reordered.
    for (int i = 0; i < n_tensors; ++i) {
        gefen_b200_step_tensor_t& t = host_table[i];
        GEFEN_CHECK_ARG(t.g != nullptr && t.codes != nullptr && t.mag != nullptr && t.p != nullptr,
                        "Tensor %d of the table has a null pointer.", i);
        GEFEN_CHECK_ARG(t.period > 0 && t.period <= 0x7FFFFFFFLL && t.num_blocks >= 0,
                        "Tensor %d of the table has a bad period or block count.", i);
        GEFEN_CHECK_ARG(is_state_dtype(t.mag_dtype) && is_state_dtype(t.v_dtype),
                        "Tensor %d of the table has a bad state dtype.", i);
        GEFEN_CHECK_ARG((t.flags & GEFEN_B200_STEP_MUON) || t.v != nullptr, "Tensor %d has a null vmean.", i);
        GEFEN_CHECK_ARG(!(t.flags & GEFEN_B200_STEP_PACKED) || !(t.flags & GEFEN_B200_STEP_PERIOD1),
                        "Tensor %d: 4-bit codes are not defined for period-1 tensors.", i);
        GEFEN_CHECK_ARG(n_grad_srcs == 0 || !(t.flags & GEFEN_B200_STEP_MUON),
                        "Tensor %d: the momentum-only step does not average gradients over ranks.", i);
        int cls = tensor_class(t, param_dtype);
        // vectors with peers: the generic kernel (no sums of squares there, so the results are the same bits)
        if (cls == 6 && (n_peers > 0 || n_grad_srcs > 0)) cls = generic_class(t);
        t.reserved_[0] = route(cls, t.period, param_dtype, n_peers, n_grad_srcs);
    }
    const int sources = grad_multicast_delta != 0 ? 1 : n_grad_srcs;   // (chunk_sources)
    int last_run = 0;   // the first row of the last run with anything to do
    for (int begin = 0; begin < n_tensors;) {
        int end = begin;
        long long first = 0;
        while (end < n_tensors && host_table[end].reserved_[0] == host_table[begin].reserved_[0]) {
            host_table[end].first_block = first;   // in work units on the fast path, in blocks elsewhere
            first += class_units(host_table[end], host_table[end].reserved_[0], param_dtype, sources);
            ++end;
        }
        host_table[begin].reserved_[1] = end - begin;  // run length, read back below
        if (first > 0) last_run = begin;
        begin = end;
    }
    // Few tensors: their descriptors go with the launches. Not while the stream is being captured: a replay of the graph
    // reads the host table again, as it did before.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    GEFEN_CHECK_CUDA(cudaStreamIsCapturing(stream, &capture));
    const bool in_params = n_tensors <= kParamRows && capture == cudaStreamCaptureStatusNone;
    if (!in_params)
        GEFEN_CHECK_CUDA(cudaMemcpyAsync(device_table, host_table, sizeof(gefen_b200_step_tensor_t) * n_tensors,
                                         cudaMemcpyHostToDevice, stream));
    StepRows rows = {};
    bool launched = false;
    for (int begin = 0; begin < n_tensors;) {
        const int run = host_table[begin].reserved_[1];
        const gefen_b200_step_tensor_t& last = host_table[begin + run - 1];
        const long long total = last.first_block + class_units(last, last.reserved_[0], param_dtype, sources);
        long long max_period = 0;   // largest need of a warp: the elements of one unit on the fast path
        for (int i = begin; i < begin + run; ++i) {
            const int cls = host_table[begin].reserved_[0];
            const long long need = staged_class(cls) ? unit_floats(host_table[i].period, class_chunk(cls), dtype_size(param_dtype), sources) : host_table[i].period;
            max_period = need > max_period ? need : max_period;
        }
        if (total > 0) {
            StepLaunch L;
            L.table = in_params ? nullptr : static_cast<const gefen_b200_step_tensor_t*>(device_table) + begin;
            if (in_params) memcpy(rows.row, host_table + begin, sizeof(gefen_b200_step_tensor_t) * run);
            L.n_tensors = run;
            L.stage_floats = 0;
            L.total_blocks = total;
            L.ws = static_cast<const unsigned char*>(codebook_ws);
            L.stepsize = nullptr;
            L.n_peers = n_peers;
            for (int r = 0; r < n_peers; ++r) L.peer_delta[r] = peer_deltas[r];
            L.n_grad_srcs = n_grad_srcs;
            L.grad_scale = static_cast<float>(grad_scale);
            for (int r = 0; r < n_grad_srcs; ++r) L.grad_delta[r] = grad_deltas[r];
            L.grad_mc_delta = grad_multicast_delta;
            L.param_mc_delta = param_multicast_delta;
            L.spin_limit = g_stage_spin_limit;
            L.input_limit = g_input_spin_limit;
            L.follows = launched && n_peers == 0 && n_grad_srcs == 0;
            L.leads = begin < last_run && n_peers == 0 && n_grad_srcs == 0;
            launched = true;
            const int rc = launch_class(host_table[begin].reserved_[0], param_dtype, L, rows, max_period, stream);
            if (rc != GEFEN_B200_OK) return rc;
        }
        begin += run;
    }
    return GEFEN_B200_OK;
}

}  // extern "C"
