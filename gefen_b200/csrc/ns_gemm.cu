// bf16 GEMM on the 5th-generation tensor cores for GefenMuon's Newton-Schulz iteration
// (reference: gefen_muon.py:16-51, where the three products per iteration are torch.addmm / `@`,
// i.e. cuBLAS):
//
//     D[M,N] = alpha * A[M,K] * B[N,K]^T + beta * C[M,N]        (bf16 in/out, fp32 accumulation)
//
// and optionally Dt[N,M] = D^T in the same pass. Both operands are K-major (row-major with K
// contiguous), which covers every product of the iteration once X and X^T are both kept:
//     G  = X X^T               A = B = X
//     Bm = b*G + c*G*G         A = B = C = G      (G is symmetric, so G*G = G*G^T)
//     X' = a*X + Bm*X          A = Bm, B = X^T, C = X, Dt receives X'^T for the next iteration
//
// Structure (128 x BN output tiles, 6 warps; one tile per CTA, or - PERSIST - one CTA per SM that
// walks over tiles with two accumulator buffers in TMEM, so that the epilogue of a tile runs while
// the tensor cores already work on the next one):
//   warp 4  : TMA producer. cp.async.bulk.tensor 2-D loads of 128x64 (A) and BNx64 (B) bf16 boxes,
//             128-byte swizzle, into a STAGES-deep shared-memory ring, completion on mbarriers.
//   warp 5  : allocates TMEM and issues tcgen05.mma (cta_group::1, kind::f16, M=128, N=BN, K=16)
//             from one thread; tcgen05.commit releases ring slots and finally signals the epilogue.
//   warps 0-3: epilogue. tcgen05.ld of the fp32 accumulators (lane = row), alpha/beta, bf16 stores.
// Every mbarrier wait is bounded: on a time-out the CTA raises a flag in global memory, the
// roles drain, TMEM is released and the kernel returns.
#include "common.cuh"

#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <cuda.h>
#include <algorithm>
#include <mutex>
#include <new>
#include <vector>

namespace gefen {

constexpr int kBM = 128;
constexpr int kBK = 64;                 // 64 bf16 = one 128-byte swizzle row
constexpr int kGemmThreads = 192;
constexpr uint32_t kSpinLimit = 20000000u;

// One product of a group (see ns_group below): its operands' tensor maps and its matrices.
struct alignas(64) GroupEntry {
    CUtensorMap a, b;
    const __nv_bfloat16* c;
    __nv_bfloat16* d;
    int M, N, K;
    int ldc, ldd;
    int reserved_[7];
};
static_assert(sizeof(GroupEntry) == 320, "tensor maps start on 64 bytes");
struct GroupTile {
    int entry, m0, n0, reserved_;
};

struct GemmArgs {
    const GroupEntry* entries;   // GROUP only: the products of the launch, and their tiles in the order they are taken
    const GroupTile* tiles;
    const __nv_bfloat16* c;
    __nv_bfloat16* d;
    __nv_bfloat16* dt;
    int M, N, K;
    long long ldc, ldd, lddt;
    float alpha, beta;
    int n_tiles;     // PERSIST: number of tiles to compute (see tile_coords)
    int symmetric;   // the result is known to be symmetric (M == N): compute the tiles that touch the upper
                     // triangle only and write every element above the diagonal to its mirror position too
    int* status;
};

__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t it = 0; it < kSpinLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 1023u) == 1023u && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// Shared-memory matrix descriptor of a K-major, 128-byte-swizzled tile whose rows are 128 bytes
// apart: 8-row groups 1024 bytes apart (stride byte offset), descriptor version 1 (sm_100),
// layout type 2 (SWIZZLE_128B). The leading byte offset is not used by swizzled K-major layouts.
__device__ __forceinline__ uint64_t umma_desc_k_major_sw128(uint32_t smem_addr) {
    uint64_t desc = 0;
    desc |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    desc |= static_cast<uint64_t>(1) << 16;
    desc |= static_cast<uint64_t>(1024 >> 4) << 32;
    desc |= static_cast<uint64_t>(1) << 46;
    desc |= static_cast<uint64_t>(2) << 61;
    return desc;
}

// MN-major operand ([K rows][MN contiguous] in memory), 128-byte swizzle: the tile is stored as
// groups of 64 MN-elements (one 128-byte row per K index, 8-row swizzle atoms 1024 bytes apart =
// stride byte offset); successive 64-element groups are `group_bytes` apart (leading byte offset).
__device__ __forceinline__ uint64_t umma_desc_mn_major_sw128(uint32_t smem_addr, uint32_t group_bytes) {
    uint64_t desc = 0;
    desc |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    desc |= static_cast<uint64_t>(group_bytes >> 4) << 16;
    desc |= static_cast<uint64_t>(1024 >> 4) << 32;
    desc |= static_cast<uint64_t>(1) << 46;
    desc |= static_cast<uint64_t>(2) << 61;
    return desc;
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The products of a group follow each other with programmatic launches: a product's CTAs start on idle SMs while the one
// before still runs, set up and fetch their first tile's plan entry (written long before), and wait until it has ended
// before they touch a matrix. Four matrices of 64 to 1026 rows, whole GefenMuon step: 270 -> 245 us; one matrix of 300 x 500:
// 218 -> 191 us, 2048 x 6144: 620 -> 609 us.
__device__ __forceinline__ void let_next_product_in() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_last_product() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A tensor map in global memory, made visible to the tensor-map proxy and fetched ahead of its first use.
__device__ __forceinline__ void fetch_map(const CUtensorMap* map) {
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// Tile t of the persistent schedule: row-major over the tiles that are computed (all of them, or for
// a symmetric result those that reach the upper triangle: n0 + bn > m0).
__host__ __device__ inline bool tile_coords(int M, int N, int bm, int bn, int symmetric, long long t, int* m0, int* n0) {
    const int tiles_m = (M + bm - 1) / bm, tiles_n = (N + bn - 1) / bn;
    if (!symmetric) {
        if (t >= static_cast<long long>(tiles_m) * tiles_n) return false;
        *m0 = static_cast<int>(t / tiles_n) * bm;
        *n0 = static_cast<int>(t % tiles_n) * bn;
        return true;
    }
    for (int mi = 0; mi < tiles_m; ++mi) {
        const int row0 = mi * bm;
        const int first = row0 >= bn ? (row0 - bn) / bn + 1 : 0;
        const int cnt = tiles_n - first;
        if (t < cnt) {
            *m0 = row0;
            *n0 = (first + static_cast<int>(t)) * bn;
            return true;
        }
        t -= cnt;
    }
    return false;
}

// A tile of a launch: its operands, its product's sizes and its place.
struct TileView {
    const CUtensorMap* map_a;
    const CUtensorMap* map_b;
    const __nv_bfloat16* c;
    __nv_bfloat16* d;
    int M, N, K, m0, n0;
    long long ldc, ldd;
};
// Stores one accumulator of 128 rows from row m0 and BN columns from column t.n0: alpha, beta * C, bf16, and the mirror
// image of a symmetric result. Four warps; warp w owns TMEM lanes (rows) 32w .. 32w+31. `wait` returns when the
// accumulator is complete (false: given up).
template <int BN, typename Wait>
__device__ __forceinline__ bool epilogue_tile(const GemmArgs& args, const TileView& t, int m0, uint32_t tmem_acc, int warp, int lane, Wait wait) {
    const int n0 = t.n0;
        const int row = m0 + warp * 32 + lane;
        const bool row_ok = row < t.M;
        // C does not depend on the accumulators: the first chunk's row segment is fetched while the main
        // loop runs, and chunk j+1's while chunk j is converted and stored.
        const bool use_c = row_ok && args.beta != 0.0f;
        const __nv_bfloat16* crow_base = use_c ? t.c + static_cast<long long>(row) * t.ldc : nullptr;
        const bool c_vec = use_c && ((reinterpret_cast<uintptr_t>(crow_base) & 15u) == 0) && (t.ldc % 8 == 0) && (n0 % 8 == 0);
        uint4 cnext[4];
        auto fetch_c = [&](int j) {
            const int col0 = n0 + j * 32;
            if (c_vec && col0 + 32 <= t.N) {
#pragma unroll
                for (int q = 0; q < 4; ++q) cnext[q] = reinterpret_cast<const uint4*>(crow_base + col0)[q];
            }
        };
        fetch_c(0);
        const bool ok = wait();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!ok) return false;
        {
#pragma unroll 2
            for (int j = 0; j < BN / 32; ++j) {
                uint32_t r[32];
                const uint32_t taddr = tmem_acc + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(j * 32);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                    "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                      "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                      "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                    : "r"(taddr)
                    : "memory");
                uint4 ccur[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) ccur[q] = cnext[q];
                if (j + 1 < BN / 32) fetch_c(j + 1);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const int col0 = n0 + j * 32;
                if (col0 >= t.N) continue;
                const bool full_cols = col0 + 32 <= t.N;
                float v[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = args.alpha * __uint_as_float(r[i]);
                if (use_c) {
                    const __nv_bfloat16* crow = crow_base + col0;
                    if (full_cols && c_vec) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const uint4 raw = ccur[q];
                            const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                v[q * 8 + 2 * e] = fmaf(args.beta, __uint_as_float(w[e] << 16), v[q * 8 + 2 * e]);
                                v[q * 8 + 2 * e + 1] = fmaf(args.beta, __uint_as_float(w[e] & 0xFFFF0000u), v[q * 8 + 2 * e + 1]);
                            }
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col0 + i < t.N) v[i] = fmaf(args.beta, __bfloat162float(crow[i]), v[i]);
                    }
                }
                if (row_ok) {
                    __nv_bfloat16* drow = t.d + static_cast<long long>(row) * t.ldd + col0;
                    if (args.symmetric && col0 < row) {
                        // chunk crosses or lies left of the diagonal: only the elements with column >= row
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col0 + i < t.N && col0 + i >= row) drow[i] = __float2bfloat16_rn(v[i]);
                    } else if (full_cols && ((reinterpret_cast<uintptr_t>(drow) & 15u) == 0)) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t w[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const __nv_bfloat162 h = __floats2bfloat162_rn(v[q * 8 + 2 * e], v[q * 8 + 2 * e + 1]);
                                w[e] = *reinterpret_cast<const uint32_t*>(&h);
                            }
                            reinterpret_cast<uint4*>(drow)[q] = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col0 + i < t.N) drow[i] = __float2bfloat16_rn(v[i]);
                    }
                    if (args.dt != nullptr) {
                        // transposed copy: for a fixed column the lanes of a warp write consecutive addresses
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col0 + i < t.N)
                                args.dt[static_cast<long long>(col0 + i) * args.lddt + row] = __float2bfloat16_rn(v[i]);
                    }
                }
                if (args.symmetric) {
                    // mirror: element (row, c) with c > row also goes to (c, row)
                    const int warp_row0 = m0 + warp * 32;
                    if (col0 > warp_row0 + 31 && warp_row0 + 31 < t.M && full_cols) {
                        // the whole chunk is right of every row of this warp (warp-uniform): lanes pair up so
                        // that each store carries two consecutive rows of one column (4 bytes)
                        const bool odd = (lane & 1) != 0;
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const float send = odd ? v[i] : v[i + 1];
                            const float recv = __shfl_xor_sync(0xffffffffu, send, 1);
                            const float lo = odd ? recv : v[i];          // value of the even row
                            const float hi = odd ? v[i + 1] : recv;      // value of the odd row
                            const int c = col0 + i + (odd ? 1 : 0);
                            const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
                            *reinterpret_cast<__nv_bfloat162*>(t.d + static_cast<long long>(c) * t.ldd + (row & ~1)) = h;
                        }
                    } else if (row_ok && col0 + 31 > row) {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col0 + i < t.N && col0 + i > row)
                                t.d[static_cast<long long>(col0 + i) * t.ldd + row] = __float2bfloat16_rn(v[i]);
                    }
                }
            }
        }
    return true;
}

// B_MN = false: B is [N, K] row-major (K-major operand). B_MN = true: B is [K, N] row-major
// (MN-major operand), i.e. D = alpha * A * B + beta * C without any transposed copy of B.
// A_MN: likewise A given as [K, M] row-major (D = alpha * A^T * B ...), used for the Gram matrix of a
// tall matrix, Y^T Y, without transposing Y.
// Variants whose ring is at most 96 KB run two CTAs per SM: the epilogue of one overlaps the main
// loop of the other (each holds BN <= 256 of the 512 TMEM columns).
// GROUP (a persistent variant): the launch computes the products of many matrices; a tile names its product, whose
// tensor maps and sizes come from global memory (the host has copied them there before the launch).
template <int BN, int STAGES, bool A_MN, bool B_MN, bool PERSIST, bool GROUP = false>
__global__ void __launch_bounds__(kGemmThreads, (STAGES * (kBM + BN) * kBK * 2 <= 96 * 1024) ? 2 : 1) ns_gemm_tn_kernel(const __grid_constant__ CUtensorMap map_a,
                                                                     const __grid_constant__ CUtensorMap map_b,
                                                                     const __grid_constant__ GemmArgs args) {
    constexpr int kABytes = kBM * kBK * 2;
    constexpr int kBBytes = BN * kBK * 2;
    constexpr int kStageBytes = kABytes + kBBytes;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    __shared__ uint64_t full_bar[STAGES];
    __shared__ uint64_t empty_bar[STAGES];
    __shared__ uint64_t acc_full[2];    // accumulator buffer complete (MMA -> epilogue)
    __shared__ uint64_t acc_empty[2];   // accumulator buffer drained (4 epilogue warps -> MMA); PERSIST only
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    constexpr int kTmemCols = PERSIST ? 2 * BN : BN;
    if (!PERSIST && args.symmetric && static_cast<int>(blockIdx.x) * BN + BN <= static_cast<int>(blockIdx.y) * kBM)
        return;   // tile entirely below the diagonal: its mirror image computes it
    // li-th tile of this CTA
    auto my_tile = [&](int li, TileView& t) -> bool {
        const long long index = static_cast<long long>(blockIdx.x) + static_cast<long long>(li) * gridDim.x;
        if constexpr (GROUP) {
            if (index >= args.n_tiles) return false;
            const GroupTile g = args.tiles[index];
            const GroupEntry* e = args.entries + g.entry;
            t.map_a = &e->a;
            t.map_b = &e->b;
            t.c = e->c;
            t.d = e->d;
            t.M = e->M; t.N = e->N; t.K = e->K;
            t.ldc = e->ldc; t.ldd = e->ldd;
            t.m0 = g.m0; t.n0 = g.n0;
            return true;
        }
        t.map_a = &map_a;
        t.map_b = &map_b;
        t.c = args.c;
        t.d = args.d;
        t.M = args.M; t.N = args.N; t.K = args.K;
        t.ldc = args.ldc; t.ldd = args.ldd;
        if (!PERSIST) {
            t.m0 = blockIdx.y * kBM;
            t.n0 = blockIdx.x * BN;
            return li == 0;
        }
        return index < args.n_tiles && tile_coords(args.M, args.N, kBM, BN, args.symmetric, index, &t.m0, &t.n0);
    };

    if constexpr (GROUP) {
        let_next_product_in();
        TileView first;
        if (threadIdx.x == 32 * 4 && my_tile(0, first)) { fetch_map(first.map_a); fetch_map(first.map_b); }
    }
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4); }
        fence_mbar_init();
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    if constexpr (GROUP) wait_for_last_product();

    if (warp == 4) {
        // ---------------- producer
        if (lane == 0) {
            if constexpr (!GROUP) {
                asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
                asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
            }
            uint32_t it = 0;   // k-blocks issued so far, over all tiles: ring slot and phase
            bool ok = true;
            TileView t;
            for (int li = 0; ok && my_tile(li, t); ++li) {
            const int m0 = t.m0, n0 = t.n0, k_blocks = (t.K + kBK - 1) / kBK;
            if constexpr (GROUP) {   // maps in global memory: make the host's copy visible to the tensor-map proxy
                asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(t.map_a) : "memory");
                asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(t.map_b) : "memory");
            }
            for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                const int s = it % STAGES;
                const uint32_t parity = ((it / STAGES) & 1) ^ 1;
                if (!wait_or_abort(&empty_bar[s], parity, &abort_flag)) { ok = false; break; }
                mbar_expect_tx(&full_bar[s], kStageBytes);
                unsigned char* a_dst = smem + s * kStageBytes;
                if (!A_MN) {
                    tma_load_2d(a_dst, t.map_a, kb * kBK, m0, &full_bar[s]);
                } else {
#pragma unroll
                    for (int j = 0; j < kBM / 64; ++j)
                        tma_load_2d(a_dst + j * (kBK * 128), t.map_a, m0 + 64 * j, kb * kBK, &full_bar[s]);
                }
                if (!B_MN && GROUP) {   // (one map serves both operands: boxes of 128 rows)
#pragma unroll
                    for (int j = 0; j < BN / kBM; ++j)
                        tma_load_2d(a_dst + kABytes + j * kABytes, t.map_b, kb * kBK, n0 + kBM * j, &full_bar[s]);
                } else if (!B_MN) {
                    tma_load_2d(a_dst + kABytes, t.map_b, kb * kBK, n0, &full_bar[s]);
                } else {
#pragma unroll
                    for (int j = 0; j < BN / 64; ++j)   // 64 K-rows x 64 N-columns per box
                        tma_load_2d(a_dst + kABytes + j * (kBK * 128), t.map_b, n0 + 64 * j, kb * kBK, &full_bar[s]);
                }
            }
            }
        }
        __syncwarp();
    } else if (warp == 5) {
        // ---------------- MMA issuer
        if (lane == 0) {
            // instruction descriptor: fp32 accumulate, bf16 x bf16, both K-major, N = BN, M = 128
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (A_MN ? (1u << 15) : 0u) | (B_MN ? (1u << 16) : 0u) |
                                       (static_cast<uint32_t>(BN >> 3) << 17) | (static_cast<uint32_t>(kBM >> 4) << 24);
            bool ok = true;
            uint32_t it = 0;
            TileView t;
            for (int li = 0; ok && my_tile(li, t); ++li) {
            const int k_blocks = (t.K + kBK - 1) / kBK;
            const int buf = PERSIST ? (li & 1) : 0;
            const uint32_t tmem_acc = tmem_base + static_cast<uint32_t>(buf * BN);
            if (PERSIST) {   // the epilogue has drained this buffer (passes at once for the first two tiles)
                ok = wait_or_abort(&acc_empty[buf], ((li >> 1) & 1) ^ 1, &abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            for (int kb = 0; kb < k_blocks && ok; ++kb, ++it) {
                const int s = it % STAGES;
                const uint32_t parity = (it / STAGES) & 1;
                ok = wait_or_abort(&full_bar[s], parity, &abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_addr = smem_u32(smem + s * kStageBytes);
                const uint64_t desc_a = A_MN ? umma_desc_mn_major_sw128(a_addr, kBK * 128) : umma_desc_k_major_sw128(a_addr);
                const uint64_t desc_b = B_MN ? umma_desc_mn_major_sw128(a_addr + kABytes, kBK * 128)
                                             : umma_desc_k_major_sw128(a_addr + kABytes);
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k) {
                    // K-major: 16 bf16 along K = 32 bytes inside the swizzle row (+2 in the address field);
                    // MN-major: 16 K-rows of 128 bytes = 2048 bytes (+128)
                    umma_bf16(tmem_acc, desc_a + (A_MN ? 128 : 2) * k, desc_b + (B_MN ? 128 : 2) * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                }
                umma_commit(&empty_bar[s]);   // the slot is free once these MMAs have read it
            }
            umma_commit(&acc_full[buf]);      // accumulators complete (or abandoned)
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: warp w owns TMEM lanes (rows) 32w .. 32w+31
        TileView t;
        for (int li = 0; my_tile(li, t); ++li) {
        const int buf = PERSIST ? (li & 1) : 0;
        const bool ok = epilogue_tile<BN>(args, t, t.m0, tmem_base + static_cast<uint32_t>(buf * BN), warp, lane, [&]() {
            return wait_or_abort(&acc_full[buf], PERSIST ? ((li >> 1) & 1) : 0, &abort_flag) && !abort_flag;
        });
        if (!ok) break;
        if (PERSIST) {   // this warp has read its rows of the buffer: one arrival per warp
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (warp == 5) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
    if (threadIdx.x == 0 && abort_flag && args.status != nullptr) atomicExch(args.status, 1);
}

// --------------------------------------------------------------------------- pairs of CTAs
// The grouped products on pairs of SMs: tcgen05.mma.cta_group::2 on tiles of 256 x 256. Each CTA stages its 128 rows of A
// and its half of B's 256 columns (32 KB per 64 k instead of 48 KB for the 128 x 256 tile of a single CTA, whose
// operand stream the L2 cannot feed at the tensor cores' rate) and holds its 128 rows of the accumulator in its own TMEM.
// The first CTA's thread issues the products and the commits; "slot full" barriers live in the first CTA (both CTAs'
// copies complete on them), "slot free" and "accumulator full" arrive in both, "accumulator drained" in the first.
// Products of 28 Qwen3-1.7B-shaped matrices (6.83 TFLOP): 6.43 ms with 128 x 256 tiles, 6.04 on pairs, 5.55 with the
// epilogue through shared memory = 1230 TFLOP/s, 0.88 of the measured sustained rate; what is left is the tensor
// cores at the clock that the power limit leaves. 24 matrices of a 768-wide transformer: 0.85 -> 0.74 ms.
// Every wait gives up after kPairWaitCycles; the roles then leave, a grace period lets copies in flight land, and the
// CTAs part at a cluster barrier that all their threads reach.
constexpr int kPairStages = 6;
constexpr int kPairBN = 256;
constexpr long long kPairWaitCycles = 1000000000ll;   // about half a second

__device__ __forceinline__ uint32_t cluster_address(const void* local, uint32_t rank) {
    uint32_t out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(smem_u32(local)), "r"(rank));
    return out;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool pair_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    const uint32_t addr = smem_u32(bar);
    const long long begin = clock64();
    for (uint32_t it = 1;; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 15u) == 0u && (*abort_flag || clock64() - begin > kPairWaitCycles)) break;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void pair_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void pair_commit(uint64_t* bar) {   // arrives on this barrier of both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
}

// The same through shared memory, 64 columns at a time: a row of the accumulator belongs to a lane, so that direct loads
// of C and stores of D touch 32 rows with 16 bytes each per instruction, which costs the memory pipe as much time as a
// product of 2048 k takes; here an instruction moves four rows of 128 bytes. `stage`: this warp's 32 rows of
// kStagePitch elements. C and D: 16-byte aligned rows, N a multiple of 8 (groups guarantee both).
constexpr int kStagePitch = 72;
__device__ __forceinline__ void tmem_load32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
template <int BN, typename Wait>
__device__ __forceinline__ bool epilogue_tile_staged(const GemmArgs& args, const TileView& t, int m0, uint32_t tmem_acc, int warp, int lane,
                                                     __nv_bfloat16* stage, Wait wait) {
    const int row0 = m0 + warp * 32, row = row0 + lane;
    const bool use_c = args.beta != 0.0f;
    const int piece_row = lane >> 3, piece_col = (lane & 7) * 8;   // of the coalesced accesses: four rows of 128 bytes each
    uint4 cnext[8];
    auto fetch_c = [&](int col0) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int r = row0 + 4 * q + piece_row, c = col0 + piece_col;
            if (r < t.M && c < t.N) cnext[q] = *reinterpret_cast<const uint4*>(t.c + static_cast<long long>(r) * t.ldc + c);
        }
    };
    if (use_c) fetch_c(t.n0);
    if (!wait()) return false;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __nv_bfloat16* const own = stage + lane * kStagePitch;
    for (int j = 0; j < BN / 64; ++j) {
        const int col0 = t.n0 + 64 * j;
        if (col0 >= t.N) break;
        uint32_t r[64];
        const uint32_t taddr = tmem_acc + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(j * 64);
        tmem_load32(taddr, r);
        tmem_load32(taddr + 32, r + 32);
        if (use_c) {
#pragma unroll
            for (int q = 0; q < 8; ++q) *reinterpret_cast<uint4*>(stage + (4 * q + piece_row) * kStagePitch + piece_col) = cnext[q];
            if (j + 1 < BN / 64) fetch_c(col0 + 64);
            __syncwarp();
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float v[64];
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i] = args.alpha * __uint_as_float(r[i]);
        if (use_c) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint4 raw = *reinterpret_cast<const uint4*>(own + 8 * q);
                const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    v[q * 8 + 2 * e] = fmaf(args.beta, __uint_as_float(w[e] << 16), v[q * 8 + 2 * e]);
                    v[q * 8 + 2 * e + 1] = fmaf(args.beta, __uint_as_float(w[e] & 0xFFFF0000u), v[q * 8 + 2 * e + 1]);
                }
            }
        }
        // (a lane overwrites its own row of C only: no other lane reads it any more)
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(v[q * 8 + 2 * e], v[q * 8 + 2 * e + 1]);
                w[e] = *reinterpret_cast<const uint32_t*>(&h);
            }
            *reinterpret_cast<uint4*>(own + 8 * q) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int rr = row0 + 4 * q + piece_row, c = col0 + piece_col;
            if (rr >= t.M || c >= t.N) continue;
            const __nv_bfloat16* from = stage + (4 * q + piece_row) * kStagePitch + piece_col;
            __nv_bfloat16* to = t.d + static_cast<long long>(rr) * t.ldd + c;
            if (!args.symmetric || c >= rr) {
                *reinterpret_cast<uint4*>(to) = *reinterpret_cast<const uint4*>(from);
            } else {   // crosses or lies left of the diagonal: only the elements with column >= row
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (c + e >= rr) to[e] = from[e];
            }
        }
        if (args.symmetric) {
            // mirror: element (row, c) with c > row also goes to (c, row)
            if (col0 > row0 + 31 && row0 + 31 < t.M && col0 + 64 <= t.N) {
                // the whole chunk is right of every row of this warp (warp-uniform): lanes pair up so that each store
                // carries two consecutive rows of one column (4 bytes)
                const bool odd = (lane & 1) != 0;
#pragma unroll
                for (int i = 0; i < 64; i += 2) {
                    const float send = odd ? v[i] : v[i + 1];
                    const float recv = __shfl_xor_sync(0xffffffffu, send, 1);
                    const float lo = odd ? recv : v[i];          // value of the even row
                    const float hi = odd ? v[i + 1] : recv;      // value of the odd row
                    const int c = col0 + i + (odd ? 1 : 0);
                    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
                    *reinterpret_cast<__nv_bfloat162*>(t.d + static_cast<long long>(c) * t.ldd + (row & ~1)) = h;
                }
            } else if (row < t.M && col0 + 63 > row) {
#pragma unroll
                for (int i = 0; i < 64; ++i)
                    if (col0 + i < t.N && col0 + i > row) t.d[static_cast<long long>(col0 + i) * t.ldd + row] = __float2bfloat16_rn(v[i]);
            }
        }
        __syncwarp();   // the stage is free for the next 64 columns
    }
    return true;
}

template <bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1) ns_gemm_pair_kernel(const __grid_constant__ GemmArgs args) {
    constexpr int kABytes = kBM * kBK * 2;            // this CTA's rows of A
    constexpr int kBBytes = kPairBN / 2 * kBK * 2;    // and its half of B
    constexpr int kStageBytes = kABytes + kBBytes;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    __shared__ uint64_t full_bar[kPairStages];    // first CTA: operands of both CTAs have arrived
    __shared__ uint64_t empty_bar[kPairStages];   // each CTA: its slot has been read
    __shared__ uint64_t acc_full[2];              // each CTA: accumulator complete
    __shared__ uint64_t acc_empty[2];             // first CTA: drained by the eight epilogue warps of the pair
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    // (behind the ring of slots: the epilogue warps' stages)
    __nv_bfloat16* const stages = reinterpret_cast<__nv_bfloat16*>(smem + kPairStages * kStageBytes);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int pair_index = static_cast<int>(blockIdx.x >> 1), pairs = static_cast<int>(gridDim.x >> 1);
    auto my_tile = [&](int li, TileView& t) -> bool {
        const long long index = static_cast<long long>(pair_index) + static_cast<long long>(li) * pairs;
        if (index >= args.n_tiles) return false;
        const GroupTile g = args.tiles[index];
        const GroupEntry* e = args.entries + g.entry;
        t.map_a = &e->a;
        t.map_b = &e->b;
        t.c = e->c;
        t.d = e->d;
        t.M = e->M; t.N = e->N; t.K = e->K;
        t.ldc = e->ldc; t.ldd = e->ldd;
        t.m0 = g.m0; t.n0 = g.n0;
        return true;
    };

    let_next_product_in();
    if (threadIdx.x == 32 * 4) {
        TileView first;
        if (my_tile(0, first)) { fetch_map(first.map_a); fetch_map(first.map_b); }
    }
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < kPairStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8); }
        fence_mbar_init();
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(2 * kPairBN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();   // both CTAs' barriers exist before either signals the other's
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    wait_for_last_product();

    if (warp == 4) {
        // ---------------- producer of this CTA's operands
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            TileView t;
            for (int li = 0; ok && my_tile(li, t); ++li) {
                const int m0 = t.m0 + static_cast<int>(rank) * kBM, n0 = t.n0 + static_cast<int>(rank) * (kPairBN / 2);
                const int k_blocks = (t.K + kBK - 1) / kBK;
                asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(t.map_a) : "memory");
                asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(t.map_b) : "memory");
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % kPairStages;
                    if (!pair_wait(&empty_bar[s], ((it / kPairStages) & 1) ^ 1, &abort_flag)) { ok = false; break; }
                    if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * kStageBytes);
                    const uint32_t bar = cluster_address(&full_bar[s], 0);
                    unsigned char* a_dst = smem + s * kStageBytes;
                    pair_load_2d(a_dst, t.map_a, kb * kBK, m0, bar);
                    if (!B_MN) {
                        pair_load_2d(a_dst + kABytes, t.map_b, kb * kBK, n0, bar);
                    } else {
#pragma unroll
                        for (int j = 0; j < kPairBN / 2 / 64; ++j)   // 64 K-rows x 64 N-columns per box
                            pair_load_2d(a_dst + kABytes + j * (kBK * 128), t.map_b, n0 + 64 * j, kb * kBK, bar);
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 5) {
        // ---------------- MMA issuer of the pair
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (B_MN ? (1u << 16) : 0u) |
                                       (static_cast<uint32_t>(kPairBN >> 3) << 17) | (static_cast<uint32_t>(2 * kBM >> 4) << 24);
            bool ok = true;
            uint32_t it = 0;
            TileView t;
            for (int li = 0; ok && my_tile(li, t); ++li) {
                const int k_blocks = (t.K + kBK - 1) / kBK;
                const int buf = li & 1;
                const uint32_t tmem_acc = tmem_base + static_cast<uint32_t>(buf * kPairBN);
                ok = pair_wait(&acc_empty[buf], ((li >> 1) & 1) ^ 1, &abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % kPairStages;
                    ok = pair_wait(&full_bar[s], (it / kPairStages) & 1, &abort_flag);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_addr = smem_u32(smem + s * kStageBytes);
                    const uint64_t desc_a = umma_desc_k_major_sw128(a_addr);
                    const uint64_t desc_b = B_MN ? umma_desc_mn_major_sw128(a_addr + kABytes, kBK * 128) : umma_desc_k_major_sw128(a_addr + kABytes);
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k) {
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                            ::"r"(tmem_acc), "l"(desc_a + 2 * k), "l"(desc_b + (B_MN ? 128 : 2) * k), "r"(idesc), "r"((kb > 0 || k > 0) ? 1u : 0u)
                            : "memory");
                    }
                    pair_commit(&empty_bar[s]);   // the slot is free in both CTAs once these products have read it
                }
                if (ok) pair_commit(&acc_full[buf]);
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue of this CTA's rows
        TileView t;
        for (int li = 0; my_tile(li, t); ++li) {
            const int buf = li & 1;
            const bool ok = epilogue_tile_staged<kPairBN>(args, t, t.m0 + static_cast<int>(rank) * kBM, tmem_base + static_cast<uint32_t>(buf * kPairBN),
                                                          warp, lane, stages + warp * 32 * kStagePitch,
                                                          [&]() { return pair_wait(&acc_full[buf], (li >> 1) & 1, &abort_flag); });
            if (!ok) break;
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_address(&acc_empty[buf], 0)) : "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (abort_flag) {   // given up: copies and products in flight get time to end before their memory goes
        const long long begin = clock64();
        while (clock64() - begin < 4000000ll) __nanosleep(1000);
    }
    cluster_sync_all();
    if (warp == 5) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * kPairBN) : "memory");
    }
    if (threadIdx.x == 0 && abort_flag && args.status != nullptr) atomicExch(args.status, 1);
    cluster_sync_all();   // (neither CTA's TMEM permits or shared memory go before the other is done with the pair)
}

// ------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &res) == cudaSuccess &&
            res == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
        }
    });
    return fn;
}

// [rows, cols] bf16 row-major with leading dimension ld (elements); box = 64 (inner) x box_rows, 128-byte swizzle.
static int make_map(CUtensorMap* map, const void* base, long long rows, long long k, long long ld, int box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) return fail(GEFEN_B200_ECUDA, "cuTensorMapEncodeTiled is not available from the driver.");
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
    cuuint32_t box[2] = {static_cast<cuuint32_t>(kBK), static_cast<cuuint32_t>(box_rows)};
    cuuint32_t elem[2] = {1, 1};
    const CUresult rc = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) return fail(GEFEN_B200_ECUDA, "cuTensorMapEncodeTiled failed with code %d.", static_cast<int>(rc));
    return GEFEN_B200_OK;
}

// Tiles a launch computes (see tile_coords).
static int count_tiles(int M, int N, int bm, int bn, int symmetric) {
    const int tiles_m = (M + bm - 1) / bm, tiles_n = (N + bn - 1) / bn;
    if (!symmetric) return tiles_m * tiles_n;
    int total = 0;
    for (int mi = 0; mi < tiles_m; ++mi) {
        const int row0 = mi * bm;
        total += tiles_n - (row0 >= bn ? (row0 - bn) / bn + 1 : 0);
    }
    return total;
}

// A product of a group: overlapped with the end of whatever precedes it (see let_next_product_in).
template <typename K, typename... Args>
static int launch_product(K kernel, int grid, int smem, cudaStream_t stream, const Args&... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(grid));
    config.blockDim = dim3(kGemmThreads);
    config.dynamicSmemBytes = static_cast<size_t>(smem);
    config.stream = stream;
    cudaLaunchAttribute overlap = {};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &overlap;
    config.numAttrs = 1;
    GEFEN_CHECK_CUDA(cudaLaunchKernelEx(&config, kernel, args...));
    return GEFEN_B200_OK;
}

template <int BN, int STAGES, bool A_MN, bool B_MN, bool PERSIST, bool GROUP = false>
static int launch_gemm_variant(const CUtensorMap& ma, const CUtensorMap& mb, GemmArgs args, cudaStream_t stream) {
    constexpr int smem = STAGES * (kBM * kBK * 2 + BN * kBK * 2) + 1024;
    static bool configured[64];
    int dev = 0;
    GEFEN_CHECK_CUDA(cudaGetDevice(&dev));
    auto kernel = ns_gemm_tn_kernel<BN, STAGES, A_MN, B_MN, PERSIST, GROUP>;
    if (dev < 64 && !configured[dev]) {
        GEFEN_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured[dev] = true;
    }
    if (!GROUP) args.n_tiles = count_tiles(args.M, args.N, kBM, BN, args.symmetric);
    dim3 grid(GROUP ? 1 : (args.N + BN - 1) / BN, GROUP ? 1 : (args.M + kBM - 1) / kBM);
    if (PERSIST) grid = dim3(args.n_tiles < sm_count() ? args.n_tiles : sm_count(), 1);
    if constexpr (GROUP) return launch_product(kernel, static_cast<int>(grid.x), smem, stream, ma, mb, args);
    kernel<<<grid, kGemmThreads, smem, stream>>>(ma, mb, args);
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

// More tiles than SMs: one persistent CTA per SM with two accumulator buffers, so that a tile's
// epilogue overlaps the next tile's main loop. Otherwise one CTA per tile.
// GEFEN_B200_NS_PERSIST=0/1 forces the choice (measurements).
template <int BN, int STAGES, bool A_MN, bool B_MN>
static int launch_gemm(const CUtensorMap& ma, const CUtensorMap& mb, const GemmArgs& args, cudaStream_t stream) {
    static int forced = -2;
    if (forced == -2) {
        const char* e = getenv("GEFEN_B200_NS_PERSIST");
        forced = e == nullptr ? -1 : (e[0] == '0' ? 0 : 1);
    }
    bool persist = count_tiles(args.M, args.N, kBM, BN, args.symmetric) > sm_count();
    if (forced >= 0) persist = forced == 1;
    if constexpr (STAGES * (kBM + BN) * kBK * 2 > 96 * 1024) {   // the two-CTAs-per-SM variants stay one tile per CTA
        if (persist) return launch_gemm_variant<BN, STAGES, A_MN, B_MN, true>(ma, mb, args, stream);
    }
    return launch_gemm_variant<BN, STAGES, A_MN, B_MN, false>(ma, mb, args, stream);
}

}  // namespace gefen

using namespace gefen;

static int ns_gemm(const void* a, bool a_is_km, const void* b, bool b_is_kn, const void* c, void* d, void* dt, int M, int N, int K,
                   int64_t lda, int64_t ldb, int64_t ldc, int64_t ldd, int64_t lddt, double alpha, double beta,
                   int symmetric, int* status, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(a != nullptr && b != nullptr && d != nullptr, "Expected non-null A, B and D.");
    GEFEN_CHECK_ARG(M > 0 && N > 0 && K > 0, "Expected positive GEMM sizes.");
    GEFEN_CHECK_ARG(beta == 0.0 || c != nullptr, "Expected C when beta != 0.");
    GEFEN_CHECK_ARG(!symmetric || (M == N && ldd % 2 == 0 && (reinterpret_cast<uintptr_t>(d) & 3u) == 0 && dt == nullptr),
                    "A symmetric result needs M == N, an even leading dimension and no transposed output.");
    GEFEN_CHECK_ARG(aligned16(a) && aligned16(b) && lda % 8 == 0 && ldb % 8 == 0 && lda >= (a_is_km ? M : K) &&
                        ldb >= (b_is_kn ? N : K),
                    "Expected 16-byte aligned A and B with leading dimensions that are multiples of 8 elements.");
    GEFEN_CHECK_ARG(ldd >= N && (c == nullptr || ldc >= N) && (dt == nullptr || lddt >= M), "Bad leading dimension.");
    // 128 x 256 tiles have the better arithmetic intensity; 128 x 128 tiles are used for small problems
    // that would leave most SMs without a tile (measured: for 2048-wide outputs the wider tile wins
    // even when a symmetric result computes only 72 of them)
    int bn = (N >= 2048 || (static_cast<long long>((M + 127) / 128) * ((N + 255) / 256)) >= sm_count()) ? 256 : 128;
    // GEFEN_B200_NS_TILE=<bn>x<stages> picks a variant by hand (measurements): 256x4, 256x2, 128x6, 128x3
    static int forced_bn = -1, forced_stages = 0;
    if (forced_bn < 0) {
        forced_bn = 0;
        const char* e = getenv("GEFEN_B200_NS_TILE");
        if (e != nullptr) sscanf(e, "%dx%d", &forced_bn, &forced_stages);
    }
    if (forced_bn == 256 || forced_bn == 128) bn = forced_bn;
    const bool shallow = forced_stages == 2 || forced_stages == 3;
    CUtensorMap ma, mb;
    int rc = a_is_km ? make_map(&ma, a, K, M, lda, kBK) : make_map(&ma, a, M, K, lda, kBM);
    if (rc != GEFEN_B200_OK) return rc;
    rc = b_is_kn ? make_map(&mb, b, K, N, ldb, kBK) : make_map(&mb, b, N, K, ldb, bn);
    if (rc != GEFEN_B200_OK) return rc;
    GemmArgs args = {};
    args.c = static_cast<const __nv_bfloat16*>(c);
    args.d = static_cast<__nv_bfloat16*>(d);
    args.dt = static_cast<__nv_bfloat16*>(dt);
    args.M = M; args.N = N; args.K = K;
    args.ldc = ldc; args.ldd = ldd; args.lddt = lddt;
    args.alpha = static_cast<float>(alpha);
    args.beta = static_cast<float>(beta);
    args.symmetric = symmetric;
    args.status = status;
    if (a_is_km && b_is_kn) {
        if (shallow) return bn == 256 ? launch_gemm<256, 2, true, true>(ma, mb, args, stream)
                                      : launch_gemm<128, 3, true, true>(ma, mb, args, stream);
        if (bn == 256) return launch_gemm<256, 4, true, true>(ma, mb, args, stream);
        return launch_gemm<128, 6, true, true>(ma, mb, args, stream);
    }
    if (a_is_km) return fail(GEFEN_B200_EUNSUPPORTED, "A given as [K, M] is only combined with B given as [K, N].");
    if (b_is_kn) {
        if (shallow) return bn == 256 ? launch_gemm<256, 2, false, true>(ma, mb, args, stream)
                                      : launch_gemm<128, 3, false, true>(ma, mb, args, stream);
        if (bn == 256) return launch_gemm<256, 4, false, true>(ma, mb, args, stream);
        return launch_gemm<128, 6, false, true>(ma, mb, args, stream);
    }
    if (shallow) return bn == 256 ? launch_gemm<256, 2, false, false>(ma, mb, args, stream)
                                  : launch_gemm<128, 3, false, false>(ma, mb, args, stream);
    if (bn == 256) return launch_gemm<256, 4, false, false>(ma, mb, args, stream);
    return launch_gemm<128, 6, false, false>(ma, mb, args, stream);
}

// The Newton-Schulz iteration of one already normalised matrix in the caller's buffers, for callers of the C interface
// (the package itself runs groups, see below): fifteen GEMM launches for five steps, a tall matrix as it lies (Y^T Y, Y B).
static int enqueue_newton_schulz(void* x0, void* x1, void* gram, void* poly, int rows, int cols, int steps, double a,
                                 double b, double c, int* status, void* stream) {
    const int m = rows < cols ? rows : cols;
    void* cur = x0;
    void* nxt = x1;
    for (int it = 0; it < steps; ++it) {
        int rc;
        if (rows <= cols) {
            // G = X X^T ; B = b G + c G G ; X' = a X + B X
            rc = ns_gemm(cur, false, cur, false, nullptr, gram, nullptr, m, m, cols, cols, cols, 0, m, 0, 1.0, 0.0, 1, status, stream);
            if (rc != GEFEN_B200_OK) return rc;
            rc = ns_gemm(gram, false, gram, false, gram, poly, nullptr, m, m, m, m, m, m, m, 0, c, b, 1, status, stream);
            if (rc != GEFEN_B200_OK) return rc;
            rc = ns_gemm(poly, false, cur, true, cur, nxt, nullptr, rows, cols, m, m, cols, cols, cols, 0, 1.0, a, 0, status, stream);
            if (rc != GEFEN_B200_OK) return rc;
        } else {
            // G = Y^T Y ; B = b G + c G G ; Y' = a Y + Y B
            rc = ns_gemm(cur, true, cur, true, nullptr, gram, nullptr, m, m, rows, cols, cols, 0, m, 0, 1.0, 0.0, 1, status, stream);
            if (rc != GEFEN_B200_OK) return rc;
            rc = ns_gemm(gram, false, gram, false, gram, poly, nullptr, m, m, m, m, m, m, m, 0, c, b, 1, status, stream);
            if (rc != GEFEN_B200_OK) return rc;
            rc = ns_gemm(cur, false, poly, true, cur, nxt, nullptr, rows, cols, m, cols, m, cols, cols, 0, 1.0, a, 0, status, stream);
            if (rc != GEFEN_B200_OK) return rc;
        }
        void* t = cur; cur = nxt; nxt = t;
    }
    return GEFEN_B200_OK;
}

extern "C" int gefen_b200_newton_schulz(void* x0, void* x1, void* gram, void* poly, int rows, int cols, int steps,
                                        double a, double b, double c, int* status, void* stream) {
    GEFEN_CHECK_ARG(x0 && x1 && gram && poly, "Expected non-null buffers.");
    GEFEN_CHECK_ARG(rows > 0 && cols > 0 && rows % 8 == 0 && cols % 8 == 0, "Expected dimensions that are multiples of 8.");
    GEFEN_CHECK_ARG(steps >= 0 && steps < 100, "Number of steps must be less than 100.");
    return enqueue_newton_schulz(x0, x1, gram, poly, rows, cols, steps, a, b, c, status, stream);
}

extern "C" int gefen_b200_ns_gemm_tn(const void* a, const void* b, const void* c, void* d, void* dt, int M, int N, int K,
                                     int64_t lda, int64_t ldb, int64_t ldc, int64_t ldd, int64_t lddt, double alpha,
                                     double beta, int symmetric, int* status, void* stream) {
    return ns_gemm(a, false, b, false, c, d, dt, M, N, K, lda, ldb, ldc, ldd, lddt, alpha, beta, symmetric, status, stream);
}

extern "C" int gefen_b200_ns_gemm_nn(const void* a, const void* b, const void* c, void* d, int M, int N, int K,
                                     int64_t lda, int64_t ldb, int64_t ldc, int64_t ldd, double alpha, double beta,
                                     int* status, void* stream) {
    return ns_gemm(a, false, b, true, c, d, nullptr, M, N, K, lda, ldb, ldc, ldd, 0, alpha, beta, 0, status, stream);
}

extern "C" int gefen_b200_ns_gemm_tt(const void* a, const void* b, const void* c, void* d, int M, int N, int K,
                                     int64_t lda, int64_t ldb, int64_t ldc, int64_t ldd, double alpha, double beta,
                                     int symmetric, int* status, void* stream) {
    return ns_gemm(a, true, b, true, c, d, nullptr, M, N, K, lda, ldb, ldc, ldd, 0, alpha, beta, symmetric, status, stream);
}

// --------------------------------------------------------------------------- many matrices at once
// The matrices of an optimizer step go through the iteration together: one launch per product for all of them, so
// that the tiles of small matrices fill the GPU (one 768 x 768 Gram matrix has 12 tiles of 128 x 256 for 148 SMs) and
// the last wave is paid once per product instead of once per matrix and product, and so that the host enqueues
// 3 * steps + 3 launches instead of that many per matrix. Measured, whole GefenMuon steps: 24 matrices of a 768-wide
// transformer 3.86 -> 1.25 ms, four matrices of 64 to 1026 rows 0.61 -> 0.27 ms, 28 Qwen3-1.7B-shaped matrices
// 9.5 -> 8.3 ms (7.6 ms on pairs of CTAs). Tall matrices enter transposed (Y^T Y = X X^T for X = Y^T), so
// every product has one of two forms: A * B^T with both operands K-major, or A * B with B MN-major.
namespace gefen {

// What the element-wise kernels read of a matrix; uploaded with every call (the step's scalars are in it).
typedef gefen_b200_ns_matrix_t NsMatrix;

constexpr int kNormParts = 64;      // CTAs per matrix of the norm
constexpr int kElemThreads = 256;
constexpr int kTile = 64;           // transposing tile
constexpr int kTilePitch = 72;      // its rows start on 16 bytes

__device__ __forceinline__ bool ns_tall(const NsMatrix& m) { return m.rows > m.cols; }
__device__ __forceinline__ int ns_wide_rows(const NsMatrix& m) { return (static_cast<int>(m.rows < m.cols ? m.rows : m.cols) + 7) / 8 * 8; }
__device__ __forceinline__ int ns_wide_cols(const NsMatrix& m) { return (static_cast<int>(m.rows < m.cols ? m.cols : m.rows) + 7) / 8 * 8; }

template <typename S> __device__ __forceinline__ float as_bf16(const S* p) { return __bfloat162float(__float2bfloat16_rn(ScalarIO<S>::load(p))); }

// Partial sums of squares of the matrix rounded to bf16, in a fixed order.
template <typename S>
__global__ void __launch_bounds__(kElemThreads) ns_norm_kernel(const NsMatrix* __restrict__ table, float* __restrict__ parts) {
    __shared__ float red[kElemThreads / 32];
    const NsMatrix& m = table[blockIdx.y];
    const long long n = m.rows * m.cols;
    const S* src = static_cast<const S*>(m.src);
    constexpr int kVec = 16 / static_cast<int>(sizeof(S));
    const long long per = ((n + kNormParts - 1) / kNormParts + kVec - 1) / kVec * kVec;   // (src starts on 16 bytes)
    const long long begin = per * blockIdx.x;
    const long long end = begin + per < n ? begin + per : n;
    float acc = 0.0f;
    long long i = begin + static_cast<long long>(threadIdx.x) * kVec;
    auto take = [&](const uint4& raw) {
        const S* v = reinterpret_cast<const S*>(&raw);
#pragma unroll
        for (int e = 0; e < kVec; ++e) { const float f = as_bf16(v + e); acc = fmaf(f, f, acc); }
    };
    constexpr int kAhead = 8;   // pieces in flight (28 matrices, 0.2 G bf16 elements: 102 -> 94 us)
    for (; i + (kAhead - 1) * kElemThreads * kVec + kVec <= end; i += kAhead * kElemThreads * kVec) {
        uint4 raw[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) raw[q] = *reinterpret_cast<const uint4*>(src + i + q * kElemThreads * kVec);
#pragma unroll
        for (int q = 0; q < kAhead; ++q) take(raw[q]);
    }
    for (; i + kVec <= end; i += kElemThreads * kVec) take(*reinterpret_cast<const uint4*>(src + i));
    for (; i < end; ++i) { const float f = as_bf16(src + i); acc = fmaf(f, f, acc); }   // (at most one thread)
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int w = 0; w < kElemThreads / 32; ++w) t += red[w];
        parts[blockIdx.y * kNormParts + blockIdx.x] = t;
    }
}

// x0 <- bf16(src) / max(norm, eps), wide and padded with zeros; norm and quotient rounded to bf16 as torch's
// x.div_(x.norm().clamp(min=eps)) on a bf16 tensor rounds them (reference: gefen_muon.py:38). The quotient goes through the
// norm's reciprocal where that gives the same bits (NormDivider): 28 matrices, 0.2 G bf16 elements, 204 -> 164 us; 24 fp32
// matrices, 42 M elements, 59 -> 54.
template <typename S>
__global__ void __launch_bounds__(kElemThreads) ns_normalise_kernel(const NsMatrix* __restrict__ table, const float* __restrict__ parts, float eps) {
    __shared__ __align__(16) __nv_bfloat16 tile[kTile][kTilePitch];
    __shared__ float norm_shared;
    const NsMatrix& m = table[blockIdx.y];
    if (threadIdx.x < 32) {
        float t = parts[blockIdx.y * kNormParts + threadIdx.x] + parts[blockIdx.y * kNormParts + 32 + threadIdx.x];
        t = warp_sum(t);
        if (threadIdx.x == 0) {
            const float n = __bfloat162float(__float2bfloat16_rn(sqrtf(t))), least = __bfloat162float(__float2bfloat16_rn(eps));
            norm_shared = n < least ? least : n;   // (a NaN norm stays one, as torch's clamp leaves it)
        }
    }
    __syncthreads();
    const NormDivider quotient(norm_shared);
    const S* src = static_cast<const S*>(m.src);
    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(m.x0);
    const int rows = static_cast<int>(m.rows), cols = static_cast<int>(m.cols);
    const int wr = ns_wide_rows(m), wc = ns_wide_cols(m);
    if (!ns_tall(m) && wr == rows && wc == cols) {
        const long long chunks = m.rows * m.cols / 8;
        for (long long c = static_cast<long long>(blockIdx.x) * kElemThreads + threadIdx.x; c < chunks; c += static_cast<long long>(gridDim.x) * kElemThreads) {
            uint32_t w[4];
            alignas(16) S v[8];
            constexpr int kWide = static_cast<int>(sizeof(S)) / 2;   // 16-byte pieces of eight values
#pragma unroll
            for (int q = 0; q < kWide; ++q) reinterpret_cast<uint4*>(v)[q] = reinterpret_cast<const uint4*>(src)[kWide * c + q];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(quotient(as_bf16(v + 2 * e)), quotient(as_bf16(v + 2 * e + 1)));
                w[e] = *reinterpret_cast<const uint32_t*>(&h);
            }
            reinterpret_cast<uint4*>(dst)[c] = make_uint4(w[0], w[1], w[2], w[3]);
        }
        return;
    }
    // any other matrix tile by tile of the wide result, through shared memory where it is transposed
    const int tiles_c = (wc + kTile - 1) / kTile, tiles = tiles_c * ((wr + kTile - 1) / kTile);
    const int x = threadIdx.x % kTile, y0 = threadIdx.x / kTile;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int r0 = t / tiles_c * kTile, c0 = t % tiles_c * kTile;
        if (ns_tall(m)) {
            __syncthreads();
            // a thread reads eight columns of source row c0 + x (16 or 32 bytes where rows start on 16) and leaves them
            // in the tile transposed: neighbouring threads write neighbouring elements
            const bool vec = cols % 8 == 0;
            for (int piece = y0; piece < kTile / 8; piece += kElemThreads / kTile) {
                float f[8];
                const int row = c0 + x, col = r0 + 8 * piece;
                const S* from = src + static_cast<long long>(row) * cols + col;
                if (vec && row < rows && col < cols) {
                    alignas(16) S v[8];
#pragma unroll
                    for (int q = 0; q < static_cast<int>(sizeof(S)) / 2; ++q) reinterpret_cast<uint4*>(v)[q] = reinterpret_cast<const uint4*>(from)[q];
#pragma unroll
                    for (int e = 0; e < 8; ++e) f[e] = quotient(as_bf16(v + e));
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) f[e] = row < rows && col + e < cols ? quotient(as_bf16(from + e)) : 0.0f;
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) tile[8 * piece + e][x] = __float2bfloat16_rn(f[e]);
            }
            __syncthreads();
            for (int i = threadIdx.x; i < kTile * kTile / 8; i += kElemThreads) {   // (wide columns come in eights)
                const int y = i / (kTile / 8), c = c0 + i % (kTile / 8) * 8;
                if (r0 + y < wr && c < wc)
                    *reinterpret_cast<uint4*>(dst + static_cast<long long>(r0 + y) * wc + c) = *reinterpret_cast<const uint4*>(&tile[y][c - c0]);
            }
        } else {
            for (int y = y0; y < kTile; y += kElemThreads / kTile) {
                if (r0 + y >= wr || c0 + x >= wc) continue;
                float f = 0.0f;
                if (r0 + y < rows && c0 + x < cols) f = quotient(as_bf16(src + static_cast<long long>(r0 + y) * cols + c0 + x));
                dst[static_cast<long long>(r0 + y) * wc + c0 + x] = __float2bfloat16_rn(f);
            }
        }
    }
}

struct ApplyPeers {
    int n;
    long long delta[GEFEN_B200_MAX_PEERS];
};

// p <- round(p * wd_mul); p <- round(p + alpha * u), u the (bf16) result of the iteration, which lies wide: what
// muon_apply_kernel does for one matrix (reference: gefen_muon.py:326-329), peer stores included.
template <typename S>
__global__ void __launch_bounds__(kElemThreads) ns_apply_kernel(const NsMatrix* __restrict__ table, int in_x1, const __grid_constant__ ApplyPeers peers) {
    __shared__ __align__(16) __nv_bfloat16 tile[kTile][kTilePitch];
    const NsMatrix& m = table[blockIdx.y];
    const __nv_bfloat16* u = static_cast<const __nv_bfloat16*>(in_x1 ? m.x1 : m.x0);
    S* p = static_cast<S*>(m.p);
    const float wd_mul = m.wd_mul, alpha = m.alpha;
    const bool decay = m.decay != 0;
    const int rows = static_cast<int>(m.rows), cols = static_cast<int>(m.cols);
    const int wr = ns_wide_rows(m), wc = ns_wide_cols(m);
    auto update = [&](float pv, float uv) {
        if (decay) pv = ScalarIO<S>::round(pv * wd_mul);
        return fmaf(alpha, uv, pv);
    };
    auto put = [&](long long at, float v) {
        ScalarIO<S>::store(p + at, v);
        for (int r = 0; r < peers.n; ++r) ScalarIO<S>::store(reinterpret_cast<S*>(reinterpret_cast<uintptr_t>(p + at) + peers.delta[r]), v);
    };
    if (!ns_tall(m) && wc == cols && wr == rows && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
        const long long chunks = m.rows * m.cols / 8;
        for (long long c = static_cast<long long>(blockIdx.x) * kElemThreads + threadIdx.x; c < chunks; c += static_cast<long long>(gridDim.x) * kElemThreads) {
            const uint4 raw = reinterpret_cast<const uint4*>(u)[c];
            const __nv_bfloat16* uv = reinterpret_cast<const __nv_bfloat16*>(&raw);
            constexpr int kWide = static_cast<int>(sizeof(S)) / 2;   // 16-byte pieces of eight parameters
            alignas(16) S v[8];
#pragma unroll
            for (int q = 0; q < kWide; ++q) reinterpret_cast<uint4*>(v)[q] = reinterpret_cast<const uint4*>(p)[kWide * c + q];
#pragma unroll
            for (int e = 0; e < 8; ++e) ScalarIO<S>::store(v + e, update(ScalarIO<S>::load(v + e), __bfloat162float(uv[e])));
#pragma unroll
            for (int q = 0; q < kWide; ++q) {
                reinterpret_cast<uint4*>(p)[kWide * c + q] = reinterpret_cast<uint4*>(v)[q];
                for (int r = 0; r < peers.n; ++r)
                    reinterpret_cast<uint4*>(reinterpret_cast<uintptr_t>(p) + peers.delta[r])[kWide * c + q] = reinterpret_cast<uint4*>(v)[q];
            }
        }
        return;
    }
    const int tiles_c = (cols + kTile - 1) / kTile, tiles = tiles_c * ((rows + kTile - 1) / kTile);   // of the parameter
    const int x = threadIdx.x % kTile, y0 = threadIdx.x / kTile;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int r0 = t / tiles_c * kTile, c0 = t % tiles_c * kTile;
        if (ns_tall(m)) {
            __syncthreads();
            for (int piece = y0; piece < kTile / 8; piece += kElemThreads / kTile) {   // eight columns of u row c0 + x
                const int row = c0 + x, col = r0 + 8 * piece;
                alignas(16) __nv_bfloat16 v[8] = {};
                if (row < wr && col < wc) *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(u + static_cast<long long>(row) * wc + col);
#pragma unroll
                for (int e = 0; e < 8; ++e) tile[8 * piece + e][x] = v[e];
            }
            __syncthreads();
            if (cols % 8 == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
                for (int i = threadIdx.x; i < kTile * kTile / 8; i += kElemThreads) {
                    const int y = i / (kTile / 8), c = c0 + i % (kTile / 8) * 8;
                    if (r0 + y >= rows || c >= cols) continue;
                    constexpr int kWide = static_cast<int>(sizeof(S)) / 2;
                    S* at = p + static_cast<long long>(r0 + y) * cols + c;
                    alignas(16) S v[8];
#pragma unroll
                    for (int q = 0; q < kWide; ++q) reinterpret_cast<uint4*>(v)[q] = reinterpret_cast<const uint4*>(at)[q];
#pragma unroll
                    for (int e = 0; e < 8; ++e) ScalarIO<S>::store(v + e, update(ScalarIO<S>::load(v + e), __bfloat162float(tile[y][c - c0 + e])));
#pragma unroll
                    for (int q = 0; q < kWide; ++q) {
                        reinterpret_cast<uint4*>(at)[q] = reinterpret_cast<uint4*>(v)[q];
                        for (int r = 0; r < peers.n; ++r)
                            reinterpret_cast<uint4*>(reinterpret_cast<uintptr_t>(at) + peers.delta[r])[q] = reinterpret_cast<uint4*>(v)[q];
                    }
                }
            } else {
                for (int y = y0; y < kTile; y += kElemThreads / kTile) {
                    if (r0 + y >= rows || c0 + x >= cols) continue;
                    const long long at = static_cast<long long>(r0 + y) * cols + c0 + x;
                    put(at, update(ScalarIO<S>::load(p + at), __bfloat162float(tile[y][x])));
                }
            }
        } else {
            for (int y = y0; y < kTile; y += kElemThreads / kTile) {
                if (r0 + y >= rows || c0 + x >= cols) continue;
                const long long at = static_cast<long long>(r0 + y) * cols + c0 + x;
                put(at, update(ScalarIO<S>::load(p + at), __bfloat162float(u[static_cast<long long>(r0 + y) * wc + c0 + x])));
            }
        }
    }
}

// The plan of a group: five lists of products (Gram matrix of x0 / of x1, polynomial, update x0 -> x1 / x1 -> x0) and
// two lists of tiles (of the symmetric m x m results, of the m x k results).
struct TileKind {
    int bm, bn;            // 256 x 256: pairs of CTAs
};
struct GroupShape {
    TileKind gram, update;
    int64_t gram_tiles, update_tiles, entries_bytes, bytes;
};
static void wide_dims(const NsMatrix& m, int* wr, int* wc) {
    const int64_t a = (m.rows + 7) / 8 * 8, b = (m.cols + 7) / 8 * 8;
    *wr = static_cast<int>(std::min(a, b));
    *wc = static_cast<int>(std::max(a, b));
}
// Kind of tiles for a list of products: the fewest rounds of the persistent CTAs, weighed with what a round of the kind
// takes (all kinds give the same bits). Chosen for the symmetric products and the updates apart. Five iterations of
// single matrices and groups, us, with the symmetric products forced to 256 x 256 / 128 x 256 / 128 x 128, then the updates:
//   768 x 2304        312 / 302 / 261     280 / 281 / 262        2048 x 6144      652 / 646 / 608     616 / 622 / 754
//   2048 x 2048       402 / 382 / 360     358 / 352 / 391        2560 x 2560      524 / 513 / 616     522 / 534 / 571
//   4096 x 4096       1357 / 1378 / 1787  1318 / 1420 / 1718     8 of 1024 x 4096 862 / 879 / 785     821 / 867 / 966
// (One kind for all products, the first whose symmetric tiles fill the GPU, took 797 us for 2048 x 6144 and 436 for
// 2048 x 2048 where this rule takes 620 and 355.)
static TileKind choose_tiles(const NsMatrix* mats, int n, bool symmetric, int64_t* tiles) {
    static const struct { TileKind kind; double round; } kinds[3] = {{{256, 256}, 1.0}, {{128, 256}, 1.15}, {{128, 128}, 0.88}};
    TileKind best = {};
    double least = 0.0;
    for (const auto& k : kinds) {
        int64_t count = 0;
        for (int i = 0; i < n; ++i) {
            int m, c;
            wide_dims(mats[i], &m, &c);
            count += count_tiles(m, symmetric ? m : c, k.kind.bm, k.kind.bn, symmetric);
        }
        const int64_t at_once = k.kind.bm == 256 ? sm_count() / 2 : sm_count();
        const double cost = static_cast<double>((count + at_once - 1) / at_once) * k.round;
        if (best.bm == 0 || cost < least) {
            best = k.kind;
            least = cost;
            *tiles = count;
        }
    }
    return best;
}
static GroupShape group_shape(const NsMatrix* mats, int n) {
    GroupShape g;
    g.gram = choose_tiles(mats, n, true, &g.gram_tiles);
    g.update = choose_tiles(mats, n, false, &g.update_tiles);
    g.entries_bytes = static_cast<int64_t>(5) * n * static_cast<int64_t>(sizeof(GroupEntry));
    g.bytes = g.entries_bytes + (g.gram_tiles + g.update_tiles) * static_cast<int64_t>(sizeof(GroupTile));
    return g;
}
static int check_group(const NsMatrix* mats, int n) {
    GEFEN_CHECK_ARG(n >= 1 && n <= GEFEN_B200_NS_GROUP_MATRICES && mats != nullptr, "Expected between 1 and %d matrices, got %d.",
                    GEFEN_B200_NS_GROUP_MATRICES, n);
    for (int i = 0; i < n; ++i) {
        GEFEN_CHECK_ARG(mats[i].rows > 0 && mats[i].cols > 0 && mats[i].rows <= (1 << 30) && mats[i].cols <= (1 << 30),
                        "Matrix %d has bad dimensions.", i);
        GEFEN_CHECK_ARG(mats[i].x0 && mats[i].x1 && mats[i].gram && mats[i].poly, "Matrix %d has a null buffer.", i);
        GEFEN_CHECK_ARG(aligned16(mats[i].x0) && aligned16(mats[i].x1) && aligned16(mats[i].gram) && aligned16(mats[i].poly),
                        "Matrix %d has a buffer that is not 16-byte aligned.", i);
    }
    return GEFEN_B200_OK;
}

static int build_group_plan(const NsMatrix* mats, int n, const GroupShape& g, std::vector<unsigned char>& image) {
    image.assign(static_cast<size_t>(g.bytes), 0);
    GroupEntry* entries = reinterpret_cast<GroupEntry*>(image.data());
    GroupTile* gram_tiles = reinterpret_cast<GroupTile*>(image.data() + g.entries_bytes);
    GroupTile* update_tiles = gram_tiles + g.gram_tiles;
    std::vector<int> order(n);   // longest products first: the last wave is made of the short ones
    for (int i = 0; i < n; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return std::max(mats[x].rows, mats[x].cols) > std::max(mats[y].rows, mats[y].cols);
    });
    int64_t gt = 0, ut = 0;
    for (int i = 0; i < n; ++i) {
        const NsMatrix& mat = mats[order[i]];
        int m, k;
        wide_dims(mat, &m, &k);
        CUtensorMap x[2], x_mn[2], gram, poly;
        void* xs[2] = {mat.x0, mat.x1};
        int rc;
        for (int q = 0; q < 2; ++q) {
            if ((rc = make_map(&x[q], xs[q], m, k, k, kBM)) != GEFEN_B200_OK) return rc;
            if ((rc = make_map(&x_mn[q], xs[q], m, k, k, kBK)) != GEFEN_B200_OK) return rc;
        }
        if ((rc = make_map(&gram, mat.gram, m, m, m, kBM)) != GEFEN_B200_OK) return rc;
        if ((rc = make_map(&poly, mat.poly, m, m, m, kBM)) != GEFEN_B200_OK) return rc;
        auto fill = [&](int list, const CUtensorMap& a, const CUtensorMap& b, const void* c, void* d, int N, int K) {
            GroupEntry& e = entries[list * n + i];
            e.a = a;
            e.b = b;
            e.c = static_cast<const __nv_bfloat16*>(c);
            e.d = static_cast<__nv_bfloat16*>(d);
            e.M = m; e.N = N; e.K = K;
            e.ldc = N; e.ldd = N;
        };
        fill(0, x[0], x[0], nullptr, mat.gram, m, k);
        fill(1, x[1], x[1], nullptr, mat.gram, m, k);
        fill(2, gram, gram, mat.gram, mat.poly, m, m);
        fill(3, poly, x_mn[0], mat.x0, mat.x1, k, m);
        fill(4, poly, x_mn[1], mat.x1, mat.x0, k, m);
        int m0, n0;
        for (int64_t t = 0; tile_coords(m, m, g.gram.bm, g.gram.bn, 1, t, &m0, &n0); ++t) gram_tiles[gt++] = {i, m0, n0, 0};
        for (int64_t t = 0; tile_coords(m, k, g.update.bm, g.update.bn, 0, t, &m0, &n0); ++t) update_tiles[ut++] = {i, m0, n0, 0};
    }
    return GEFEN_B200_OK;
}

template <bool B_MN>
static int launch_group(const TileKind& kind, GemmArgs args, cudaStream_t stream) {
    if (kind.bm == 256) {
        constexpr int smem = kPairStages * (kBM + kPairBN / 2) * kBK * 2 + 4 * 32 * kStagePitch * 2 + 1024;
        static std::once_flag configured[64];
        int dev = 0;
        GEFEN_CHECK_CUDA(cudaGetDevice(&dev));
        GEFEN_CHECK_ARG(dev >= 0 && dev < 64, "Unsupported device ordinal %d.", dev);
        cudaError_t err = cudaSuccess;
        std::call_once(configured[dev], [&] {
            err = cudaFuncSetAttribute(ns_gemm_pair_kernel<B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        });
        GEFEN_CHECK_CUDA(err);
        const int pairs = std::min(args.n_tiles, sm_count() / 2);
        return launch_product(ns_gemm_pair_kernel<B_MN>, 2 * pairs, smem, stream, args);
    }
    const CUtensorMap none = {};
    if (kind.bn == 256) return launch_gemm_variant<256, 4, false, B_MN, true, true>(none, none, args, stream);
    return launch_gemm_variant<128, 6, false, B_MN, true, true>(none, none, args, stream);
}

// Tables travel as kernel parameters, one launch per kUploadBytes: no host memory that a copy reads later (a pageable
// copy of more than 64 KB first waits for the stream), and a captured upload carries its bytes with it.
constexpr int kUploadBytes = 4000;
struct UploadPiece {
    uint4 word[kUploadBytes / 16];
};
__global__ void __launch_bounds__(256) upload_kernel(uint4* __restrict__ dst, int words, const __grid_constant__ UploadPiece piece) {
    if (static_cast<int>(threadIdx.x) < words) dst[threadIdx.x] = piece.word[threadIdx.x];
    asm volatile("fence.proxy.tensormap::generic.release.gpu;" ::: "memory");   // (there may be tensor maps among the words)
}
static_assert(kUploadBytes % 16 == 0 && kUploadBytes / 16 <= 256 && sizeof(UploadPiece) + 16 <= 4096, "one word per thread, kernel parameter space");
constexpr int64_t kMostUploadLaunches = 64;

}  // namespace gefen

extern "C" int gefen_b200_upload(void* dst, const void* src, int64_t bytes, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    GEFEN_CHECK_ARG(bytes >= 0 && bytes % 16 == 0, "Expected a multiple of 16 bytes.");
    if (bytes == 0) return GEFEN_B200_OK;
    GEFEN_CHECK_ARG(dst != nullptr && src != nullptr && aligned16(dst), "Expected a source and a 16-byte aligned destination.");
    if (bytes > kMostUploadLaunches * kUploadBytes) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        GEFEN_CHECK_CUDA(cudaStreamIsCapturing(stream, &capture));
        if (capture == cudaStreamCaptureStatusNone) {
            GEFEN_CHECK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream));
            return GEFEN_B200_OK;
        }
    }
    UploadPiece piece;
    for (int64_t done = 0; done < bytes; done += kUploadBytes) {
        const int n = static_cast<int>(std::min<int64_t>(bytes - done, kUploadBytes));
        memcpy(piece.word, static_cast<const unsigned char*>(src) + done, n);
        upload_kernel<<<1, 256, 0, stream>>>(reinterpret_cast<uint4*>(static_cast<unsigned char*>(dst) + done), n / 16, piece);
    }
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}

extern "C" int gefen_b200_ns_matrix_size(void) { return static_cast<int>(sizeof(gefen_b200_ns_matrix_t)); }

extern "C" int64_t gefen_b200_ns_group_plan_bytes(const gefen_b200_ns_matrix_t* mats, int n) {
    if (check_group(mats, n) != GEFEN_B200_OK) return 0;
    return group_shape(mats, n).bytes;
}

extern "C" int gefen_b200_ns_group_plan(const gefen_b200_ns_matrix_t* mats, int n, void* host_plan) {
    int rc = check_group(mats, n);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(host_plan != nullptr, "Expected a non-null plan buffer.");
    try {
        std::vector<unsigned char> image;
        const GroupShape g = group_shape(mats, n);
        rc = build_group_plan(mats, n, g, image);
        if (rc == GEFEN_B200_OK) memcpy(host_plan, image.data(), image.size());
        return rc;
    } catch (const std::bad_alloc&) {
        return fail(GEFEN_B200_ERUNTIME, "Out of host memory for the plan of %d matrices.", n);
    }
}

extern "C" int gefen_b200_ns_group(const gefen_b200_ns_matrix_t* mats, int n, const void* device_mats, const void* device_plan,
                                   float* partials, int src_dtype, int steps, double a, double b, double c, double eps, int* status,
                                   void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_group(mats, n);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(device_mats && device_plan && partials && aligned16(device_mats) && (reinterpret_cast<uintptr_t>(device_plan) & 63u) == 0,
                    "Expected non-null tables, the plan on a 64-byte boundary.");
    GEFEN_CHECK_ARG(steps >= 0 && steps < 100, "Number of steps must be less than 100.");
    for (int i = 0; i < n; ++i) GEFEN_CHECK_ARG(mats[i].src != nullptr && aligned16(mats[i].src), "Matrix %d needs a 16-byte aligned source.", i);
    const GroupShape g = group_shape(mats, n);
    const NsMatrix* table = static_cast<const NsMatrix*>(device_mats);
    int64_t most = 1;
    for (int i = 0; i < n; ++i) most = std::max(most, (mats[i].rows + 7) * (mats[i].cols + 7));
    const dim3 elem(static_cast<unsigned>(std::min<int64_t>((most + 4095) / 4096, 4 * sm_count())), static_cast<unsigned>(n));
    switch (src_dtype) {
#define GEFEN_NS_SRC(tag, S)                                                                         \
    case tag:                                                                                        \
        ns_norm_kernel<S><<<dim3(kNormParts, n), kElemThreads, 0, stream>>>(table, partials);        \
        ns_normalise_kernel<S><<<elem, kElemThreads, 0, stream>>>(table, partials, static_cast<float>(eps)); \
        break;
        GEFEN_NS_SRC(GEFEN_B200_F32, float)
        GEFEN_NS_SRC(GEFEN_B200_F16, __half)
        GEFEN_NS_SRC(GEFEN_B200_BF16, __nv_bfloat16)
        GEFEN_NS_SRC(GEFEN_B200_F64, double)
#undef GEFEN_NS_SRC
        default: return fail(GEFEN_B200_EINVAL, "Unsupported source dtype tag %d.", src_dtype);
    }
    GEFEN_CHECK_CUDA(cudaGetLastError());
    const GroupEntry* entries = static_cast<const GroupEntry*>(device_plan);
    const GroupTile* tiles = reinterpret_cast<const GroupTile*>(static_cast<const unsigned char*>(device_plan) + g.entries_bytes);
    for (int it = 0; it < steps; ++it) {
        GemmArgs args = {};
        args.status = status;
        // G = X X^T ; B = b G + c G G ; X' = a X + B X
        args.tiles = tiles;
        args.n_tiles = static_cast<int>(g.gram_tiles);
        args.symmetric = 1;
        args.entries = entries + (it & 1) * n;
        args.alpha = 1.0f;
        args.beta = 0.0f;
        if ((rc = launch_group<false>(g.gram, args, stream)) != GEFEN_B200_OK) return rc;
        args.entries = entries + 2 * n;
        args.alpha = static_cast<float>(c);
        args.beta = static_cast<float>(b);
        if ((rc = launch_group<false>(g.gram, args, stream)) != GEFEN_B200_OK) return rc;
        args.tiles = tiles + g.gram_tiles;
        args.n_tiles = static_cast<int>(g.update_tiles);
        args.symmetric = 0;
        args.entries = entries + (3 + (it & 1)) * n;
        args.alpha = 1.0f;
        args.beta = static_cast<float>(a);
        if ((rc = launch_group<true>(g.update, args, stream)) != GEFEN_B200_OK) return rc;
    }
    return GEFEN_B200_OK;
}

extern "C" int gefen_b200_ns_group_apply(const gefen_b200_ns_matrix_t* mats, int n, const void* device_mats, int dtype, int steps,
                                         const int64_t* peer_deltas, int n_peers, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_group(mats, n);
    if (rc != GEFEN_B200_OK) return rc;
    GEFEN_CHECK_ARG(device_mats != nullptr, "Expected a non-null table.");
    GEFEN_CHECK_ARG(n_peers >= 0 && n_peers <= GEFEN_B200_MAX_PEERS, "Expected between 0 and %d peers, got %d.", GEFEN_B200_MAX_PEERS, n_peers);
    GEFEN_CHECK_ARG(n_peers == 0 || peer_deltas != nullptr, "Expected peer offsets for %d peers.", n_peers);
    ApplyPeers peers = {};
    peers.n = n_peers;
    for (int r = 0; r < n_peers; ++r) {
        GEFEN_CHECK_ARG(peer_deltas[r] % 16 == 0, "Peer offset %d is not a multiple of 16 bytes.", r);
        peers.delta[r] = peer_deltas[r];
    }
    int64_t most = 1;
    for (int i = 0; i < n; ++i) {
        GEFEN_CHECK_ARG(mats[i].p != nullptr, "Matrix %d has no parameter.", i);
        most = std::max(most, mats[i].rows * mats[i].cols);
    }
    const dim3 elem(static_cast<unsigned>(std::min<int64_t>((most + 4095) / 4096, 4 * sm_count())), static_cast<unsigned>(n));
    const NsMatrix* table = static_cast<const NsMatrix*>(device_mats);
    const int in_x1 = steps & 1;
    switch (dtype) {
        case GEFEN_B200_F32: ns_apply_kernel<float><<<elem, kElemThreads, 0, stream>>>(table, in_x1, peers); break;
        case GEFEN_B200_F16: ns_apply_kernel<__half><<<elem, kElemThreads, 0, stream>>>(table, in_x1, peers); break;
        case GEFEN_B200_BF16: ns_apply_kernel<__nv_bfloat16><<<elem, kElemThreads, 0, stream>>>(table, in_x1, peers); break;
        default: return fail(GEFEN_B200_EINVAL, "The GefenMuon apply supports fp32, fp16 and bf16 parameters.");
    }
    GEFEN_CHECK_CUDA(cudaGetLastError());
    return GEFEN_B200_OK;
}
