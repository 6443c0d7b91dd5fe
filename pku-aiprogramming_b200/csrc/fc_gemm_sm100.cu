// Fully connected layer GEMMs for sm_100a: C[M,N] = op(A) op(B) (+ bias), bf16 in, fp32
// accumulation in tensor memory, bf16 out.
//
// The reference's FcForward / FcBackward (src/Layers.cu:9-79 of the reference project) are
// cublasSgemm calls that create and destroy a handle and synchronise the device per call
// (src/Layers_kernels.cu:10-30), with the bias added by a second rank-1 GEMM against a ones
// vector.  Here one persistent kernel serves the three products of the layer
//     forward   y  = x W + b        A = x  [M,K]  K-major,   B = W  [K,N]  MN-major
//     backward  dx = dy W^T         A = dy [M,N]  K-major,   B = W  [K,N]  K-major (as [N_out rows of K])
//               dW = x^T dy         A = x  [M,K]  MN-major,  B = dy [M,N]  MN-major
// straight from the row-major tensors (no transposed copies), the bias joins in the epilogue,
// and db = column sums of dy is one small HBM-bound reduction.
//
// Kernel structure (192 threads, one CTA per SM, static round-robin over 128x256 output tiles in
// bands of 16 tile rows so that one wave of CTAs shares its operand panels in L2):
//   warp 0      TMA producer: 4-stage ring of {A 128x64, B 256x64} bf16 tiles, 128-byte swizzle
//   warp 1      issues tcgen05.mma (M128 N256 K16, 4 per stage); a commit frees the stage, a
//               commit per tile hands the accumulator to the epilogue
//   warps 2-5   epilogue: accumulator (256 tensor-memory columns, double buffered so the next
//               tile's MMAs run meanwhile) -> registers -> + bias -> bf16 -> global
// Every wait is bounded (see sm100_ptx.cuh); an expired wait aborts the CTA through the common exit.
#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>

#include "common.h"
#include "fc_tiles.cuh"
#include "sm100_ptx.cuh"

namespace ttk {
using namespace sm100;

namespace {

constexpr int kBM = 128, kBN = 256, kBK = 64, kStages = 4;
constexpr int kABytes = kBM * kBK * 2;          // 16 KB
constexpr int kBBytes = kBN * kBK * 2;          // 32 KB
constexpr int kStageBytes = kABytes + kBBytes;  // 48 KB
constexpr int kSubBytes = 64 * 128;             // one 64-wide MN-major sub-block: 64 K-rows x 128 B
constexpr int kGemmSmem = kStages * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
constexpr int kSplitPitch = kBN + 4;             // floats; rows of a share's accumulator in shared memory
static_assert(kBM * kSplitPitch * 4 <= kStages * kStageBytes, "a share's accumulator takes the ring's place");

// One thread's accumulator row (256 fp32 columns of tensor memory starting at `taddr`) -> + bias -> bf16 ->
// row `row` of C, columns n0...  Hands the accumulator buffer back (one arrival: on `acc_empty` of this CTA,
// or, in a CTA pair, on the barrier at `acc_empty_cluster` in the pair's rank-0 CTA) as soon as the row has
// been read.
template <bool kPair>
__device__ __forceinline__ void store_acc_row(uint32_t taddr, long long row, int n0, __nv_bfloat16* __restrict__ C,
                                              const __nv_bfloat16* __restrict__ bias, int M, int N, int wide,
                                              uint64_t* acc_empty, uint32_t acc_empty_cluster) {
    __nv_bfloat16* crow = C + row * (long long)N;
#pragma unroll 1
    for (int c = 0; c < kBN / 32; ++c) {
        uint32_t r[32];
        tmem_ld32(taddr + (uint32_t)(c * 32), r);
        tmem_wait_ld();
        if (c == kBN / 32 - 1) {   // this thread has read its whole accumulator row
            tc_fence_before();
            if (kPair) mbar_arrive_cluster(acc_empty_cluster);
            else mbar_arrive(acc_empty);
        }
        const int col0 = n0 + c * 32;
        if (row < M) {
#pragma unroll
            for (int g2 = 0; g2 < 2; ++g2) {
                uint32_t o8[8];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int g = g2 * 2 + h;
                    const int col = col0 + g * 8;
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[g * 8 + e]);
                    if (bias && col < N) {
                        const uint4 bb = *reinterpret_cast<const uint4*>(bias + col);
                        const uint32_t bw[4] = {bb.x, bb.y, bb.z, bb.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            v[2 * e] += __uint_as_float(bw[e] << 16);
                            v[2 * e + 1] += __uint_as_float(bw[e] & 0xffff0000u);
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) o8[h * 4 + e] = pack_bf16x2(v[2 * e], v[2 * e + 1]);
                }
                // N % 8 == 0: a group of 8 columns is inside or outside as a whole
                const int col = col0 + g2 * 16;
                if (wide && col + 16 <= N) {
                    st_global_32B(crow + col, o8);   // one full sector per lane and instruction
                } else {
                    if (col < N) *reinterpret_cast<uint4*>(crow + col) = make_uint4(o8[0], o8[1], o8[2], o8[3]);
                    if (col + 8 < N) *reinterpret_cast<uint4*>(crow + col + 8) = make_uint4(o8[4], o8[5], o8[6], o8[7]);
                }
            }
        }
    }
}

// kSplit: launched as clusters, one output tile per cluster.  Each CTA sums its share of K; the shares' accumulators go to
// shared memory (the ring is empty by then), and each CTA adds up its rows of the tile through distributed shared memory,
// in rank order.  No workspace and no second launch, where few tiles over a long K (the weight gradient of a narrow layer)
// would leave most SMs idle.
template <bool kAMn, bool kBMn, bool kSplit>
__global__ void __launch_bounds__(192, 1)
fc_gemm_sm100_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     __nv_bfloat16* __restrict__ C, const __nv_bfloat16* __restrict__ bias, int M, int N, int K,
                     int tiles_m, int tiles_n, int wide, unsigned int* status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
    uint64_t* full = bars;                    // [kStages] producer -> MMA
    uint64_t* empty = bars + kStages;         // [kStages] MMA -> producer
    uint64_t* acc_full = bars + 2 * kStages;  // [2] MMA -> epilogue
    uint64_t* acc_empty = acc_full + 2;       // [2] epilogue -> MMA (128 arrivals)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = uniform_warp_idx(), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 128);
        }
        fence_barrier_init();
        fence_proxy_async_smem();
    }
    __syncwarp();
    if (warp == 0) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
        if (elect_one()) {
            tma_prefetch_desc(&tmA);
            tma_prefetch_desc(&tmB);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    WaitCtx wctx{status, abort_flag, warp};
    grid_let_next_start();
    grid_wait_for_previous();

    namespace cg = cooperative_groups;
    const int total = tiles_m * tiles_n;
    const int n_cta = kSplit ? (int)cg::this_cluster().num_blocks() : 1, rank = kSplit ? (int)cg::this_cluster().block_rank() : 0;
    const int t_first = kSplit ? (int)blockIdx.x / n_cta : (int)blockIdx.x, t_step = kSplit ? total : (int)gridDim.x;
    const int all_blocks = (K + kBK - 1) / kBK, share = (all_blocks + n_cta - 1) / n_cta;
    const int kb_first = rank * share, kblocks = max(0, min(share, all_blocks - kb_first));

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        int it = 0;
        bool live = true;
        for (int t = t_first; t < total && live; t += t_step) {
            int mb, nb;
            fc_tile_coords(t, tiles_m, tiles_n, mb, nb);
            const int m0 = mb * kBM, n0 = nb * kBN;
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const int s = it % kStages;
                const uint32_t ph = (uint32_t)(it / kStages) & 1u;
                if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ph ^ 1u, wctx, 10 + s, it))) {
                    live = false;
                    break;
                }
                if (elect_one()) {
                    unsigned char* sA = smem + s * kStageBytes;
                    unsigned char* sB = sA + kABytes;
                    const int k0 = (kb_first + kb) * kBK;
                    mbar_arrive_expect_tx(&full[s], kStageBytes);
                    if (kAMn) {
                        tma_load_3d(sA, &tmA, &full[s], m0, k0, 0);
                        tma_load_3d(sA + kSubBytes, &tmA, &full[s], m0 + 64, k0, 0);
                    } else {
                        tma_load_3d(sA, &tmA, &full[s], k0, m0, 0);
                    }
                    if (kBMn) {
#pragma unroll
                        for (int j = 0; j < kBN / 64; ++j) tma_load_3d(sB + j * kSubBytes, &tmB, &full[s], n0 + 64 * j, k0, 0);
                    } else {
                        tma_load_3d(sB, &tmB, &full[s], k0, n0, 0);
                    }
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        constexpr uint32_t idesc = umma_idesc_bf16(kBM, kBN, kAMn, kBMn);
        constexpr uint32_t a_step = kAMn ? 2048u : 32u;   // one K=16 step inside the stage
        constexpr uint32_t b_step = kBMn ? 2048u : 32u;
        int it = 0, lt = 0;
        bool live = true;
        for (int t = t_first; t < total && live; t += t_step, ++lt) {
            const int buf = lt & 1;
            const uint32_t use = (uint32_t)(lt >> 1) & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], use ^ 1u, wctx, 30 + buf, lt))) break;
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)buf * kBN;
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const int s = it % kStages;
                const uint32_t ph = (uint32_t)(it / kStages) & 1u;
                if (!__all_sync(0xffffffffu, mbar_wait(&full[s], ph, wctx, 20 + s, it))) {
                    live = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sA = smem_u32(smem + s * kStageBytes);
                const uint32_t sB = sA + kABytes;
                const uint32_t a0 = umma_desc_lo(sA, kAMn ? kSubBytes : 16), b0 = umma_desc_lo(sB, kBMn ? kSubBytes : 16);
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; ++kk)
                        umma_ss_one(d_tmem, a0 + (kk * a_step >> 4), b0 + (kk * b_step >> 4), umma_desc_hi(1024), idesc,
                                    (uint32_t)((kb | kk) != 0));
                }
                __syncwarp();
                tc_commit(&empty[s]);
            }
            if (live) tc_commit(&acc_full[buf]);
        }
    } else {
        // ------------------------------------------------------------------ epilogue (warps 2..5)
        const int lane_group = warp & 3;                 // tensor-memory lanes 32*lane_group .. +31
        const uint32_t lane_off = (uint32_t)(lane_group * 32) << 16;
        int lt = 0;
        for (int t = t_first; t < total; t += t_step, ++lt) {
            int mb, nb;
            fc_tile_coords(t, tiles_m, tiles_n, mb, nb);
            const int buf = lt & 1;
            const uint32_t use = (uint32_t)(lt >> 1) & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[buf], use, wctx, 40 + buf, lt))) break;
            tc_fence_after();
            if (kSplit) {
                float* dst = reinterpret_cast<float*>(smem) + (lane_group * 32 + lane) * kSplitPitch;
#pragma unroll 1
                for (int c = 0; c < kBN; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(tmem_base + lane_off + (uint32_t)c, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 32; e += 4)   // a share without blocks has no accumulator
                        *reinterpret_cast<uint4*>(dst + c + e) = kblocks > 0 ? make_uint4(v[e], v[e + 1], v[e + 2], v[e + 3]) : make_uint4(0u, 0u, 0u, 0u);
                }
                break;
            }
            const long long row = (long long)mb * kBM + lane_group * 32 + lane;
            store_acc_row<false>(tmem_base + lane_off + (uint32_t)(buf * kBN), row, nb * kBN, C, bias, M, N, wide,
                                 &acc_empty[buf], 0u);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if (kSplit) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();   // every share's accumulator is in shared memory
        int mb, nb;
        fc_tile_coords(t_first, tiles_m, tiles_n, mb, nb);
        const int rows = kBM / n_cta;
        float* tile = reinterpret_cast<float*>(smem);
        for (int i = threadIdx.x; i < rows * (kBN / 8); i += 192) {
            const int r = rank * rows + i / (kBN / 8), c = (i % (kBN / 8)) * 8, m = mb * kBM + r, n = nb * kBN + c;
            if (m >= M || n >= N) continue;   // N % 8 == 0: a group of 8 columns is inside or outside as a whole
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int q = 0; q < n_cta; ++q) {
                const float4* x = reinterpret_cast<const float4*>(cluster.map_shared_rank(tile, q) + r * kSplitPitch + c);
                const float4 x0 = x[0], x1 = x[1];
                v[0] += x0.x; v[1] += x0.y; v[2] += x0.z; v[3] += x0.w;
                v[4] += x1.x; v[5] += x1.y; v[6] += x1.z; v[7] += x1.w;
            }
            if (bias) {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] += __bfloat162float(bias[n + e]);
            }
            *reinterpret_cast<uint4*>(C + (long long)m * N + n) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
        }
        __syncwarp();
        cluster.sync();   // a peer may still be reading this CTA's share
    }
}

// ---- the same GEMM on CTA pairs (clusters of two, tcgen05 cta_group::2) ----------------------------------
// A pair owns a 256x256 output tile: CTA r of the pair holds rows [128r, 128r+128) of the A tile and
// rows [128r, 128r+128) of the B tile's N extent, so every K=64 stage is 16 KB + 16 KB per CTA and a
// M256 N256 K16 instruction reads 8 KB of shared memory per SM in its 128 cycles (64 B/clk, against
// 96 B/clk for the one-CTA 128x256 tile).  Both CTAs run the TMA producer (their loads count on the
// rank-0 CTA's `full` barrier) and the epilogue (each drains its own 128 accumulator rows); only the
// rank-0 CTA issues MMAs, and hands stages and accumulators back to both CTAs with one commit each.
constexpr int kPStages = 6;
constexpr int kPABytes = 128 * kBK * 2;             // 16 KB: this CTA's 128 rows of A
constexpr int kPBBytes = 128 * kBK * 2;             // 16 KB: this CTA's half of the 256 B rows
constexpr int kPStageBytes = kPABytes + kPBBytes;   // 32 KB
constexpr int kPairSmem = kPStages * kPStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;

template <bool kAMn, bool kBMn>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(192, 1)
fc_gemm_pair_sm100_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          __nv_bfloat16* __restrict__ C, const __nv_bfloat16* __restrict__ bias, int M, int N, int K,
                          int tiles_m, int tiles_n, int wide, unsigned int* status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kPStages * kPStageBytes);
    uint64_t* full = bars;                     // [kPStages] both producers -> MMA (the rank-0 CTA's copy is used)
    uint64_t* empty = bars + kPStages;         // [kPStages] MMA -> this CTA's producer
    uint64_t* acc_full = bars + 2 * kPStages;  // [2] MMA -> this CTA's epilogue
    uint64_t* acc_empty = acc_full + 2;        // [2] both epilogues -> MMA (256 arrivals; rank-0 CTA's copy)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = uniform_warp_idx(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < kPStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 256);
        }
        fence_barrier_init();
        fence_proxy_async_smem();
    }
    __syncwarp();
    if (warp == 0) {
        tmem_alloc_pair(tmem_slot, 512);
        tmem_relinquish_pair();
        if (elect_one()) {
            tma_prefetch_desc(&tmA);
            tma_prefetch_desc(&tmB);
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer's barriers are initialised and its tensor memory allocated
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    WaitCtx wctx{status, abort_flag, warp};
    grid_let_next_start();
    grid_wait_for_previous();

    const int total = tiles_m * tiles_n;   // 256x256 tiles
    const int kblocks = (K + kBK - 1) / kBK;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (both CTAs)
        int it = 0;
        bool live = true;
        for (int t = pair; t < total && live; t += n_pairs) {
            int mb, nb;
            fc_tile_coords(t, tiles_m, tiles_n, mb, nb);
            const int m0 = mb * 256 + (int)rank * 128, n0 = nb * 256 + (int)rank * 128;
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const int s = it % kPStages;
                const uint32_t ph = (uint32_t)(it / kPStages) & 1u;
                if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ph ^ 1u, wctx, 10 + s, it))) {
                    live = false;
                    break;
                }
                if (elect_one()) {
                    unsigned char* sA = smem + s * kPStageBytes;
                    unsigned char* sB = sA + kPABytes;
                    const int k0 = kb * kBK;
                    if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * kPStageBytes);   // both CTAs' bytes
                    const uint32_t full0 = map_to_cta(smem_u32(&full[s]), 0);
                    if (kAMn) {
                        tma_load_3d_pair(sA, &tmA, full0, m0, k0, 0);
                        tma_load_3d_pair(sA + kSubBytes, &tmA, full0, m0 + 64, k0, 0);
                    } else {
                        tma_load_3d_pair(sA, &tmA, full0, k0, m0, 0);
                    }
                    if (kBMn) {
                        tma_load_3d_pair(sB, &tmB, full0, n0, k0, 0);
                        tma_load_3d_pair(sB + kSubBytes, &tmB, full0, n0 + 64, k0, 0);
                    } else {
                        tma_load_3d_pair(sB, &tmB, full0, k0, n0, 0);
                    }
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (rank-0 CTA only)
        if (rank == 0) {
            constexpr uint32_t idesc = umma_idesc_bf16(256, 256, kAMn, kBMn);
            constexpr uint32_t a_step = kAMn ? 2048u : 32u;   // one K=16 step inside the stage
            constexpr uint32_t b_step = kBMn ? 2048u : 32u;
            int it = 0, lt = 0;
            bool live = true;
            for (int t = pair; t < total && live; t += n_pairs, ++lt) {
                const int buf = lt & 1;
                const uint32_t use = (uint32_t)(lt >> 1) & 1u;
                if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], use ^ 1u, wctx, 30 + buf, lt))) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)buf * kBN;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % kPStages;
                    const uint32_t ph = (uint32_t)(it / kPStages) & 1u;
                    if (!__all_sync(0xffffffffu, mbar_wait(&full[s], ph, wctx, 20 + s, it))) {
                        live = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sA = smem_u32(smem + s * kPStageBytes);
                    const uint32_t sB = sA + kPABytes;
                    const uint64_t a0 = umma_smem_desc(sA, kAMn ? kSubBytes : 16, 1024);
                    const uint64_t b0 = umma_smem_desc(sB, kBMn ? kSubBytes : 16, 1024);
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; ++kk)
                        umma_ss_pair(d_tmem, umma_desc_advance(a0, kk * a_step), umma_desc_advance(b0, kk * b_step), idesc,
                                     (uint32_t)((kb | kk) != 0));
                    const uint32_t e0 = smem_u32(&empty[s]);
                    tc_commit_pair(e0);                  // this CTA's producer may refill the stage ...
                    tc_commit_pair(map_to_cta(e0, 1));   // ... and so may the peer's
                }
                if (live) {
                    const uint32_t f0 = smem_u32(&acc_full[buf]);
                    tc_commit_pair(f0);
                    tc_commit_pair(map_to_cta(f0, 1));
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue (warps 2..5, both CTAs)
        const int lane_group = warp & 3;                 // tensor-memory lanes 32*lane_group .. +31
        const uint32_t lane_off = (uint32_t)(lane_group * 32) << 16;
        int lt = 0;
        for (int t = pair; t < total; t += n_pairs, ++lt) {
            int mb, nb;
            fc_tile_coords(t, tiles_m, tiles_n, mb, nb);
            const int buf = lt & 1;
            const uint32_t use = (uint32_t)(lt >> 1) & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[buf], use, wctx, 40 + buf, lt))) break;
            tc_fence_after();
            const long long row = (long long)mb * 256 + (int)rank * 128 + lane_group * 32 + lane;
            store_acc_row<true>(tmem_base + lane_off + (uint32_t)(buf * kBN), row, nb * kBN, C, bias, M, N, wide,
                                nullptr, map_to_cta(smem_u32(&acc_empty[buf]), 0));
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // neither CTA leaves while the other may still read its shared memory or signal its barriers
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// fp32-arithmetic SIMT GEMM for bf16 shapes the tensor-core kernel does not take (row pitches that are not multiples of
// 16 bytes), and for floats where TT_FC_PATH=simt asks for it.  64x64 tiles, 4x4 outputs per thread.
template <typename T> __device__ __forceinline__ float g_ld(const T* p, long long i);
template <> __device__ __forceinline__ float g_ld<float>(const float* p, long long i) { return p[i]; }
template <> __device__ __forceinline__ float g_ld<__nv_bfloat16>(const __nv_bfloat16* p, long long i) { return __bfloat162float(p[i]); }
template <typename T> __device__ __forceinline__ void g_st(T* p, long long i, float v);
template <> __device__ __forceinline__ void g_st<float>(float* p, long long i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void g_st<__nv_bfloat16>(__nv_bfloat16* p, long long i, float v) { p[i] = __float2bfloat16_rn(v); }

template <typename T>
__global__ void __launch_bounds__(256) fc_gemm_simt_kernel(const T* __restrict__ A, const T* __restrict__ B,
                                                          T* __restrict__ C, const T* __restrict__ bias, int M, int N,
                                                          int K, int a_mn, int b_mn) {
    grid_let_next_start();
    grid_wait_for_previous();
    __shared__ float sA[16][64 + 1];
    __shared__ float sB[16][64 + 1];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const long long m0 = (long long)blockIdx.y * 64;
    const int n0 = blockIdx.x * 64;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += 16) {
        for (int i = threadIdx.x; i < 16 * 64; i += 256) {
            // the faster-running index follows the contiguous axis of each operand
            const int kk_a = a_mn ? i / 64 : i % 16, mm = a_mn ? i % 64 : i / 16;
            const long long m = m0 + mm;
            const int k = k0 + kk_a;
            sA[kk_a][mm] = (m < M && k < K) ? g_ld<T>(A, a_mn ? (long long)k * M + m : m * K + k) : 0.f;
            const int kk_b = b_mn ? i / 64 : i % 16, nn = b_mn ? i % 64 : i / 16;
            const int n = n0 + nn, kb = k0 + kk_b;
            sB[kk_b][nn] = (n < N && kb < K) ? g_ld<T>(B, b_mn ? (long long)kb * N + n : (long long)n * K + kb) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                a[i] = sA[kk][ty * 4 + i];
                b[i] = sB[kk][tx * 4 + i];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < N) g_st<T>(C, m * N + n, acc[i][j] + (bias ? g_ld<T>(bias, n) : 0.f));
        }
    }
}

// Column sums of a row-major [M,N] matrix: partial[split][n] over a fixed row range per split, then a second pass adds
// the splits in order (deterministic).  A warp reads 32 x kV consecutive values of a row (16 bytes per lane where
// the pitch allows it), four rows in flight per thread; 8 warps take every eighth row each.
template <typename T, int kV>
__device__ __forceinline__ void add_values(const T* p, float (&s)[kV]) {
    if constexpr (kV == 1) {
        s[0] += g_ld<T>(p, 0);
    } else {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if constexpr (sizeof(T) == 2) {
                s[2 * i] += __uint_as_float(w[i] << 16);
                s[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
            } else {
                s[i] += __uint_as_float(w[i]);
            }
        }
    }
}
template <typename T, int kV>
__global__ void __launch_bounds__(256) colsum_partial_kernel(const T* __restrict__ X, float* __restrict__ partial,
                                                            long long M, int N, int rows_per_split) {
    grid_let_next_start();
    grid_wait_for_previous();
    __shared__ float red[8][32 * kV];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col0 = blockIdx.x * 32 * kV, col = col0 + lane * kV;
    const long long r0 = (long long)blockIdx.y * rows_per_split;
    const long long r1 = min(M, r0 + rows_per_split);
    float s[kV] = {};
    if (col < N) {   // kV > 1: N is a multiple of it
#pragma unroll 4
        for (long long r = r0 + warp; r < r1; r += 8) add_values<T, kV>(X + r * N + col, s);
    }
#pragma unroll
    for (int e = 0; e < kV; ++e) red[warp][lane * kV + e] = s[e];
    __syncthreads();
    for (int c = threadIdx.x; c < 32 * kV && col0 + c < N; c += 256) {
        float v = red[0][c];
#pragma unroll
        for (int w = 1; w < 8; ++w) v += red[w][c];
        partial[(long long)blockIdx.y * N + col0 + c] = v;
    }
}
// A warp adds every eighth split of 32 columns.
template <typename T>
__global__ void __launch_bounds__(256) colsum_final_kernel(const float* __restrict__ partial, T* __restrict__ out, int N, int splits,
                                                          int scalar_bias) {
    grid_let_next_start();
    grid_wait_for_previous();
    __shared__ float red[256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float s = 0.f;
    if (scalar_bias) {   // one CTA: the reference's single-value bias gets the sum over all columns too
        const long long values = (long long)splits * N;
        for (long long i = threadIdx.x; i < values; i += 256) s += partial[i];
        red[threadIdx.x] = s;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) g_st<T>(out, 0, red[0]);
        return;
    }
    const int n = blockIdx.x * 32 + lane;
    if (n < N) {
#pragma unroll 4
        for (int p = warp; p < splits; p += 8) s += partial[(long long)p * N + n];
    }
    red[threadIdx.x] = s;
    __syncthreads();
    if (warp == 0 && n < N) {
#pragma unroll
        for (int w = 1; w < 8; ++w) s += red[w * 32 + lane];
        g_st<T>(out, n, s);
    }
}

template <bool kAMn, bool kBMn>
cudaError_t launch_tc(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, cudaStream_t st) {
    TmapStorage ta, tb;
    const char* why = nullptr;
    if (!make_tmap_bf16(&ta, A, kAMn ? (uint64_t)M : (uint64_t)K, kAMn ? (uint64_t)K : (uint64_t)M, 1, kAMn ? 64 : kBM, &why))
        return cudaErrorInvalidValue;
    if (!make_tmap_bf16(&tb, B, kBMn ? (uint64_t)N : (uint64_t)K, kBMn ? (uint64_t)K : (uint64_t)N, 1, kBMn ? 64 : kBN, &why))
        return cudaErrorInvalidValue;
    const int tiles_m = (M + kBM - 1) / kBM, tiles_n = (N + kBN - 1) / kBN;
    const int wide = ((reinterpret_cast<uintptr_t>(C) & 31) == 0 && N % 16 == 0) ? 1 : 0;   // 32-byte stores possible
    const CUtensorMap &ma = *reinterpret_cast<CUtensorMap*>(ta.bytes), &mb = *reinterpret_cast<CUtensorMap*>(tb.bytes);
    LaunchScope ls(K_FC_GEMM, st);
    const int n_cta = fc_k_ctas((long long)tiles_m * tiles_n, (K + kBK - 1) / kBK);
    if (n_cta > 1) {
        const cudaError_t e = TT_ALLOW_SMEM((fc_gemm_sm100_kernel<kAMn, kBMn, true>), kGemmSmem);
        if (e != cudaSuccess) return e;
        return launch_overlapped_cluster(fc_gemm_sm100_kernel<kAMn, kBMn, true>, (unsigned)(tiles_m * tiles_n * n_cta), 192, kGemmSmem, st, n_cta,
                                         ma, mb, (__nv_bfloat16*)C, (const __nv_bfloat16*)bias, M, N, K, tiles_m, tiles_n, wide, device_status_word());
    }
    const cudaError_t e = TT_ALLOW_SMEM((fc_gemm_sm100_kernel<kAMn, kBMn, false>), kGemmSmem);
    if (e != cudaSuccess) return e;
    launch_overlapped(fc_gemm_sm100_kernel<kAMn, kBMn, false>, std::min(tiles_m * tiles_n, sm_count()), 192, kGemmSmem, st, ma, mb,
                      (__nv_bfloat16*)C, (const __nv_bfloat16*)bias, M, N, K, tiles_m, tiles_n, wide, device_status_word());
    return cudaGetLastError();
}


// true: the CTA-pair kernel takes this launch.  It needs enough 256x256 tiles to fill the pairs; smaller
// problems spread better as 128x256 tiles over single CTAs.  TT_FC_PATH=1cta / 2cta forces either (tests).
bool use_pair_kernel(int M, int N) {
    const char* f = getenv("TT_FC_PATH");
    if (f && f[0] == '1') return false;
    if (f && f[0] == '2') return true;
    const long long tiles = (long long)((M + 255) / 256) * ((N + 255) / 256);
    return tiles >= sm_count();   // two or more tiles per pair
}

template <bool kAMn, bool kBMn>
cudaError_t launch_tc_pair(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, cudaStream_t st) {
    TmapStorage ta, tb;
    const char* why = nullptr;
    if (!make_tmap_bf16(&ta, A, kAMn ? (uint64_t)M : (uint64_t)K, kAMn ? (uint64_t)K : (uint64_t)M, 1, kAMn ? 64 : 128, &why))
        return cudaErrorInvalidValue;
    if (!make_tmap_bf16(&tb, B, kBMn ? (uint64_t)N : (uint64_t)K, kBMn ? (uint64_t)K : (uint64_t)N, 1, kBMn ? 64 : 128, &why))
        return cudaErrorInvalidValue;
    cudaError_t e = TT_ALLOW_SMEM((fc_gemm_pair_sm100_kernel<kAMn, kBMn>), kPairSmem);
    if (e != cudaSuccess) return e;
    const int tiles_m = (M + 255) / 256, tiles_n = (N + 255) / 256;
    // pairs that can be resident at once (a GPC with an odd number of usable SMs leaves one without a partner)
    static int max_pairs[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!max_pairs[dev]) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)sm_count() & ~1u);
        cfg.blockDim = dim3(192);
        cfg.dynamicSmemBytes = kPairSmem;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 2;
        at.val.clusterDim.y = 1;
        at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, fc_gemm_pair_sm100_kernel<kAMn, kBMn>, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = sm_count() / 2;
        }
        max_pairs[dev] = n;
    }
    const int pairs = std::min(tiles_m * tiles_n, max_pairs[dev]);
    LaunchScope ls(K_FC_GEMM, st);
    launch_overlapped(fc_gemm_pair_sm100_kernel<kAMn, kBMn>, 2 * pairs, 192, kPairSmem, st, *reinterpret_cast<CUtensorMap*>(ta.bytes), *reinterpret_cast<CUtensorMap*>(tb.bytes), (__nv_bfloat16*)C,
        (const __nv_bfloat16*)bias, M, N, K, tiles_m, tiles_n,
        ((reinterpret_cast<uintptr_t>(C) & 31) == 0 && N % 16 == 0) ? 1 : 0, device_status_word());
    return cudaGetLastError();
}

}  // namespace

bool fc_gemm_tc_supported(const void* A, const void* B, const void* C, const void* bias, long long M, int N, int K,
                          int a_mn, int b_mn, int bf16) {
    if (!bf16 || M < 1 || M > 0x7fffffffLL || N < 1 || K < 1) return false;
    const long long a_cols = a_mn ? M : K, b_cols = b_mn ? N : K;
    if (a_cols % 8 || b_cols % 8 || N % 8) return false;
    if (((uintptr_t)A | (uintptr_t)B | (uintptr_t)C | (uintptr_t)bias) & 15) return false;
    const char* f = getenv("TT_FC_PATH");
    if (f && f[0] == 's') return false;   // "simt": force the fp32-arithmetic kernel (tests)
    return true;
}

cudaError_t fc_gemm(const void* A, const void* B, void* C, const void* bias, long long M, int N, int K, int a_mn,
                    int b_mn, int bf16, cudaStream_t st) {
    if (fc_gemm_tc_supported(A, B, C, bias, M, N, K, a_mn, b_mn, bf16)) {
        if (use_pair_kernel((int)M, N)) {
            if (!a_mn && b_mn) return launch_tc_pair<false, true>(A, B, C, bias, (int)M, N, K, st);
            if (!a_mn && !b_mn) return launch_tc_pair<false, false>(A, B, C, bias, (int)M, N, K, st);
            if (a_mn && b_mn) return launch_tc_pair<true, true>(A, B, C, bias, (int)M, N, K, st);
            return launch_tc_pair<true, false>(A, B, C, bias, (int)M, N, K, st);
        }
        if (!a_mn && b_mn) return launch_tc<false, true>(A, B, C, bias, (int)M, N, K, st);
        if (!a_mn && !b_mn) return launch_tc<false, false>(A, B, C, bias, (int)M, N, K, st);
        if (a_mn && b_mn) return launch_tc<true, true>(A, B, C, bias, (int)M, N, K, st);
        return launch_tc<true, false>(A, B, C, bias, (int)M, N, K, st);
    }
    if (fc_f32_tc_supported(M, N, K, a_mn, b_mn, bf16)) return fc_gemm_f32_sm100(A, B, C, bias, (int)M, N, K, a_mn, b_mn, st);
    dim3 grid((unsigned)((N + 63) / 64), (unsigned)((M + 63) / 64));
    if (grid.y > 65535u) return cudaErrorInvalidValue;
    LaunchScope ls(K_FC_SIMT, st);
    if (bf16)
        launch_overlapped(fc_gemm_simt_kernel<__nv_bfloat16>, grid, 256, 0, st, (const __nv_bfloat16*)A, (const __nv_bfloat16*)B,
                                                                (__nv_bfloat16*)C, (const __nv_bfloat16*)bias, (int)M, N, K, a_mn, b_mn);
    else
        launch_overlapped(fc_gemm_simt_kernel<float>, grid, 256, 0, st, (const float*)A, (const float*)B, (float*)C, (const float*)bias,
                                                        (int)M, N, K, a_mn, b_mn);
    return cudaGetLastError();
}

// Row ranges: about four CTAs of 256 columns per SM, each of at least 64 rows (eight per warp); for the sake of precision never
// fewer than one per 256 rows up to 64, because a thread adds the rows of a range one after the other.  Float [16384,152000]:
// error 2.2e-7 in one range, 1431 us, 4.9e-8 in 64, 1384 us (two-level sums inside one range: 5.4e-8, 1512 us).
static int fc_colsum_splits(long long M, int N) {
    const long long blocks = (N + 255) / 256, most = std::max(1LL, (4LL * sm_count() + blocks - 1) / blocks);
    const long long least = std::min(64LL, (M + 255) / 256);
    return (int)std::max(std::max(1LL, least), std::min(std::min(most, 256LL), M / 64));
}
size_t fc_colsum_workspace(long long M, int N) { return align256((size_t)fc_colsum_splits(M, N) * (size_t)N * sizeof(float)); }

template <typename T>
static cudaError_t launch_colsum_partial(const void* X, float* partial, long long M, int N, int splits, cudaStream_t st) {
    constexpr int kV = 16 / sizeof(T);
    const int rows = (int)((M + splits - 1) / splits);
    if (N % kV == 0 && ((uintptr_t)X & 15) == 0)
        return launch_overlapped(colsum_partial_kernel<T, kV>, dim3((unsigned)((N + 32 * kV - 1) / (32 * kV)), (unsigned)splits), 256, 0, st,
                                 (const T*)X, partial, M, N, rows);
    return launch_overlapped(colsum_partial_kernel<T, 1>, dim3((unsigned)((N + 31) / 32), (unsigned)splits), 256, 0, st, (const T*)X, partial, M, N, rows);
}
cudaError_t fc_colsum(const void* X, void* out, long long M, int N, int bf16, int scalar_bias, void* workspace,
                      cudaStream_t st) {
    const int splits = fc_colsum_splits(M, N);
    float* partial = (float*)workspace;
    {
        LaunchScope ls(K_FC_COLSUM, st);
        const cudaError_t e = bf16 ? launch_colsum_partial<__nv_bfloat16>(X, partial, M, N, splits, st)
                                   : launch_colsum_partial<float>(X, partial, M, N, splits, st);
        if (e != cudaSuccess) return e;
    }
    LaunchScope ls(K_FC_COLSUM, st, false);
    const unsigned fgrid = scalar_bias ? 1u : (unsigned)((N + 31) / 32);
    if (bf16) launch_overlapped(colsum_final_kernel<__nv_bfloat16>, fgrid, 256, 0, st, partial, (__nv_bfloat16*)out, N, splits, scalar_bias);
    else launch_overlapped(colsum_final_kernel<float>, fgrid, 256, 0, st, partial, (float*)out, N, splits, scalar_bias);
    return cudaGetLastError();
}

}  // namespace ttk
