// The fully connected layer's GEMMs over float tensors on the tensor cores: C[M,N] = op(A) op(B) (+ bias).
//
// As in the float attention kernels a float is the sum of three bf16 parts and the six largest of the nine part
// products are kept (what is left out is below 2^-26 of the product).  No sum runs through the tensor core for longer
// than one chunk of 64 along K: its additions may truncate, so every chunk's accumulator is added to float
// registers, which round to nearest.
//
// One CTA computes a 128 x 128 tile (or its share of K):
//   warps 0-7    accumulate: thread <-> row of the tile, warps 0-3 columns 0-63, warps 4-7 columns 64-127
//   warps 8-15   convert: global floats -> three bf16 parts -> shared memory (128-byte swizzle), one chunk ahead in registers
//   warp  16     issues 24 MMAs (M128 N128 K16) per chunk
// Both operands are read as they lie: contiguous along K (K-major tile [128 x 64]) or along M / N (MN-major [64 x 128]),
// at any pitch and alignment.  Shared memory is what bounds a chunk: 24 MMAs read 192 KB and the converters write 96 KB,
// about 2300 cycles at 128 B per cycle, 240 TFLOP/s on 148 SMs.
//
// Where there are fewer tiles than SMs, a cluster of up to 8 CTAs cuts K and each CTA adds its rows of the tile
// through distributed shared memory, in rank order: no workspace, no second launch, the same bits every time.
//
// Measured, forward and backward of a layer: [2048,2048]x[2048,2048] 2637 -> 337 us (153 TFLOP/s), [1000,8192]x[8192,3000] 8.29 ->
// 1.08 ms, [16384,64]x[64,64] 1709 -> 69 us, [300,300]x[300,300] 118 -> 48 us against the FMA kernel.  Errors (2-norm, against
// float64) 5e-8 to 1.7e-7; the FMA kernel's 6e-8 to 2.3e-6, growing with K.
//
// The parts of an infinity sum to NaN, and the part products of two factors whose product overflows are infinities of
// either sign.  Both reach the accumulator, so a thread whose share of a row is not finite computes it again with plain
// fused multiply-adds.
#include <cooperative_groups.h>
#include <stdlib.h>

#include <algorithm>

#include "common.h"
#include "f32_parts.cuh"
#include "fc_tiles.cuh"

namespace ttk {
using namespace sm100;

namespace {

constexpr int kTile = 128, kK = 64, kStages = 2;
constexpr int kPart = kTile * kK * 2;                  // one bf16 part of an operand's chunk
constexpr int kOperand = 3 * kPart, kStage = 2 * kOperand;
constexpr int kSub = 64 * 128;                         // MN-major: one 64-wide block of 64 K-rows
constexpr int kSmem = kStages * kStage + 256 + 1024;
constexpr int kAccPitch = kTile + 4;                   // floats; rows of the finished tile in shared memory
constexpr int kThreads = 640, kConvert = 256;           // warps 17-19 only complete the last warpgroup
// registers per thread after setmaxnreg; the sum draws on what the launch allocated (640 x 96)
constexpr int kRegsRows = 104, kRegsConvert = 112, kRegsIssue = 48;
static_assert(2 * kRegsRows + 2 * kRegsConvert + kRegsIssue <= 5 * 96, "register split exceeds the CTA's pool");
static_assert(kTile * kAccPitch * 4 <= kStages * kStage, "the finished tile takes the operands' place");

struct FcF32Params {
    const float *A, *B, *bias;
    float* C;
    int M, N, K;
    int tiles_m, tiles_n;
    int wide;               // 16-byte stores of C possible
    unsigned int* status;
};

// This thread's share of a chunk of one operand: ROWS x COLS floats from (row0, col0) of a [n_rows, n_cols] matrix, four
// groups of 8 consecutive values; what lies past the matrix reads as zero.
template <int ROWS, int COLS, bool kVec>
struct ChunkRegs {
    static constexpr int kGroups = ROWS * COLS / 8 / kConvert;
    float x[kGroups][8];
    __device__ __forceinline__ void load(const float* src, int row0, int col0, int n_rows, int n_cols, int tid) {
#pragma unroll
        for (int i = 0; i < kGroups; ++i) {
            const int idx = i * kConvert + tid, r = row0 + idx / (COLS / 8), c = col0 + (idx % (COLS / 8)) * 8;
            const float* g = src + (long long)r * n_cols + c;
            if (kVec) {   // n_cols is a multiple of 4: four values lie inside or outside together
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (r < n_rows && c + 4 * h < n_cols) v = __ldg(reinterpret_cast<const float4*>(g) + h);
                    x[i][4 * h] = v.x; x[i][4 * h + 1] = v.y; x[i][4 * h + 2] = v.z; x[i][4 * h + 3] = v.w;
                }
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) x[i][e] = (r < n_rows && c + e < n_cols) ? __ldg(g + e) : 0.f;
            }
        }
    }
    // -> three parts at dst
    __device__ __forceinline__ void store(unsigned char* dst, int tid) const {
#pragma unroll
        for (int i = 0; i < kGroups; ++i) {
            const int idx = i * kConvert + tid, r = idx / (COLS / 8), c = idx % (COLS / 8);
            unsigned char* p = dst + (c >> 3) * (ROWS * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4);
            uint4 h, m, l;
            split8(x[i], h, m, l);
            *reinterpret_cast<uint4*>(p) = h;
            *reinterpret_cast<uint4*>(p + kPart) = m;
            *reinterpret_cast<uint4*>(p + 2 * kPart) = l;
        }
    }
};

template <bool kAMn, bool kBMn, bool kVec>
__global__ void __launch_bounds__(kThreads, 1) fc_f32_sm100_kernel(const FcF32Params p) {
    namespace cg = cooperative_groups;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStage);   // [2] converters -> MMA
    uint64_t* empty = full + 2;       // [2] MMA -> converters
    uint64_t* acc_full = full + 4;    // [2] MMA -> accumulating threads
    uint64_t* acc_free = full + 6;    // [2] accumulating threads -> MMA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = uniform_warp_idx(), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int b = 0; b < 2; ++b) {
            mbar_init(&full[b], kConvert);
            mbar_init(&empty[b], 1);
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_free[b], 256);
        }
        fence_barrier_init();
    }
    if (warp == 16) {
        tmem_alloc(tmem_slot, 256);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    WaitCtx ctx{p.status, abort_flag, warp};
    grid_let_next_start();
    grid_wait_for_previous();

    cg::cluster_group cluster = cg::this_cluster();
    const int n_cta = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    int mb, nb;
    fc_tile_coords((int)blockIdx.x / n_cta, p.tiles_m, p.tiles_n, mb, nb);
    const int m0 = mb * kTile, n0 = nb * kTile;
    const int chunks = (p.K - 1) / kK + 1, share = (chunks + n_cta - 1) / n_cta;
    const int u0 = rank * share, n_it = max(0, min(share, chunks - u0));

    float* tile = reinterpret_cast<float*>(smem);
    if (warp < 8) {
        // ---- accumulate
        setmaxnreg_inc<kRegsRows>();
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * 64);
        float acc[64];
#pragma unroll
        for (int e = 0; e < 64; ++e) acc[e] = 0.f;
        for (int u = 0; u < n_it; ++u) {
            const int b = u & 1;
            mbar_wait(&acc_full[b], (u >> 1) & 1, ctx, 30 + b, u);
            __syncwarp();
            tc_fence_after();
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                uint32_t t[32];
                tmem_ld32(lane_base + (uint32_t)(b * kTile + g * 32), t);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 32; ++e) acc[g * 32 + e] += __uint_as_float(t[e]);
            }
            tc_fence_before();
            mbar_arrive(&acc_free[b]);
        }
        const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 64;
        float zero[4] = {};   // NaN where something is not finite
#pragma unroll
        for (int e = 0; e < 64; ++e) zero[e & 3] = fmaf(acc[e], 0.f, zero[e & 3]);
        if (zero[0] + zero[1] + zero[2] + zero[3] != 0.f) {
            const int m = m0 + r, k_end = (int)min((long long)p.K, (long long)(u0 + n_it) * kK);
#pragma unroll
            for (int e = 0; e < 64; ++e) acc[e] = 0.f;
            for (int k = u0 * kK; k < k_end && m < p.M; ++k) {
                const float x = kAMn ? p.A[(long long)k * p.M + m] : p.A[(long long)m * p.K + k];
#pragma unroll
                for (int e = 0; e < 64; ++e) {
                    const int n = n0 + c0 + e;
                    if (n < p.N) acc[e] = fmaf(x, kBMn ? p.B[(long long)k * p.N + n] : p.B[(long long)n * p.K + k], acc[e]);
                }
            }
        }
        // Every chunk's MMAs are done: nothing uses the operands' shared memory any more.
#pragma unroll
        for (int e = 0; e < 64; e += 4)
            *reinterpret_cast<float4*>(tile + r * kAccPitch + c0 + e) = make_float4(acc[e], acc[e + 1], acc[e + 2], acc[e + 3]);
    } else if (warp < 16) {
        // ---- convert
        setmaxnreg_inc<kRegsConvert>();
        const int tid = (int)threadIdx.x - 256;
        ChunkRegs<kAMn ? kK : kTile, kAMn ? kTile : kK, kVec> a;
        ChunkRegs<kBMn ? kK : kTile, kBMn ? kTile : kK, kVec> b;
        auto load_a = [&](int u) {
            const int k0 = (u0 + u) * kK;
            if (kAMn) a.load(p.A, k0, m0, p.K, p.M, tid);
            else a.load(p.A, m0, k0, p.M, p.K, tid);
        };
        auto load_b = [&](int u) {
            const int k0 = (u0 + u) * kK;
            if (kBMn) b.load(p.B, k0, n0, p.K, p.N, tid);
            else b.load(p.B, n0, k0, p.N, p.K, tid);
        };
        if (n_it > 0) {
            load_a(0);
            load_b(0);
        }
        for (int u = 0; u < n_it; ++u) {
            const int s = u & 1;
            mbar_wait(&empty[s], ((u >> 1) & 1) ^ 1, ctx, 10 + s, u);
            unsigned char* dst = smem + s * kStage;
            a.store(dst, tid);
            if (u + 1 < n_it) load_a(u + 1);
            b.store(dst + kOperand, tid);
            fence_proxy_async_smem();
            mbar_arrive(&full[s]);
            if (u + 1 < n_it) load_b(u + 1);
        }
    } else {
        setmaxnreg_dec<kRegsIssue>();
    }
    if (warp == 16) {
        // ---- issue
        constexpr uint32_t idesc = umma_idesc_bf16(kTile, kTile, kAMn, kBMn), hi = umma_desc_hi(1024);
        constexpr uint32_t a_step = kAMn ? 2048u : 32u, b_step = kBMn ? 2048u : 32u;   // 16 along K
        const uint32_t base = __shfl_sync(0xffffffffu, smem_u32(smem), 0), tm = __shfl_sync(0xffffffffu, tmem, 0);
        for (int u = 0; u < n_it; ++u) {
            const int s = u & 1;
            mbar_wait(&full[s], (u >> 1) & 1, ctx, 20 + s, u);
            mbar_wait(&acc_free[s], ((u >> 1) & 1) ^ 1, ctx, 22 + s, u);
            __syncwarp();
            tc_fence_after();
            const uint32_t a0 = umma_desc_lo(base + s * kStage, kAMn ? kSub : 16), b0 = umma_desc_lo(base + s * kStage + kOperand, kBMn ? kSub : 16);
            if (elect_one()) {
#pragma unroll
                for (int t = 0; t < 6; ++t)
#pragma unroll
                    for (int kk = 0; kk < kK / 16; ++kk)
                        umma_ss_one(tm + (uint32_t)(s * kTile), a0 + ((term_a(t) * kPart + kk * a_step) >> 4),
                                    b0 + ((term_b(t) * kPart + kk * b_step) >> 4), hi, idesc, (t > 0 || kk > 0) ? 1u : 0u);
            }
            __syncwarp();
            tc_commit(&empty[s]);
            tc_commit(&acc_full[s]);
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 16) {
        tc_fence_after();
        tmem_dealloc(tmem, 256);
    }
    __syncwarp();
    cluster.sync();
    // ---- this CTA's rows of the tile: the shares in rank order, + bias; a warp stores 512 consecutive bytes
    const int rows = kTile / n_cta, r0 = rank * rows;
    for (int i = threadIdx.x; i < rows * (kTile / 4); i += kThreads) {
        const int r = r0 + i / (kTile / 4), c = (i % (kTile / 4)) * 4, m = m0 + r, n = n0 + c;
        if (m >= p.M || n >= p.N) continue;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int q = 0; q < n_cta; ++q) {
            const float4 x = *reinterpret_cast<const float4*>(cluster.map_shared_rank(tile, q) + r * kAccPitch + c);
            v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        }
        float* dst = p.C + (long long)m * p.N + n;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (p.bias && n + e < p.N) v[e] += __ldg(p.bias + n + e);
        if (p.wide) {
            *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n + e < p.N) dst[e] = v[e];
        }
    }
    __syncwarp();
    cluster.sync();           // a peer may still be reading this CTA's tile
}

template <bool kAMn, bool kBMn, bool kVec>
cudaError_t launch(const FcF32Params& p, int n_cta, cudaStream_t st) {
    auto kernel = fc_f32_sm100_kernel<kAMn, kBMn, kVec>;
    const cudaError_t e = TT_ALLOW_SMEM((fc_f32_sm100_kernel<kAMn, kBMn, kVec>), kSmem);
    if (e != cudaSuccess) return e;
    LaunchScope ls(K_FC_GEMM, st);
    return launch_overlapped_cluster(kernel, (unsigned)(p.tiles_m * p.tiles_n * n_cta), kThreads, kSmem, st, n_cta, p);
}

}  // namespace

// Every pitch and alignment; the operand forms of the layer: (a_mn, b_mn) = (0, 1), (0, 0) or (1, 1).
bool fc_f32_tc_supported(long long M, int N, int K, int a_mn, int b_mn, int bf16) {
    if (bf16 || M < 1 || M > 0x7fffffffLL || N < 1 || K < 1 || (a_mn && !b_mn)) return false;
    if (((M - 1) / kTile + 1) * ((N - 1) / kTile + 1) * 8 >= (1LL << 31)) return false;
    const char* f = getenv("TT_FC_PATH");
    return !(f && f[0] == 's');   // "simt": force the fp32-arithmetic kernel (tests)
}
cudaError_t fc_gemm_f32_sm100(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int a_mn, int b_mn,
                              cudaStream_t st) {
    FcF32Params p = {};
    p.A = (const float*)A; p.B = (const float*)B; p.bias = (const float*)bias; p.C = (float*)C;
    p.M = M; p.N = N; p.K = K;
    p.tiles_m = (M - 1) / kTile + 1;
    p.tiles_n = (N - 1) / kTile + 1;
    p.wide = N % 4 == 0 && ((uintptr_t)C & 15) == 0;
    p.status = device_status_word();
    const int a_ld = a_mn ? M : K, b_ld = b_mn ? N : K;
    const bool vec = a_ld % 4 == 0 && b_ld % 4 == 0 && (((uintptr_t)A | (uintptr_t)B) & 15) == 0;
    const int n_cta = fc_k_ctas((long long)p.tiles_m * p.tiles_n, (K - 1) / kK + 1);
    if (a_mn && b_mn) return vec ? launch<true, true, true>(p, n_cta, st) : launch<true, true, false>(p, n_cta, st);
    if (!a_mn && b_mn) return vec ? launch<false, true, true>(p, n_cta, st) : launch<false, true, false>(p, n_cta, st);
    return vec ? launch<false, false, true>(p, n_cta, st) : launch<false, false, false>(p, n_cta, st);
}

}  // namespace ttk
