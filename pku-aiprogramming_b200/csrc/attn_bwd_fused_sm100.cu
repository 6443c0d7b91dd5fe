// Single-pass attention backward for B200 (sm_100a): bf16 tensors, fp32 accumulation, head dim 64 or
// 128.  One launch computes dK, dV AND dQ: nothing is recomputed, five GEMMs per (key tile, query tile)
// pair -- the five the backward is counted as -- against the seven of the two-pass kernel
// (attn_bwd_sm100.cu), which stays as the bit-reproducible alternative.
//
//   P^T = exp(scale*K Q^T - lse)   dP^T = V dO^T   dS^T = P^T * (dP^T - delta)
//   dV += P^T dO      dK += dS^T Q      dQ_partial = dS K  -> added to an fp32 accumulator in global memory
//
// A CTA owns 128 keys (K, V tiles resident in shared memory) and streams the query tiles (Q_i, dO_i)
// that can see them; scores are computed transposed (keys on the TMEM lanes).  Per streamed tile:
//   G1: S^T  = K Q^T        (A, B shared memory, K-major)                       -> X
//   G2: dP^T = V dO^T       (A, B shared memory, K-major)                       -> Y
//   G3: dV  += P^T dO       (A = bf16 P^T in tensor memory over S^T, B = dO MN-major)
//   G4: dK  += dS^T Q       (A = bf16 dS^T in SHARED memory, K-major;  B = Q MN-major)
//   G5: dQ_t = dS K         (A = the same dS^T bytes read MN-major;    B = K MN-major)   -> Y
// Tensor memory (512 columns): X [0,128) S^T | Y [128,256) dP^T | dV [256,256+D) | dK [256+D,256+2D).  At D = 128 that is all
// of it: P^T overlays X and dQ_t overlays Y, and the MMA warp issues, per tile t, G3(t) G1(t+1) G5(t) G4(t) G2(t+1).  At D = 64
// dQ_t and P^T have columns of their own, S^T(t+1) is issued as soon as S^T(t) is in registers and dP^T(t+1) as soon as
// dS^T(t) is: G1(t+1) G3(t) G2(t+1) G5(t) G4(t).
// dS^T cannot stay in tensor memory as in the two-pass kernel: G5 needs it with the queries on the M side, and a
// tensor-memory operand is always M = lanes = keys here.  So the compute threads write it to a 32 KB shared-memory tile in
// the 128-byte-swizzled layout both descriptors read.
//
// dQ_t leaves through a warpgroup of its own: tensor memory -> registers (Y is released at once) -> 16 KB pieces in shared
// memory -> cp.reduce.async.bulk add.f32 into a [D/4][128 rows][4] block per (query slice, query tile).  A small second
// kernel converts the accumulator to bf16 dQ (times scale).  The L2 takes about 3-4 KB of fp32 additions per cycle from the
// whole chip, and what waits for it must not be a warp's memory instruction: with red.global.add the additions held up the
// memory queue that the compute warps' tensor-memory and shared-memory accesses share, from whichever warps they were
// issued (cycles per tile, S = 4096 not causal: red from the compute warps 5069 at D = 128, 4546 at D = 64; red from the
// adding warpgroup 5536, 4727; bulk additions 4043, 3842).  Statistics by bulk copies, already negated and padded to whole
// tiles, and positions stepped instead of divided out: 3818, 3125.  Of those 3818, the additions of 64 KB take ~3200.
// The additions arrive in no fixed order, so dQ is reproducible to fp32 rounding only; dK and dV are bit-reproducible.
//
// Roles: warps 0-7 = two compute warpgroups (thread <-> resident key row; warpgroup w owns query columns [64w, 64w+64) of X
// and Y, and columns [w*D/2, +D/2) of dV, dK), warps 8-11 = the adding warpgroup (thread <-> query row), warp 12 = MMA
// issuer, warp 13 = TMA loader and work-item scheduler.
// Shared memory at D = 128: K, V, two Q slots, one dO slot, the dS^T tile, 2 x 16 KB of dQ_t pieces (7 x 32 KB) + 2.5 KB of
// barriers and per-query statistics.
#include "attn_bwd_common.cuh"
#include <stdlib.h>
#include <string.h>
#include <algorithm>
#include <atomic>
#include <type_traits>

namespace ttk {
using namespace sm100;

template <int D>
struct Bwd1Cfg {
    // warps 0-7 compute, 8-11 add dQ_t, 12 issues MMAs, 13 loads, 14 and 15 only complete a warpgroup for setmaxnreg
    static constexpr int kThreads = 512;
    static constexpr int kRegsLaunch = 128, kRegsCompute = 144, kRegsAdd = 152, kRegsOther = 72;
    static_assert(256 * kRegsCompute + 128 * kRegsAdd + 128 * kRegsOther <= kThreads * kRegsLaunch, "register split exceeds the CTA's pool");
    static constexpr int kSub = D / 64;
    static constexpr int kSubBytes = 128 * 128;
    static constexpr int kTileBytes = kSub * kSubBytes;
    static constexpr int kDsBytes = 2 * kSubBytes;               // 128 keys x 128 queries, bf16
    // Q(t) is read by G1(t) early and by G4(t) late, Q(t+1) in between; dO(t) by G2(t) and G3(t), and
    // dO(t+1) only by the last GEMM of the next iteration, so ONE dO slot is enough.
    static constexpr int kNQ = (D == 128) ? 2 : 4;
    static constexpr int kNdO = (D == 128) ? 1 : 3;
    static_assert(kNQ >= 2 && kNQ <= 4 && kNdO >= 1 && kNdO <= 4, "ring lengths the barrier arrays are sized for");
    static constexpr int kTmemCols = 512;
    static constexpr int kBarBytes = 512;
    static constexpr int kStatBytes = 2 * 128 * 4;               // -lse2 and -delta of a tile's 128 queries; two such slots
    static constexpr int kAuxBytes = kBarBytes + 2 * kStatBytes;
    static constexpr int kStageBytes = 128 * 32 * 4;             // 32 columns of dQ_t; two such buffers
    static constexpr int kSmemBytes = (2 + kNQ + kNdO) * kTileBytes + kDsBytes + 2 * kStageBytes + kAuxBytes;
    static_assert(kSmemBytes <= 227 * 1024, "exceeds the shared memory of one CTA");
};

enum Bwd1BarId { B1_RES = 0, B1_QFULL = 10, B1_QEMPTY = 14, B1_DOFULL = 18, B1_DOEMPTY = 22, B1_SFULL = 30, B1_DPFULL = 31,
                 B1_PFULL = 32, B1_DSFULL = 33, B1_FINAL = 34, B1_STAT = 35, B1_DSFREE = 36, B1_DQFULL = 37, B1_DQFREE = 38,
                 B1_ACCFREE = 39, B1_SREAD = 40, B1_PFREE = 41 };

// The u-th streamed tile of an item: as in the two-pass kernel (heads of a group one after the other), but
// without a causal mask every key tile of a slice meets ALL query tiles, and CTAs that started together
// would walk them in step and add their dQ_t into the same 64 KB at the same moment; so key tile r starts
// its walk at query tile r and wraps round.  (Under the causal mask key tile r starts at query tile r anyway.)
// Walked step by step: the divisions of a position's closed form are some 400 cycles of latency per tile and role.
struct FusedStream {
    int t, slice;    // query tile and query slice (packed batches: query head) of the current position
    int first, j;    // the slice's first tile index (relative to t_begin) and the position in its walk
    __device__ __forceinline__ FusedStream(const BwdItem& w, const BwdParams& p, bool packed)
        : slice((packed ? w.head : w.bh) * p.group), first(p.causal || w.nt == 0 ? 0 : (w.r0 >> 7) % w.nt), j(0) { t = w.t_begin + first; }
    __device__ __forceinline__ void next(const BwdItem& w) {
        if (++j == w.nt) {
            j = 0;
            ++slice;
            t = w.t_begin + first;
        } else if (++t == w.t_end) {
            t = w.t_begin;
        }
    }
};

// What the loader publishes of a packed batch's item, so that the other roles need no search of their own.
struct PackedItem { int head, r0, S, L, q_lo, k_lo, tile0, item; };   // item: the adding warps' copy alone
struct FusedItem : BwdItem {
    long long blk0;   // accumulator and statistics of query tile t of query slice s: block s * n_qt + blk0 + t
};
template <bool kVarlen>
__device__ __forceinline__ FusedItem fused_item(int item, const PackedItem* packed, const BwdParams& p) {
    FusedItem w;
    if constexpr (kVarlen) {
        w.head = packed->head;
        w.r0 = packed->r0;
        w.S = packed->S;
        w.L = w.Lv = packed->L;
        w.q_lo = packed->q_lo;
        w.k_lo = packed->k_lo;
        w.blk0 = packed->tile0;
        w.bh = 0;
        w.t_end = (w.S + 127) >> 7;
        w.t_begin = p.causal ? (max(0, w.r0 - (w.L - w.S)) >> 7) : 0;
        w.nt = max(0, w.t_end - w.t_begin);
        w.n_it = w.nt * p.group;
    } else {
        static_cast<BwdItem&>(w) = bwd_decode_item<true>(item, p);
        w.blk0 = 0;
    }
    return w;
}

// Adds `bytes` of floats in shared memory to global memory by the TMA engine (one thread; a bulk group of its own).
__device__ __forceinline__ void bulk_add_f32(float* gptr, const void* src, uint32_t bytes) {
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;\n\tcp.async.bulk.commit_group;"
                 ::"l"(gptr), "r"(smem_u32(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
template <int kLeft>   // at most kLeft groups of this thread have shared memory still to be read
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kLeft) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

#define TT_B1TRACE(role, iter, slot)                                                               \
    do {                                                                                           \
        if (kTrace && p.trace != nullptr && (int)blockIdx.x == p.trace_block && (iter) < 64)       \
            p.trace[((role) * 64 + (iter)) * 8 + (slot)] = clock64();                              \
    } while (0)

// kTrace: compiled with the cycle stamps (tuning aid; launched only while a trace buffer is set).
// kVarlen: packed batches; work items are numbered by the batch's key tiles (see packed_seq), so that none but the unused
// numbers and the tiles that no query sees is empty.
template <int D, bool kTrace, bool kVarlen>
__global__ void __launch_bounds__(Bwd1Cfg<D>::kThreads, 1)
attn_bwd_fused_sm100_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                            const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                            const BwdParams p) {
    using Cfg = Bwd1Cfg<D>;
    constexpr int kNQ = Cfg::kNQ, kNdO = Cfg::kNdO;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw;
    if ((smem_u32(smem_raw) & 1023u) != 0u) {   // the 128-byte swizzle of TMA and UMMA needs 1024-byte aligned tiles
        if (threadIdx.x == 0 && atomicCAS(p.status, 0u, (8u << 16) | (blockIdx.x & 0xffffu)) == 0u) {
            p.status[1] = 0xA116u;   // "alignment"
            p.status[2] = smem_u32(smem_raw);
            p.status[3] = 0u;
        }
        return;                      // every thread of every CTA takes this exit together: nothing was started
    }
    unsigned char* sK = smem;                                   // resident K tile
    unsigned char* sV = smem + Cfg::kTileBytes;                 // resident V tile
    unsigned char* sQ = smem + 2 * Cfg::kTileBytes;             // kNQ slots
    unsigned char* sdO = sQ + kNQ * Cfg::kTileBytes;            // kNdO slots
    unsigned char* sDS = sdO + kNdO * Cfg::kTileBytes;          // dS^T: 2 sub-blocks of [128 keys x 64 queries]
    unsigned char* sStage = sDS + Cfg::kDsBytes;                // two buffers of 32 dQ_t columns, [8][128 rows][4] floats
    unsigned char* aux = sStage + 2 * Cfg::kStageBytes;
    uint64_t* bar_res_full = reinterpret_cast<uint64_t*>(aux);   // TMA -> MMA (K, V of the item)
    uint64_t* bar_res_empty = bar_res_full + 1;                  // MMA (last reads of K, V) -> TMA
    uint64_t* bar_q_full = bar_res_empty + 1;                    // [4]
    uint64_t* bar_q_empty = bar_q_full + 4;                      // [4]
    uint64_t* bar_do_full = bar_q_empty + 4;                     // [4]
    uint64_t* bar_do_empty = bar_do_full + 4;                    // [4]
    uint64_t* bar_s_full = bar_do_empty + 4;                     // MMA -> compute: S^T(t) is in X
    uint64_t* bar_p_full = bar_s_full + 1;                       // compute -> MMA: P^T(t) is in X
    uint64_t* bar_dp_full = bar_p_full + 1;                      // MMA -> compute: dP^T(t) is in Y
    uint64_t* bar_ds_full = bar_dp_full + 1;                     // compute -> MMA: dS^T(t) is in shared memory, Y is read
    uint64_t* bar_ds_free = bar_ds_full + 1;                     // MMA -> compute: G4(t), G5(t) are done with the dS^T tile
    uint64_t* bar_dq_full = bar_ds_free + 1;                     // MMA -> adding warps: dQ_t is in its columns
    uint64_t* bar_dq_free = bar_dq_full + 1;                     // adding warps -> MMA: dQ_t is in registers
    uint64_t* bar_final = bar_dq_free + 1;                       // MMA -> compute: dV, dK of the item are complete
    uint64_t* bar_acc_free = bar_final + 1;                      // compute (accumulators read out) -> MMA
    uint64_t* bar_sched_full = bar_acc_free + 1;                 // [2]
    uint64_t* bar_sched_empty = bar_sched_full + 2;              // [2]
    uint64_t* bar_stat_full = bar_sched_empty + 2;               // [2] TMA -> compute: a tile's statistics
    uint64_t* bar_stat_empty = bar_stat_full + 2;                // [2] compute -> TMA
    uint64_t* bar_s_read = bar_stat_empty + 2;                        // D = 64, compute -> MMA: S^T(t) is in registers
    uint64_t* bar_p_free = bar_s_read + 1;                       // D = 64, MMA -> compute: G3(t) is done with P^T(t)
    int* sched_item = reinterpret_cast<int*>(bar_p_free + 1);    // [2]
    uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(sched_item + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);
    PackedItem* add_item = reinterpret_cast<PackedItem*>(aux + 320);  // [2], the adding warps' items as warp 8 read them
    PackedItem* packed = reinterpret_cast<PackedItem*>(aux + 384);    // [2], beside sched_item
    uint64_t* bar_steal = reinterpret_cast<uint64_t*>(aux + Cfg::kBarBytes - 32);
    uint4* steal_response = reinterpret_cast<uint4*>(bar_steal + 2);
    float* s_stat = reinterpret_cast<float*>(aux + Cfg::kBarBytes);   // [2 slots][2: -lse2, -delta][128]

    const int warp = uniform_warp_idx();
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        mbar_init(bar_steal, 1);
        mbar_init(bar_res_full, 1);
        mbar_init(bar_res_empty, 1);
        for (int s = 0; s < 4; ++s) {
            mbar_init(&bar_q_full[s], 1);
            mbar_init(&bar_q_empty[s], 1);
            mbar_init(&bar_do_full[s], 1);
            mbar_init(&bar_do_empty[s], 1);
        }
        mbar_init(bar_s_full, 1);
        mbar_init(bar_p_full, 8);
        mbar_init(bar_dp_full, 1);
        mbar_init(bar_ds_full, 8);
        mbar_init(bar_ds_free, 1);
        mbar_init(bar_dq_full, 1);
        mbar_init(bar_dq_free, 4);
        mbar_init(bar_s_read, 8);
        mbar_init(bar_p_free, 1);
        mbar_init(bar_final, 1);
        mbar_init(bar_acc_free, 8);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_stat_full[i], 1);
            mbar_init(&bar_stat_empty[i], 8);
            mbar_init(&bar_sched_full[i], 1);
            mbar_init(&bar_sched_empty[i], 10);   // MMA warp, compute warps, the first adding warp
        }
        fence_barrier_init();
        fence_proxy_async_smem();
    }
    if (warp == 12) {
        tmem_alloc(tmem_base_slot, Cfg::kTmemCols);
        tmem_relinquish();
    }
    if (warp == 13 && lane == 0) {
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmdO);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    WaitCtx wctx{p.status, abort_flag, warp};
    ItemStream items{bar_steal, steal_response, p.n_items > p.first_wave};   // the loader warp's
    grid_let_next_start();
    grid_wait_for_previous();
    constexpr uint32_t kColX = 0, kColY = 128, kColDV = 256, kColDK = 256 + D;
    // At D = 64 the accumulators leave 128 columns, 64 for dQ_t and 64 for P^T: the scores of the next tile then wait for
    // nothing but the loads of this tile's.
    constexpr bool kApart = D == 64;
    constexpr uint32_t kColDQ = kApart ? 384 : kColY, kColP = kApart ? 448 : kColX, kPitchP = kApart ? 32 : 64;

    auto next_item = [&](int k) -> int {
        const int slot = k & 1;
        // a wait that gave up (this CTA has aborted) ends the sequence: the slot may hold anything.  Lanes may find that out one by
        // one, the warp leaves as one: what follows are warp-wide instructions
        if (!__all_sync(0xffffffffu, mbar_wait(&bar_sched_full[slot], (k >> 1) & 1, wctx, 80 + slot, k))) return -1;
        return sched_item[slot];
    };
    // one arrival per warp, behind what all its threads did
    auto warp_arrive = [&](uint64_t* bar) {
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
    };
    auto take_item = [&](int k, FusedItem& w) -> bool {   // compute warps, MMA issuer
        const int item = next_item(k);
        if (item >= 0) w = fused_item<kVarlen>(item, &packed[k & 1], p);
        warp_arrive(&bar_sched_empty[k & 1]);
        return item >= 0;
    };

    if (warp < 8) {
        // ============================================================ compute warpgroups
        setmaxnreg_inc<Cfg::kRegsCompute>();
        const int wg = warp >> 2;
        const int wq = warp & 3;
        const int r_in = wq * 32 + lane;                       // this thread's TMEM lane: key row
        const uint32_t lane_off = (uint32_t)(wq * 32) << 16;
        const uint32_t tX = tmem_base + lane_off + kColX + wg * 64;
        const uint32_t tY = tmem_base + lane_off + kColY + wg * 64;
        const uint32_t tP = tmem_base + lane_off + kColP + wg * kPitchP;
        const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2);
        unsigned char* ds_row = sDS + wg * Cfg::kSubBytes + r_in * 128;    // this thread's 128 bytes of dS^T
        uint32_t git = 0;      // streamed tiles processed so far, over all items (barrier phases)

        for (int k = 0;; ++k) {
            FusedItem w;
            if (!take_item(k, w)) break;
            const int bh = w.bh, off = w.L - w.S;
            const int rrow = w.r0 + r_in;                      // this thread's key
            const bool row_dead = rrow >= w.Lv;                // padding, or past the end of the tensor: P = dS = 0
            FusedStream pos(w, p, kVarlen);
            for (int u = 0; u < w.n_it; ++u, ++git, pos.next(w)) {
                const int c0 = pos.t * 128;                            // first streamed query of this tile
                const float* st_nlse = s_stat + (git & 1) * 256 + wg * 64;
                const float* st_ndelta = st_nlse + 128;
                const bool tr = kTrace && k == 0 && warp == 0 && lane == 0;
                if (tr) TT_B1TRACE(wg, u, 0);
                mbar_wait(&bar_stat_full[git & 1], (git >> 1) & 1, wctx, B1_STAT, u);
                // visible queries of this thread's key inside the tile: [vis_lo, 128)
                int vis_lo = p.causal ? max(0, rrow - off - c0) : 0;
                if (row_dead) vis_lo = 128;
                const bool need_mask = vis_lo > 0;
                // The statistics of a chunk of 32 queries are fetched ahead of the wait for its scores: inside the phases they
                // would sit behind the tensor-memory waits, while shared memory is busy feeding the GEMMs.
                uint64_t stat_reg[16];
                auto load_stats = [&](const float* src) {
#pragma unroll
                    for (int e4 = 0; e4 < 8; ++e4) {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src + e4 * 4);
                        stat_reg[2 * e4] = v.x;
                        stat_reg[2 * e4 + 1] = v.y;
                    }
                };
                uint64_t pf2[32];     // this thread's 64 probabilities, fp32 pairs
                // ---------------- phase A: P^T = exp2(S^T*c - lse2) -> bf16
                // (the mask test stays OUT of the unrolled loop, see the two-pass kernel; and the tensor-memory
                // store stays out of the branch: it is a warp-wide instruction and rows differ in need_mask)
                auto phase_a_body = [&](auto masked_c, int cc, const uint32_t (&sr)[32]) {
                    constexpr bool kMasked = decltype(masked_c)::value;
#pragma unroll
                    for (int e = 0; e < 32; e += 2) {
                        const int col = wg * 64 + cc * 32 + e;
                        const uint64_t x = fma_f32x2(pack_f32x2(__uint_as_float(sr[e]), __uint_as_float(sr[e + 1])), c2, stat_reg[e >> 1]);
                        float a0, a1;
                        unpack_f32x2(x, a0, a1);
                        float p0 = ex2_approx(a0), p1 = ex2_approx(a1);
                        if (kMasked) {
                            p0 = (col >= vis_lo) ? p0 : 0.f;
                            p1 = (col + 1 >= vis_lo) ? p1 : 0.f;
                        }
                        pf2[cc * 16 + (e >> 1)] = pack_f32x2(p0, p1);
                    }
                };
                load_stats(st_nlse);
                mbar_wait(bar_s_full, git & 1, wctx, B1_SFULL, u);
                __syncwarp();
                tc_fence_after();
                if (tr) TT_B1TRACE(wg, u, 1);
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {
                    uint32_t sr[32], pk[16];
                    tmem_ld32(tX + cc * 32, sr);
                    if (cc == 1) load_stats(st_nlse + 32);
                    tmem_wait_ld();
                    if (kApart && cc == 1) {
                        tc_fence_before();
                        warp_arrive(bar_s_read);
                    }
                    if (need_mask) phase_a_body(std::true_type{}, cc, sr);
                    else phase_a_body(std::false_type{}, cc, sr);
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        float q0, q1;
                        unpack_f32x2(pf2[cc * 16 + e], q0, q1);
                        pk[e] = pack_bf16x2(q0, q1);
                    }
                    __syncwarp();
                    if (kApart && cc == 0 && git > 0) {   // complete long ago: P^T(t-1) has been read
                        mbar_wait(bar_p_free, (git - 1) & 1, wctx, B1_PFREE, u);
                        __syncwarp();
                        tc_fence_after();
                    }
                    tmem_st16(tP + cc * 16, pk);
                    if (tr) TT_B1TRACE(wg, u, 2 + cc);
                }
                tmem_wait_st();
                tc_fence_before();
                warp_arrive(bar_p_full);
                if (tr) TT_B1TRACE(wg, u, 4);
                load_stats(st_ndelta);
                // ---------------- phase B: dS^T = P^T * (dP^T - delta) -> bf16 -> shared memory
                mbar_wait(bar_dp_full, git & 1, wctx, B1_DPFULL, u);
                __syncwarp();
                tc_fence_after();
                if (tr) TT_B1TRACE(wg, u, 5);
                if (git > 0) mbar_wait(bar_ds_free, (git - 1) & 1, wctx, B1_DSFREE, u);   // complete long ago
                __syncwarp();
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {
                    uint32_t dr[32];
                    tmem_ld32(tY + cc * 32, dr);
                    if (cc == 1) load_stats(st_ndelta + 32);
                    tmem_wait_ld();
                    uint32_t pk[16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const uint64_t tdiff = add_f32x2(pack_f32x2(__uint_as_float(dr[2 * e]), __uint_as_float(dr[2 * e + 1])), stat_reg[e]);
                        const uint64_t ds = mul_f32x2(pf2[cc * 16 + e], tdiff);
                        float x0, x1;
                        unpack_f32x2(ds, x0, x1);
                        pk[e] = pack_bf16x2(x0, x1);
                    }
                    // 16-byte chunk j of row r sits at chunk j ^ (r & 7) of the row (128-byte swizzle)
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj)
                        *reinterpret_cast<uint4*>(ds_row + (((cc * 4 + jj) ^ (r_in & 7)) << 4)) =
                            make_uint4(pk[4 * jj], pk[4 * jj + 1], pk[4 * jj + 2], pk[4 * jj + 3]);
                }
                fence_proxy_async_smem();          // generic-proxy stores -> visible to the MMA's async-proxy reads
                tc_fence_before();
                warp_arrive(bar_ds_full);
                if (lane == 0) mbar_arrive(&bar_stat_empty[git & 1]);
                if (tr) TT_B1TRACE(wg, u, 6);
            }
            // ---------------- epilogue: dV, dK out of tensor memory (then the MMA warp may start the next
            // item in them) -> bf16 -> global; warpgroup w owns columns [w*D/2, +D/2)
            mbar_wait(bar_final, k & 1, wctx, B1_FINAL, k);
            __syncwarp();
            tc_fence_after();
            constexpr int kHalf = D / 2;
            uint32_t o16[2][kHalf / 2];
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                uint32_t acc[kHalf];
                const uint32_t tA = tmem_base + lane_off + (a == 0 ? kColDV : kColDK) + wg * kHalf;
#pragma unroll
                for (int cc = 0; cc < kHalf / 32; ++cc) tmem_ld32(tA + cc * 32, reinterpret_cast<uint32_t(&)[32]>(acc[cc * 32]));
                tmem_wait_ld();
                const float mul = a == 0 ? 1.0f : p.scale;
#pragma unroll
                for (int e = 0; e < kHalf / 2; ++e)   // gradients of padded keys are zero
                    o16[a][e] = row_dead ? 0u : pack_bf16x2(__uint_as_float(acc[2 * e]) * mul, __uint_as_float(acc[2 * e + 1]) * mul);
            }
            tc_fence_before();
            warp_arrive(bar_acc_free);
            if (rrow < w.L) {
                const long long o = (kVarlen ? (long long)(w.k_lo + rrow) * p.Hkv + w.head : (long long)bh * w.L + rrow) * D + wg * kHalf;
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    __nv_bfloat16* dst = (a == 0 ? p.out0 : p.out1) + o;
#pragma unroll
                    for (int e = 0; e < kHalf / 2; e += 8) {
                        if (p.wide_stores) {
                            st_global_32B(dst + 2 * e, reinterpret_cast<const uint32_t(&)[8]>(o16[a][e]));
                        } else {
                            *reinterpret_cast<uint4*>(dst + 2 * e) = make_uint4(o16[a][e], o16[a][e + 1], o16[a][e + 2], o16[a][e + 3]);
                            *reinterpret_cast<uint4*>(dst + 2 * e + 8) = make_uint4(o16[a][e + 4], o16[a][e + 5], o16[a][e + 6], o16[a][e + 7]);
                        }
                    }
                }
            }
            __syncwarp();
        }
    } else if (warp < 12) {
        setmaxnreg_inc<Cfg::kRegsAdd>();

        // ============================================================ the adding warpgroup: dQ_t out of tensor memory (thread
        // <-> query row), through shared memory into the accumulator.  Its own warps, because a piece's buffer is free again only
        // when the L2 has taken what was in it: the 64 KB of a tile at D = 128 need 2400 to 3200 cycles with every SM adding.
        const int r_in = (warp & 3) * 32 + lane;
        const uint32_t tDQ = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + kColDQ;
        uint32_t git = 0, chunk = 0;
        for (int k = 0;; ++k) {
            // Warp 8 reads the item for all four: the named barriers below need the same items and tiles in each, whatever a
            // wait returned.  A slot is written again two items on, behind the barrier of the item between.
            PackedItem* mine = &add_item[k & 1];
            if (warp == 8) {
                const int item = next_item(k);
                if (lane == 0) {
                    if (kVarlen) *mine = packed[k & 1];
                    mine->item = item;
                }
                warp_arrive(&bar_sched_empty[k & 1]);
            }
            named_bar_sync(1, 128);
            const int item = mine->item;
            if (item < 0) break;
            const FusedItem w = fused_item<kVarlen>(item, mine, p);
            FusedStream pos(w, p, kVarlen);
            for (int u = 0; u < w.n_it; ++u, ++git, pos.next(w)) {
                float* dst = p.dq_acc + (size_t)((long long)pos.slice * p.n_qt + w.blk0 + pos.t) * (D / 4) * 512;
                uint32_t r[D / 32][32];
                auto add = [&](int cc) {
                    float4* stage = reinterpret_cast<float4*>(sStage + (chunk & 1) * Cfg::kStageBytes);
                    if (warp == 8) bulk_wait_read<1>();        // what left this buffer two chunks ago has been read
                    named_bar_sync(1, 128);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        stage[j * 128 + r_in] = make_float4(__uint_as_float(r[cc][4 * j]), __uint_as_float(r[cc][4 * j + 1]),
                                                            __uint_as_float(r[cc][4 * j + 2]), __uint_as_float(r[cc][4 * j + 3]));
                    fence_proxy_async_smem();
                    named_bar_sync(1, 128);
                    if (warp == 8 && lane == 0) bulk_add_f32(dst + cc * 8 * 512, stage, Cfg::kStageBytes);
                    __syncwarp();
                    ++chunk;
                };
                const bool tr = kTrace && k == 0 && warp == 8 && lane == 0;
                if (tr) TT_B1TRACE(1, u, 0);
                mbar_wait(bar_dq_full, git & 1, wctx, B1_DQFULL, u);
                __syncwarp();
                tc_fence_after();
                if (tr) TT_B1TRACE(1, u, 1);
#pragma unroll
                for (int cc = 0; cc < D / 32; ++cc) tmem_ld32(tDQ + cc * 32, r[cc]);
                tmem_wait_ld();
                tc_fence_before();
                warp_arrive(bar_dq_free);
                if (tr) TT_B1TRACE(1, u, 2);
#pragma unroll
                for (int cc = 0; cc < D / 32; ++cc) add(cc);
                if (tr) TT_B1TRACE(1, u, 3);
            }
        }
        if (warp == 8) bulk_wait_all();
    } else {
        setmaxnreg_dec<Cfg::kRegsOther>();
        if (warp == 13) {
            // ============================================================ TMA loader + scheduler (whole
            // warp runs the control flow, one elected lane issues)
            auto load_tile = [&](unsigned char* dst, const CUtensorMap* tm, uint64_t* bar, int row_start, int bh) {
#pragma unroll
                for (int sb = 0; sb < Cfg::kSub; ++sb) tma_load_3d(dst + sb * Cfg::kSubBytes, tm, bar, sb * 64, row_start, bh);
            };
            uint32_t git = 0;
            int item = (int)blockIdx.x;
            // keys that no query sees: zero gradients, and nothing of them is read
            auto zero_keys = [&](long long row, int pitch, int rows) {
                for (int i = lane; i < rows * (D / 8); i += 32) {
                    const long long o = (row + (long long)(i / (D / 8)) * pitch) * D + i % (D / 8) * 8;
                    *reinterpret_cast<uint4*>(p.out0 + o) = make_uint4(0u, 0u, 0u, 0u);
                    *reinterpret_cast<uint4*>(p.out1 + o) = make_uint4(0u, 0u, 0u, 0u);
                }
            };
            for (int k = 0;; ++k, item = items.next(wctx, 89, k)) {
                const int slot = k & 1;
                PackedItem pi;
                while (kVarlen && item >= 0) {
                    const int x = item / p.Hkv, b = packed_seq<7>(p.cu_k, p.n_seq, x);
                    bool some = false;
                    if (b >= 0) {
                        pi.k_lo = p.cu_k[b];
                        pi.q_lo = p.cu_q[b];
                        pi.L = p.cu_k[b + 1] - pi.k_lo;
                        pi.S = p.cu_q[b + 1] - pi.q_lo;
                        pi.tile0 = (pi.q_lo >> 7) + b;
                        const int base = (pi.k_lo >> 7) + b, n = ((pi.k_lo + pi.L) >> 7) + 1 - (pi.k_lo >> 7);   // numbers of the sequence
                        const int r = item - base * p.Hkv;
                        pi.head = r / n;
                        pi.r0 = (r - pi.head * n) * 128;
                        if (pi.head < p.Hkv && pi.r0 < pi.L) {
                            some = fused_item<true>(item, &pi, p).n_it > 0;
                            if (!some) zero_keys((long long)(pi.k_lo + pi.r0) * p.Hkv + pi.head, p.Hkv, min(128, pi.L - pi.r0));
                        }
                    }
                    if (some) break;
                    items.request(*abort_flag != 0);
                    item = items.next(wctx, 89, k);
                }
                while (!kVarlen && p.kv_lens != nullptr && item >= 0) {   // tiles that are all padding
                    const FusedItem w = fused_item<false>(item, nullptr, p);
                    if (w.r0 < w.Lv) break;
                    zero_keys((long long)w.bh * w.L + w.r0, 1, min(128, w.L - w.r0));
                    items.request(*abort_flag != 0);
                    item = items.next(wctx, 89, k);
                }
                // a wait that gave up: somebody may still read the slot, and parts of two items would name rows of neither
                if (!__all_sync(0xffffffffu, mbar_wait(&bar_sched_empty[slot], ((k >> 1) & 1) ^ 1, wctx, 90 + slot, k))) break;
                if (lane == 0) {
                    sched_item[slot] = item;
                    if (kVarlen) packed[slot] = pi;
                    mbar_arrive(&bar_sched_full[slot]);
                }
                __syncwarp();
                if (item < 0) break;
                const FusedItem w = fused_item<kVarlen>(item, &pi, p);
                const int key_row = (kVarlen ? w.k_lo : 0) + w.r0, key_z = kVarlen ? w.head : w.bh, q_row = kVarlen ? w.q_lo : 0;
                mbar_wait(bar_res_empty, (k & 1) ^ 1, wctx, B1_RES + 1, k);
                __syncwarp();
                if (elect_one()) {
                    mbar_arrive_expect_tx(bar_res_full, 2 * Cfg::kTileBytes);
                    load_tile(sK, &tmK, bar_res_full, key_row, key_z);
                    load_tile(sV, &tmV, bar_res_full, key_row, key_z);
                }
                __syncwarp();
                FusedStream pos(w, p, kVarlen);
                for (int u = 0; u < w.n_it; ++u, ++git, pos.next(w)) {
                    const int s0 = git % kNQ, s1 = git % kNdO, t = pos.t, ts = pos.slice;
                    mbar_wait(&bar_stat_empty[git & 1], ((git >> 1) & 1) ^ 1, wctx, B1_STAT + 10, (int)git);
                    __syncwarp();
                    if (elect_one()) {
                        const long long at = ((long long)ts * p.n_qt + w.blk0 + t) * 128;
                        float* dst = s_stat + (git & 1) * 256;
                        mbar_arrive_expect_tx(&bar_stat_full[git & 1], Cfg::kStatBytes);
                        bulk_load(dst, p.lse2 + at, Cfg::kStatBytes / 2, &bar_stat_full[git & 1]);
                        bulk_load(dst + 128, p.delta + at, Cfg::kStatBytes / 2, &bar_stat_full[git & 1]);
                    }
                    __syncwarp();
                    mbar_wait(&bar_q_empty[s0], ((git / kNQ) & 1) ^ 1, wctx, B1_QEMPTY + s0, (int)git);
                    __syncwarp();
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&bar_q_full[s0], Cfg::kTileBytes);
                        load_tile(sQ + s0 * Cfg::kTileBytes, &tmQ, &bar_q_full[s0], q_row + t * 128, ts);
                    }
                    __syncwarp();
                    mbar_wait(&bar_do_empty[s1], ((git / kNdO) & 1) ^ 1, wctx, B1_DOEMPTY + s1, (int)git);
                    __syncwarp();
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&bar_do_full[s1], Cfg::kTileBytes);
                        load_tile(sdO + s1 * Cfg::kTileBytes, &tmdO, &bar_do_full[s1], q_row + t * 128, ts);
                    }
                    __syncwarp();
                }
                items.request(*abort_flag != 0);   // an aborted CTA takes no further items
            }
        } else if (warp == 12) {
            // ============================================================ MMA issuer (whole warp runs the
            // control flow; each tcgen05.mma / commit is issued by one elected lane)
            constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, false, false);   // S^T, dP^T: both K-major
            constexpr uint32_t idesc_kn = umma_idesc_bf16(128, D, false, true);     // dV, dK: A K-major, B MN-major
            constexpr uint32_t idesc_nn = umma_idesc_bf16(128, D, true, true);      // dQ_t: A and B MN-major
            // Every operand lives at a fixed offset of the CTA's shared memory, so two descriptor templates
            // (K-major and MN-major view of the base) plus compile-time offsets describe them all.
            const uint32_t smem_addr = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
            const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
            constexpr uint32_t hi = umma_desc_hi(1024);
            const uint32_t desc_k = umma_desc_lo(smem_addr, 16);                  // K-major: rows = M or N, 128 B of K per row
            const uint32_t desc_mn = umma_desc_lo(smem_addr, Cfg::kSubBytes);     // MN-major: rows = K, 64 elements of M/N per row
            constexpr uint32_t kOffK = 0, kOffV = Cfg::kTileBytes, kOffQ = 2 * Cfg::kTileBytes,
                               kOffdO = (2 + kNQ) * Cfg::kTileBytes, kOffDS = (2 + kNQ + kNdO) * Cfg::kTileBytes;
            const uint32_t dK_k = desc_k + (kOffK >> 4);        // K as A of G1
            const uint32_t dK_mn = desc_mn + (kOffK >> 4);      // K as B of G5
            const uint32_t dV_k = desc_k + (kOffV >> 4);        // V as A of G2
            const uint32_t dQ_k = desc_k + (kOffQ >> 4);        // Q as B of G1
            const uint32_t dQ_mn = desc_mn + (kOffQ >> 4);      // Q as B of G4
            const uint32_t ddO_k = desc_k + (kOffdO >> 4);      // dO as B of G2
            const uint32_t ddO_mn = desc_mn + (kOffdO >> 4);    // dO as B of G3
            const uint32_t dDS_k = desc_k + (kOffDS >> 4);      // dS^T as A of G4 (K-major: K = queries)
            const uint32_t dDS_mn = desc_mn + (kOffDS >> 4);    // dS^T as A of G5 (MN-major: M = queries)
            // G1 / G2: tmem[col] = A B^T over K = D, both operands K-major tiles of D/64 sub-blocks
            auto issue_score = [&](uint32_t a0, uint32_t b0, uint32_t col) {
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint32_t o = ((kk >> 2) * Cfg::kSubBytes + (kk & 3) * 32) >> 4;
                        umma_ss_one(tmem_u + col, a0 + o, b0 + o, hi, idesc_s, kk > 0);
                    }
                }
                __syncwarp();
            };
            uint32_t git = 0;      // streamed tiles issued before the current item
            for (int k = 0;; ++k) {
                FusedItem w;
                if (!take_item(k, w)) break;
                __syncwarp();
                const int n_it = w.n_it;
                mbar_wait(bar_res_full, k & 1, wctx, B1_RES, k);
                __syncwarp();
                if (n_it > 0) {
                    // first scores of the item.  X is free: the G3 that read the previous P^T was issued
                    // earlier by this warp and executes in order.  Y holds the previous tile's dQ_t until
                    // the adding warps have taken it (D = 64: columns of its own).
                    const int f0 = git % kNQ, f1 = git % kNdO;
                    mbar_wait(&bar_q_full[f0], (git / kNQ) & 1, wctx, B1_QFULL + f0, (int)git);
                    __syncwarp();
                    tc_fence_after();
                    issue_score(dK_k, dQ_k + f0 * (Cfg::kTileBytes >> 4), kColX);
                    tc_commit(bar_s_full);
                    mbar_wait(&bar_do_full[f1], (git / kNdO) & 1, wctx, B1_DOFULL + f1, (int)git);
                    __syncwarp();
                    if (!kApart && git > 0) {
                        mbar_wait(bar_dq_free, (git - 1) & 1, wctx, B1_DQFREE, (int)git);
                        __syncwarp();
                    }
                    tc_fence_after();
                    issue_score(dV_k, ddO_k + f1 * (Cfg::kTileBytes >> 4), kColY);
                    tc_commit(bar_dp_full);
                }
                for (int it = 0; it < n_it; ++it) {
                    const uint32_t g = git + it;
                    const int qs = g % kNQ, os = g % kNdO;                   // slots of this tile
                    const bool has_next = it + 1 < n_it;
                    const int nqs = (g + 1) % kNQ, nos = (g + 1) % kNdO;     // slots of the next tile
                    // ---- G1(t+1): the next scores, as soon as the columns of S^T(t) are free: its values are in registers, or
                    // (P^T in the same columns) G3(t) has been issued
                    auto next_scores = [&] {
                        if (!has_next) return;
                        mbar_wait(&bar_q_full[nqs], ((g + 1) / kNQ) & 1, wctx, B1_QFULL + nqs, it + 1);
                        __syncwarp();
                        tc_fence_after();
                        issue_score(dK_k, dQ_k + nqs * (Cfg::kTileBytes >> 4), kColX);
                        tc_commit(bar_s_full);
                    };
                    if (kApart) {
                        mbar_wait(bar_s_read, g & 1, wctx, B1_SREAD, it);
                        __syncwarp();
                        next_scores();
                    }
                    // ---- G3: dV += P^T dO
                    const bool tr = kTrace && k == 0 && lane == 0;
                    if (tr) TT_B1TRACE(2, it, 0);
                    mbar_wait(bar_p_full, g & 1, wctx, B1_PFULL, it);
                    __syncwarp();
                    tc_fence_after();
                    if (tr) TT_B1TRACE(2, it, 1);
                    if (it == 0) {
                        // the accumulator columns must have been read out by the previous item's epilogue
                        mbar_wait(bar_acc_free, (k & 1) ^ 1, wctx, B1_ACCFREE, k);
                        __syncwarp();
                        tc_fence_after();
                    }
                    {
                        const uint32_t b0 = ddO_mn + os * (Cfg::kTileBytes >> 4);
                        if (elect_one()) {
#pragma unroll
                            for (int kk = 0; kk < 8; ++kk)   // K step = 16 queries = 8 columns of bf16 P^T
                                umma_ts_one(tmem_u + kColDV, tmem_u + kColP + (kk >> 2) * kPitchP + (kk & 3) * 8, b0 + kk * 128, hi, idesc_kn,
                                            (it > 0 || kk > 0) ? 1u : 0u);
                        }
                        __syncwarp();
                    }
                    tc_commit(&bar_do_empty[os]);                            // last read of dO(t)
                    if (kApart) tc_commit(bar_p_free);
                    else next_scores();
                    // ---- G5: dQ_t = dS K  and  G4: dK += dS^T Q
                    if (tr) TT_B1TRACE(2, it, 2);
                    mbar_wait(bar_ds_full, g & 1, wctx, B1_DSFULL, it);
                    __syncwarp();
                    tc_fence_after();
                    if (tr) TT_B1TRACE(2, it, 3);
                    // ---- G2(t+1): the next dP^T, once dP^T(t) is in registers and, where it uses these columns, dQ_t has left
                    auto next_dp = [&] {
                        if (!has_next) return;
                        mbar_wait(&bar_do_full[nos], ((g + 1) / kNdO) & 1, wctx, B1_DOFULL + nos, it + 1);
                        __syncwarp();
                        if (!kApart) {
                            mbar_wait(bar_dq_free, g & 1, wctx, B1_DQFREE, it);
                            __syncwarp();
                        }
                        tc_fence_after();
                        if (tr) TT_B1TRACE(2, it, 5);
                        issue_score(dV_k, ddO_k + nos * (Cfg::kTileBytes >> 4), kColY);
                        tc_commit(bar_dp_full);
                    };
                    if (kApart) {
                        next_dp();
                        if (g > 0) {
                            mbar_wait(bar_dq_free, (g - 1) & 1, wctx, B1_DQFREE, it);
                            __syncwarp();
                            tc_fence_after();
                        }
                    }
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)       // K step = 16 keys = 16 rows of both tiles
                            umma_ss_one(tmem_u + kColDQ, dDS_mn + kk * 128, dK_mn + kk * 128, hi, idesc_nn, kk > 0 ? 1u : 0u);
                    }
                    __syncwarp();
                    tc_commit(bar_dq_full);
                    {
                        const uint32_t b0 = dQ_mn + qs * (Cfg::kTileBytes >> 4);
                        if (elect_one()) {
#pragma unroll
                            for (int kk = 0; kk < 8; ++kk)   // K step = 16 queries: 32 bytes along a dS^T row, 16 rows of Q
                                umma_ss_one(tmem_u + kColDK, dDS_k + (((kk >> 2) * Cfg::kSubBytes + (kk & 3) * 32) >> 4), b0 + kk * 128, hi,
                                            idesc_kn, (it > 0 || kk > 0) ? 1u : 0u);
                        }
                        __syncwarp();
                    }
                    tc_commit(&bar_q_empty[qs]);                             // last read of Q(t)
                    tc_commit(bar_ds_free);                                  // G4, G5 are done with the dS^T tile
                    if (!has_next) tc_commit(bar_res_empty);                 // the item's last reads of K and V
                    if (tr) TT_B1TRACE(2, it, 4);
                    if (!kApart) next_dp();
                    if (tr) TT_B1TRACE(2, it, 6);
                }
                tc_commit(bar_final);
                git += (uint32_t)n_it;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 12) {
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
    if (warp == 13 && *abort_flag) items.drop_rest(wctx.budget);
}

// Statistics as the kernel above streams them: -lse*log2(e) and -rowsum(dO*O), 128 per query tile of a slice (what lies past
// the slice's last row makes P and dS zero), and the tile's dQ accumulator cleared.  D/8 lanes share a row.
// Packed batches: a block's tile is found in the numbering of packed_seq; tokens of no sequence get zero gradients here.
struct PackedBatch {
    const int *cu_q, *cu_k;
    int n_seq, total_q, total_k, H, Hkv;
    __nv_bfloat16 *dq, *dk, *dv;
};
struct TileRows {
    int n;                   // rows that exist (none where not positive)
    long long row0, pitch;   // row r of the tile is row row0 + r * pitch of a [rows, D] array
    long long stat0;         // its log-sum-exp is lse[stat0 + r]
};
template <bool kVarlen>
__device__ __forceinline__ TileRows tile_rows(long long blk, int S, int n_qt, const PackedBatch& b) {
    const long long s = blk / n_qt;
    const int t = (int)(blk - s * n_qt);
    if constexpr (kVarlen) {
        const int i = packed_seq<7>(b.cu_q, b.n_seq, t);
        if (i < 0) return {0, 0, 0, 0};
        const int lo = b.cu_q[i], r0 = (t - (lo >> 7) - i) * 128;
        return {min(128, b.cu_q[i + 1] - lo - r0), (long long)(lo + r0) * b.H + s, b.H, s * b.total_q + lo + r0};
    } else {
        return {min(128, S - t * 128), s * S + t * 128, 1, s * S + t * 128};
    }
}
__device__ __forceinline__ void zero_other_tokens(__nv_bfloat16* t, const int* cu, int n_seq, int total, int width) {
    const int lo = cu[0], hi = cu[n_seq], n = lo + total - hi;
    for (long long i = blockIdx.x; i < n; i += gridDim.x) {
        uint4* dst = reinterpret_cast<uint4*>(t + (i < lo ? i : i - lo + hi) * width);
        for (int e = threadIdx.x; e < width / 8; e += blockDim.x) dst[e] = make_uint4(0u, 0u, 0u, 0u);
    }
}
template <int D, bool kVarlen>
__global__ void __launch_bounds__(256) attn_bwd_fused_prep_kernel(const __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ dout,
                                                                  const float* __restrict__ lse, float* __restrict__ ndelta,
                                                                  float* __restrict__ nlse2, float4* __restrict__ dq_acc, int S, int n_qt, const PackedBatch pb) {
    grid_let_next_start();
    grid_wait_for_previous();
    constexpr int kLanes = D / 8, kRows = 256 / kLanes, kSteps = 128 / kRows;   // a CTA takes one query tile
    const long long blk = blockIdx.x;
    const int li = threadIdx.x % kLanes;
    const TileRows w = tile_rows<kVarlen>(blk, S, n_qt, pb);
    uint4 a[kSteps], b[kSteps];
#pragma unroll
    for (int u = 0; u < kSteps; ++u) {
        const int r = u * kRows + (int)threadIdx.x / kLanes;
        a[u] = b[u] = make_uint4(0u, 0u, 0u, 0u);
        if (r < w.n) {
            const long long at = (w.row0 + r * w.pitch) * D + li * 8;
            a[u] = __ldg(reinterpret_cast<const uint4*>(out + at));
            b[u] = __ldg(reinterpret_cast<const uint4*>(dout + at));
        }
    }
#pragma unroll
    for (int i = 0; i < D / 8; ++i) dq_acc[blk * (D * 32) + i * 256 + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < kSteps; ++u) {
        const int r = u * kRows + (int)threadIdx.x / kLanes;
        const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, bw[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
        float acc = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            acc = fmaf(__uint_as_float(aw[e] << 16), __uint_as_float(bw[e] << 16), acc);
            acc = fmaf(__uint_as_float(aw[e] & 0xffff0000u), __uint_as_float(bw[e] & 0xffff0000u), acc);
        }
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (li == 0) {
            const float l = r < w.n ? lse[w.stat0 + r] : INFINITY;
            ndelta[blk * 128 + r] = -acc;
            nlse2[blk * 128 + r] = (kVarlen && l == -INFINITY) ? -INFINITY : l * -1.4426950408889634f;   // a row that sees no key: P = 0
        }
    }
    if (kVarlen) {
        zero_other_tokens(pb.dq, pb.cu_q, pb.n_seq, pb.total_q, pb.H * D);
        zero_other_tokens(pb.dk, pb.cu_k, pb.n_seq, pb.total_k, pb.Hkv * D);
        zero_other_tokens(pb.dv, pb.cu_k, pb.n_seq, pb.total_k, pb.Hkv * D);
    }
}

// dq[slice][row][:] = bf16(scale * accumulator): one block per (query slice, 128-row query tile), thread
// (row, half of the head dim).  Reads are 16 bytes per lane and contiguous across the rows of a warp; four
// of them make the 32 contiguous bytes (one full sector) a lane writes.
template <int D, bool kVarlen>
__global__ void __launch_bounds__(256) attn_bwd_dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq,
                                                                 int S, int n_qt, float scale, int wide, const PackedBatch pb) {
    grid_let_next_start();
    grid_wait_for_previous();
    const long long blk = blockIdx.x;            // qs * n_qt + t
    const TileRows w = tile_rows<kVarlen>(blk, S, n_qt, pb);
    const int r = threadIdx.x & 127, h = threadIdx.x >> 7;
    if (r >= w.n) return;
    const float4* src = reinterpret_cast<const float4*>(acc) + (size_t)blk * (D / 4) * 128 + r;
    __nv_bfloat16* dst = dq + (w.row0 + r * w.pitch) * D + h * (D / 2);
#pragma unroll
    for (int c = 0; c < D / 8; c += 4) {
        uint32_t o8[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 a = src[(size_t)(h * (D / 8) + c + i) * 128];
            o8[2 * i] = pack_bf16x2(a.x * scale, a.y * scale);
            o8[2 * i + 1] = pack_bf16x2(a.z * scale, a.w * scale);
        }
        if (wide) {
            st_global_32B(dst + c * 4, o8);
        } else {
            *reinterpret_cast<uint4*>(dst + c * 4) = make_uint4(o8[0], o8[1], o8[2], o8[3]);
            *reinterpret_cast<uint4*>(dst + c * 4 + 8) = make_uint4(o8[4], o8[5], o8[6], o8[7]);
        }
    }
}

// ---------------------------------------------------------------- host side
bool attn_bwd_fused_supported(const AttnArgs& a) {
    return a.bf16 && (a.D == 64 || a.D == 128) && a.BH * (((long long)a.S + 127) / 128) < (1LL << 31) &&
           (!a.cu_q || (a.H * (a.total_q / 128 + a.BH / a.H) < (1LL << 31) && a.H * (a.total_k / 128 + a.BH / a.H) < (1LL << 31)));
}
// query tiles: of every slice, or of every head over a packed batch's numbering (packed_seq)
static int fused_tiles(const AttnArgs& a) { return a.cu_q ? (int)(a.total_q / 128 + a.BH / a.H) : (a.S + 127) / 128; }
static long long fused_blocks(const AttnArgs& a) { return (a.cu_q ? a.H : a.BH) * (long long)fused_tiles(a); }
size_t attn_bwd_fused_workspace(const AttnArgs& a) {
    return (size_t)fused_blocks(a) * 128 * (a.D + 2) * sizeof(float);   // dQ accumulator, two statistics
}

static long long* g_fused_trace = nullptr;
static int g_fused_trace_block = 0;
void attn_bwd_fused_set_trace(long long* device_buf, int block) {
    g_fused_trace = device_buf;
    g_fused_trace_block = block;
}

template <int D, bool kTrace, bool kVarlen>
static cudaError_t launch_fused(const AttnArgs& a, void* ws, cudaStream_t st) {
    using Cfg = Bwd1Cfg<D>;
    const int n_qt = fused_tiles(a), hkv = a.H / a.group;
    const long long n_blk = fused_blocks(a);
    const size_t rows = (size_t)n_blk * 128;
    const PackedBatch pb = {a.cu_q, a.cu_k, (int)(a.BH / a.H), (int)a.total_q, (int)a.total_k, a.H, hkv, (__nv_bfloat16*)a.dq, (__nv_bfloat16*)a.dk, (__nv_bfloat16*)a.dv};
    float* dq_acc = reinterpret_cast<float*>(ws);
    float* delta = dq_acc + rows * D;
    float* lse2 = delta + rows;
    cudaError_t e;
    {
        LaunchScope ls(K_BWD_PREP, st);
        e = launch_overlapped(attn_bwd_fused_prep_kernel<D, kVarlen>, (unsigned)n_blk, 256, 0, st, (const __nv_bfloat16*)a.out, (const __nv_bfloat16*)a.dout,
                              a.lse, delta, lse2, reinterpret_cast<float4*>(dq_acc), a.S, n_qt, pb);
        if (e != cudaSuccess) return e;
    }
    TmapStorage tq, tk, tv, tdo;
    const char* why = nullptr;
    if (kVarlen) {
        if (!make_tmap_bf16_strided(&tq, a.q, D, a.total_q, a.H, (uint64_t)a.H * D, D, 128, &why)) return cudaErrorInvalidValue;
        if (!make_tmap_bf16_strided(&tdo, a.dout, D, a.total_q, a.H, (uint64_t)a.H * D, D, 128, &why)) return cudaErrorInvalidValue;
        if (!make_tmap_bf16_strided(&tk, a.k, D, a.total_k, hkv, (uint64_t)hkv * D, D, 128, &why)) return cudaErrorInvalidValue;
        if (!make_tmap_bf16_strided(&tv, a.v, D, a.total_k, hkv, (uint64_t)hkv * D, D, 128, &why)) return cudaErrorInvalidValue;
    } else {
        if (!make_tmap_bf16(&tq, a.q, D, a.S, a.BH, 128, &why)) return cudaErrorInvalidValue;
        if (!make_tmap_bf16(&tk, a.k, D, a.L, a.BH / a.group, 128, &why)) return cudaErrorInvalidValue;
        if (!make_tmap_bf16(&tv, a.v, D, a.L, a.BH / a.group, 128, &why)) return cudaErrorInvalidValue;
        if (!make_tmap_bf16(&tdo, a.dout, D, a.S, a.BH, 128, &why)) return cudaErrorInvalidValue;
    }
    auto M = [](TmapStorage& t) -> CUtensorMap& { return *reinterpret_cast<CUtensorMap*>(t.bytes); };
    e = TT_ALLOW_SMEM((attn_bwd_fused_sm100_kernel<D, kTrace, kVarlen>), Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    BwdParams p;
    memset(&p, 0, sizeof(p));
    p.out0 = (__nv_bfloat16*)a.dv;
    p.out1 = (__nv_bfloat16*)a.dk;
    p.lse2 = lse2;
    p.delta = delta;
    p.S = a.S;
    p.L = a.L;
    p.causal = a.causal;
    p.scale = a.scale;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    p.status = device_status_word();
    p.group = a.group;
    p.kv_lens = a.kv_lens;
    p.H = a.H;
    const uintptr_t al = reinterpret_cast<uintptr_t>(a.dk) | reinterpret_cast<uintptr_t>(a.dv);
    p.wide_stores = (al & 31) == 0 ? 1 : 0;
    p.Hkv = hkv;
    p.cu_q = a.cu_q;
    p.cu_k = a.cu_k;
    p.n_seq = pb.n_seq;
    p.n_tiles = (a.L + 127) / 128;
    p.n_items = kVarlen ? (int)(hkv * (a.total_k / 128 + pb.n_seq)) : (int)(a.BH / a.group * p.n_tiles);
    p.n_light = a.causal ? p.n_tiles / 4 : 0;
    p.n_items_heavy = (int)(a.BH / a.group * (p.n_tiles - p.n_light));
    p.dq_acc = dq_acc;
    p.n_qt = n_qt;
    p.trace = kTrace ? g_fused_trace : nullptr;
    p.trace_block = g_fused_trace_block;
    p.first_wave = sm_count();
    {
        LaunchScope ls(K_BWD_FUSED, st);
        launch_overlapped(attn_bwd_fused_sm100_kernel<D, kTrace, kVarlen>, (unsigned)p.n_items, Cfg::kThreads, Cfg::kSmemBytes, st, M(tk), M(tv), M(tq), M(tdo), p);
    }
    {
        LaunchScope ls(K_BWD_DQ_CONVERT, st);
        launch_overlapped(attn_bwd_dq_convert_kernel<D, kVarlen>, (unsigned)n_blk, 256, 0, st, dq_acc, (__nv_bfloat16*)a.dq, a.S, n_qt, a.scale,
                          (reinterpret_cast<uintptr_t>(a.dq) & 31) == 0 ? 1 : 0, pb);
    }
    return cudaGetLastError();
}

cudaError_t attn_bwd_fused(const AttnArgs& a, void* ws, cudaStream_t st) {
    if (a.cu_q != nullptr) return a.D == 128 ? launch_fused<128, false, true>(a, ws, st) : launch_fused<64, false, true>(a, ws, st);
    if (g_fused_trace != nullptr) return a.D == 128 ? launch_fused<128, true, false>(a, ws, st) : launch_fused<64, true, false>(a, ws, st);
    return a.D == 128 ? launch_fused<128, false, false>(a, ws, st) : launch_fused<64, false, false>(a, ws, st);
}

// ---------------------------------------------------------------- choice between the two kernels
static std::atomic<int> g_bwd_deterministic{-1};   // -1: the caller has not said
void attn_bwd_set_deterministic(int on) { g_bwd_deterministic.store(on ? 1 : 0); }

// The single pass has only the key tiles' items to fill the SMs with, and clears, adds to and converts an accumulator; the two
// passes execute seven GEMMs for five, and up to 1.8 items per SM run both in one launch, whose items fill the SMs better.
// Backward in us, single pass / two passes (items per SM; streamed tiles per item):
//   D = 64   [8,16,1024] causal 105 / 121 (6.9; 4), [16,32,512] causal 159 / 168 (14; 2), [1,8,5000] causal 127 / 153 (2.2; 20), [4,16,700]
//            58 / 60 (2.6; 6), but [7,8,600] 40.5 / 39.3 (1.9; 5), [4,32,300] causal 42.6 / 40.7 (2.6; 2), [16,32,128] causal 40.0 / 38.6 (3.5; 1).
//            The dQ pass of few queries is as long as the chain of key tiles that each of its items walks (1800 cycles a tile, 3125 in the
//            single pass): against 9000 keys [1,4,300] 29 / 80, 12000 [1,4,128] 24 / 94, 3000 [1,8,100] 21 / 31, 4096 [1,64,128] 85 / 88, but
//            2048 [1,100,128] 72 / 64, 2000 [3,32,100] 66 / 63, 578 [1,2,106] 11.7 / 10.3.
//            One launch: full waves of long walks pay, [1,16,2048] 76 / 87 (1.7; 16), [1,4,4096] 74 / 82 (0.86; 32), [2,16,1024] 50 / 53
//            (1.7; 8), but [4,16,512] 36.9 / 35.5 (1.7; 4), [1,8,3000] 107 / 89 (1.3; 24), [1,1,20000] 534 / 483 (1.06; 157); causal ones
//            where they are longer still, [1,4,8192] 148 / 162 (1.7; 32), [1,2,16384] 237 / 283 (1.7; 64), [2,2,6900] 109 / 120 (1.5; 27),
//            [1,16/4,8192] 534 / 570, but [1,8,4096] 94.4 / 93.8 (1.7; 16), [1,16/8,4096] 168 / 159, [1,2,12288] 176 / 170 (1.3; 48),
//            [1,4,4096] 73 / 55 (0.86; 16).
//   D = 128  [4,32,4096] causal 1614 / 1700 (28; 16), [4,32,2048] causal 517 / 538 (14; 8), [4,32,1536] 509 / 523 (10; 12), [1,32,4096]
//            740 / 775 (6.9; 32), [1,32/8,8192] causal 1550 / 1600 (3.5; 32 of each head), but [4,32,1024] 259 / 255 (6.9; 8), [1,16,4096]
//            causal 226 / 220 (3.5; 16), [4,64/8,2048] causal 1053 / 1014 (3.5; 8 of each head).
//   packed   (the two passes clear the gradients and number their items for the longest sequence) 16 of 300 to 4096, 32 heads, causal
//            1236 / 1550 at D = 64, 2085 / 2330 at D = 128; 24 of 512 434 / 461, 64 of 256 490 / 483, 64 of 128 156 / 165 at D = 64, but 262 / 239
//            at D = 128.  Grouped heads at D = 128 have fewer items, and a dQ pass of as many as before: of 512, 32/8 heads 380 / 370, of 768
//            445 / 444, of 1024 511 / 512; 32/4 heads, of 1024 1009 / 977, of 1536 1284 / 1268, 40 of 100 to 1500 1489 / 1506.
static bool single_pass_pays(const AttnArgs& a) {
    const long long n_seq = a.BH / a.H, hkv = a.H / a.group, n_sm = sm_count();
    if (a.cu_q) {
        // (nor where sequences are so short that the accumulator's whole tiles are more than twice the rows)
        if (hkv * ((a.total_k + 127) / 128) < 3 * n_sm || n_seq * 128 > a.total_q) return false;
        return a.D == 64 || a.group == 1 || a.total_k >= n_seq * 128 * (a.group <= 4 ? 6 : 12);
    }
    const long long items = n_seq * hkv * ((a.L + 127) / 128), q_tiles = (a.S + 127) / 128;
    const long long tiles = a.causal ? (q_tiles + 1) / 2 : q_tiles, walk = a.group * tiles;
    if (a.D == 128) return (items >= 10 * n_sm && tiles >= 8) || (items >= 6 * n_sm && tiles >= 16) || (items >= 3 * n_sm && tiles >= 32);
    const long long waves = (items + n_sm - 1) / n_sm;
    const long long key_tiles = (a.L + 127) / 128;
    if (key_tiles >= 8 && 7 * waves * a.group * q_tiles < 4 * key_tiles) return true;
    if (5 * items > 9 * n_sm) return walk >= (items >= 3 * n_sm ? 2 : 6);
    if (a.causal) return 5 * items >= 7 * n_sm && q_tiles >= 48;
    return 5 * items >= 4 * waves * n_sm && waves * walk >= 16;
}

// A caller that has not said whether results must repeat gets what repeats to the bit for packed batches and at D = 128, and the
// faster one at D = 64; it is its choice to give that up for the time (tt_attn_bwd_set_deterministic(0)).
static bool single_pass_allowed(const AttnArgs& a) {
    const int det = g_bwd_deterministic.load();
    return det == 0 || (det < 0 && a.D == 64 && a.cu_q == nullptr);
}

// dk, dv over k, v: the single pass reads a key tile once, ahead of writing its gradients; the dQ pass reads k and v behind them.
// At D = 64, where one pass used to be taken at every size, such calls keep it.
static bool writes_over_keys(const AttnArgs& a) {
    const uintptr_t bytes = (uintptr_t)(a.BH / a.group) * a.L * a.D * sizeof(__nv_bfloat16);
    auto meet = [&](const void* x, const void* y) { return (uintptr_t)x < (uintptr_t)y + bytes && (uintptr_t)y < (uintptr_t)x + bytes; };
    return meet(a.dk, a.k) || meet(a.dk, a.v) || meet(a.dv, a.k) || meet(a.dv, a.v);
}

bool attn_bwd_single_pass(const AttnArgs& a) {
    // TT_BWD_PATH=two_pass|fused overrides the choice (tests run both kernels on the same inputs)
    const char* f = getenv("TT_BWD_PATH");
    bool fused = single_pass_allowed(a) && (single_pass_pays(a) || (a.D == 64 && a.cu_q == nullptr && writes_over_keys(a)));
    if (f && f[0] == 't') fused = false;
    if (f && f[0] == 'f') fused = true;
    return fused && attn_bwd_fused_supported(a);
}

cudaError_t attn_bwd_sm100(const AttnArgs& a, void* ws, size_t ws_bytes, cudaStream_t st) {
    if (attn_bwd_single_pass(a) && ws_bytes >= attn_bwd_fused_workspace(a)) return attn_bwd_fused(a, ws, st);
    return attn_bwd_two_pass(a, ws, st);
}

}  // namespace ttk
