// Attention over float tensors on the tensor cores (head dims up to 128): forward, dQ, dK and dV.
//
// A float is the exact sum of three bf16 values (8 + 8 + 8 bits of mantissa), so a product of two floats is nine
// bf16 products, of which the six largest are kept: x1y1, x1y2, x2y1, x2y2, x1y3, x3y1.  What is left out is below
// 2^-26 of the product, a quarter of what rounding the product to float loses.  The MMAs add in fp32; because their
// additions may truncate, no sum runs through the tensor core for longer than one tile: the small terms are issued
// before the large ones, and the row threads add each tile's accumulator to their own fp32 registers (rounded to
// nearest).  Six bf16 MMAs per product put the ceiling at a sixth of the bf16 rate, five times what the FMA pipes can do.
//
// One CTA owns 128 resident rows and walks the other side in tiles of 64 rows:
//   mode   resident            streamed (T0, T1)     per tile
//   FWD    R0 = Q              K, V                  S = R0 T0^T, P = softmax(S) (online), acc += P T1
//   DV     R0 = K              Q, dO                 S = R0 T0^T, P = exp(S - lse),        acc += P T1
//   DK     R0 = K, R1 = V      Q, dO                 S, dP = R1 T1^T, dS = P (dP - delta), acc += dS T0
//   DQ     R0 = Q, R1 = dO     K, V                  S, dP = R1 T1^T, dS = P (dP - delta), acc += dS T0
// (DV and DK recompute S once each: with both accumulators and both resident tensors in three parts each, one CTA
// has room for neither the operands in shared memory nor the accumulators in registers.)
//
//   warps 0-3  row threads: thread <-> resident row <-> tensor-memory lane
//   warps 4-7  converters: global fp32 -> three bf16 parts -> shared memory (128-byte swizzle, as TMA would write it)
//   warp  8    MMA issuer
// The streamed tiles are in shared memory; R0, R1 and the bf16 parts of P / dS are A operands in tensor memory: an MMA with
// 64 columns takes 32 cycles that way and 48 with both operands in shared memory (measured; 16 against 40 with 32 columns).
// At head dim 128 DK and DQ keep R0 in shared memory, there is no room for both.
// Parts do what a float does only while nothing overflows: the parts of an infinity sum to NaN, and the part products of two
// factors whose product overflows are infinities of either sign.  A wrong score of -infinity would pass unseen (its P is 0),
// so the operands of the scores are watched for magnitudes above 2^60, below which no score overflows; every other
// infinity or NaN reaches the row's result.  Rows of an item that has met such a magnitude, and rows whose result is not
// finite, are computed again with plain multiply-adds by their thread (f32_plain_row); what the mask hides takes no part there.
// The S accumulator is double buffered and the next tile's S is issued before this tile's P is ready.  At head dim 128
// the streamed tiles have 32 rows: with 64, shared memory holds one tile of each tensor (every tile's load is exposed)
// and the row threads' registers do not hold the accumulator row beside two rows of scores.
#include "common.h"
#include "f32_parts.cuh"
#include "sm100_ptx.cuh"

#include <algorithm>

namespace ttk {
using namespace sm100;

namespace {

enum Mode { FWD = 0, DV, DK, DQ };

struct F32Params {
    const float *q, *k, *v, *dout, *lse, *delta;
    float *out, *lse_out, *dq, *dk, *dv;
    int S, L, D, causal, group, H;
    float scale, scale_log2;
    const int* kv_lens;
    int n_qt, n_kt;              // 128-row tiles per query / key slice
    int q_slices, kv_slices;
    int rank_major;              // items numbered heaviest tile of every slice first (few slices), else slice by slice
    int first_wave;
    unsigned int* status;
};

constexpr float kLarge = 1152921504606846976.f;   // 2^60: 128 products of two values up to it are below 2^128
constexpr int kRows = 128, kThreads = 384;   // warps 9-11 only complete the third warpgroup
// registers per thread after setmaxnreg; the sum draws on what the launch allocated (384 x 168)
constexpr int kRegsRows = 232, kRegsConvert = 168, kRegsIssue = 104;
static_assert(kRegsRows + kRegsConvert + kRegsIssue <= 3 * 168, "register split exceeds the CTA's pool");

template <int DP>
struct F32Cfg {
    static constexpr int kSub = DP / 64;
    static constexpr int kCols = DP == 64 ? 64 : 32;         // rows of a streamed tile
    static constexpr int kResPart = kSub * kRows * 128;      // one bf16 part of a resident tile in shared memory
    static constexpr int kStrPart = kSub * kCols * 128;
    static constexpr int kRes = DP == 64 ? 0 : 3 * kResPart, kStr = 3 * kStrPart;
    static constexpr int kN0 = 3, kN1 = 2;                   // T0(j) is read until tile j is accumulated, T1 only by one product
    static constexpr int kAux = 1024 + 8 * 128 * 4;          // barriers, statistics of the streamed queries
    static constexpr int kSmem = kRes + (kN0 + kN1) * kStr + kAux + 1024;
    // tensor memory: S (two buffers); dP, over which the parts of dS (or P) are written once it has been read; the
    // accumulator; the parts of R1 and of R0 (at head dim 128 there is room for one of the two)
    static constexpr uint32_t kS = 0, kDP = 2 * kCols, kW = kDP, kWPart = kCols / 2, kAcc = DP == 64 ? 224 : 128,
                              kR1 = kAcc + DP, kR0 = DP == 64 ? kR1 + 96 : kR1;
    static_assert(kW + 3 * kWPart <= kAcc && kR0 + 3 * DP / 2 <= 512, "tensor memory");
    static_assert(kSmem <= 227 * 1024, "exceeds the shared memory of one CTA");
};
// ROWS x DP floats from row0 on of a [n_rows, D] matrix, 128 threads, 8 consecutive values per thread and step; what
// lies past n_rows or D reads as zero.
template <int DP, int ROWS>
struct TileRegs {
    static constexpr int kSteps = ROWS * (DP / 8) / 128;
    float x[kSteps][8];
    __device__ __forceinline__ void load(const float* src, int row0, int n_rows, int D, int tid) {
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
            const int idx = i * 128 + tid, r = idx / (DP / 8), c = (idx % (DP / 8)) * 8;
            const float* g = src + (long long)(row0 + r) * D + c;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (row0 + r < n_rows && c + 4 * h < D) v = __ldg(reinterpret_cast<const float4*>(g) + h);
                x[i][4 * h] = v.x; x[i][4 * h + 1] = v.y; x[i][4 * h + 2] = v.z; x[i][4 * h + 3] = v.w;
            }
        }
    }
    // part p of the tile at dst + p * part bytes; row r of 64-column block s at s * ROWS * 128 + r * 128, 16-byte chunks
    // swizzled.  Eight neighbouring threads write one 128-byte row: no bank conflicts.
    // Returns the largest magnitude.
    __device__ __forceinline__ float store(unsigned char* dst, int tid) const {
        constexpr int kPart = (DP / 64) * ROWS * 128;
        float top = 0.f;
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
            const int idx = i * 128 + tid, r = idx / (DP / 8), c = idx % (DP / 8);
            unsigned char* p = dst + (c >> 3) * (ROWS * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4);
            uint4 h, m, l;
            split8(x[i], h, m, l);
            *reinterpret_cast<uint4*>(p) = h;
            *reinterpret_cast<uint4*>(p + kPart) = m;
            *reinterpret_cast<uint4*>(p + 2 * kPart) = l;
#pragma unroll
            for (int e = 0; e < 8; e += 2) top = fmax3(top, fabsf(x[i][e]), fabsf(x[i][e + 1]));
        }
        return top;
    }
};

// One work item of one mode.
struct F32Item {
    int slice, r0;          // resident slice and first row
    int Lv;                 // keys that count
    int t_begin, nt;        // streamed tiles per streamed slice
    int n_it;               // nt x streamed slices
};
template <int MODE, int kCols>
__device__ __forceinline__ F32Item f32_item(int idx, const F32Params& p) {
    constexpr bool kKeys = MODE == DV || MODE == DK;   // resident rows are keys
    F32Item w;
    const int n_tiles = kKeys ? p.n_kt : p.n_qt, n_slices = kKeys ? p.kv_slices : p.q_slices;
    const int rank = p.rank_major ? idx / n_slices : idx % n_tiles;
    w.slice = p.rank_major ? idx % n_slices : idx / n_tiles;
    // under the causal mask early key tiles and late query tiles are the heavy ones
    const int tile = kKeys ? rank : n_tiles - 1 - rank;
    w.r0 = tile * kRows;
    w.Lv = valid_keys(p.kv_lens, kKeys ? (long long)w.slice * p.group / p.H : w.slice / p.H, p.L);
    const int off = p.L - p.S;
    if (kKeys) {
        const int first = p.causal ? max(0, w.r0 - off) : 0;   // first query that sees the tile's first key
        w.t_begin = min(first, p.S - 1) / kCols;
        w.nt = w.r0 >= w.Lv ? 0 : (p.S + kCols - 1) / kCols - w.t_begin;
        w.n_it = w.nt * p.group;
    } else {
        const int last = min(w.r0 + kRows, p.S) - 1;
        const int end = p.causal ? min(w.Lv, last + off + 1) : w.Lv;
        w.t_begin = 0;
        w.nt = (end + kCols - 1) / kCols;
        w.n_it = w.nt;
    }
    return w;
}

struct F32Shared {
    unsigned char *res, *t0, *t1;     // resident R0, rings of streamed tiles
    uint64_t *r0_full, *r1_full, *t0_full, *t0_empty, *t1_full, *t1_empty, *s_full, *s_free, *dp_full, *w_full, *acc_full;
    volatile int* large;              // a magnitude above kLarge in R0 or T0
    float* stat;                      // DV, DK: [8 x 128]: -lse, then -delta, of the streamed rows
    uint32_t tmem;
};

// ---------------------------------------------------------------------------- converters (128 threads)
template <int DP, int MODE>
__device__ __forceinline__ void f32_convert(const F32Params& p, const F32Item& w, const F32Shared& sh, const WaitCtx& ctx, int tid) {
    using Cfg = F32Cfg<DP>;
    constexpr int kCols = Cfg::kCols;
    constexpr bool kKeys = MODE == DV || MODE == DK;
    const int n_rows = kKeys ? p.S : w.Lv;            // streamed rows that count
    auto stream_row = [&](int u, int& slice) {
        const int hh = kKeys ? u / w.nt : 0;
        slice = kKeys ? w.slice * p.group + hh : w.slice / p.group;
        return (w.t_begin + u - hh * w.nt) * kCols;
    };
    TileRegs<DP, kCols> a, b;
    float stat_a = 0.f;
    auto load_a = [&](int u) {
        int slice;
        const int row = stream_row(u, slice);
        a.load((kKeys ? p.q : p.k) + (long long)slice * (kKeys ? p.S : p.L) * p.D, row, n_rows, p.D, tid);
        if (kKeys && tid < 2 * kCols) {   // first kCols threads: -lse, -inf (P = 0) past the end; the others: -delta
            const int r = row + tid % kCols;
            const bool ok = r < p.S;
            if (tid < kCols) stat_a = ok ? -p.lse[(long long)slice * p.S + r] : -INFINITY;
            else stat_a = (ok && MODE == DK) ? -p.delta[(long long)slice * p.S + r] : 0.f;
        }
    };
    auto load_b = [&](int u) {
        int slice;
        const int row = stream_row(u, slice);
        b.load((kKeys ? p.dout : p.v) + (long long)slice * (kKeys ? p.S : p.L) * p.D, row, n_rows, p.D, tid);
    };
    if (w.n_it > 0) {
        load_a(0);
        load_b(0);
    }
    float top = 0.f;
    for (int u = 0; u < w.n_it; ++u) {
        const int s0 = u % Cfg::kN0, s1 = u % Cfg::kN1;
        mbar_wait(&sh.t0_empty[s0], ((u / Cfg::kN0) & 1) ^ 1, ctx, 10 + s0, u);
        top = fmaxf(top, a.store(sh.t0 + s0 * Cfg::kStr, tid));
        if (kKeys && tid < 2 * kCols) sh.stat[(u & 7) * 128 + tid] = stat_a;   // row threads lag by at most five tiles
        fence_proxy_async_smem();
        mbar_arrive(&sh.t0_full[s0]);
        if (u + 1 < w.n_it) load_a(u + 1);
        mbar_wait(&sh.t1_empty[s1], ((u / Cfg::kN1) & 1) ^ 1, ctx, 15 + s1, u);
        b.store(sh.t1 + s1 * Cfg::kStr, tid);
        fence_proxy_async_smem();
        mbar_arrive(&sh.t1_full[s1]);
        if (u + 1 < w.n_it) load_b(u + 1);
    }
    if (top > kLarge) *sh.large = 1;
    __syncwarp();
    asm volatile("bar.arrive 1, 256;" ::: "memory");   // with the row threads, for `large`
}

// ---------------------------------------------------------------------------- MMA issuer (one warp)
template <int DP, int MODE>
__device__ __forceinline__ void f32_issue(const F32Item& w, const F32Shared& sh, const WaitCtx& ctx) {
    using Cfg = F32Cfg<DP>;
    constexpr int kCols = Cfg::kCols;
    constexpr bool kHasDP = MODE == DK || MODE == DQ;
    constexpr uint32_t idesc_s = umma_idesc_bf16(kRows, kCols, false, false);
    constexpr uint32_t idesc_acc = umma_idesc_bf16(kRows, DP, false, true);
    const uint32_t tm = __shfl_sync(0xffffffffu, sh.tmem, 0);
    constexpr bool kR0Tmem = DP == 64 || !kHasDP;
    constexpr uint32_t hi = umma_desc_hi(1024);
    const uint32_t res_lo = umma_desc_lo(__shfl_sync(0xffffffffu, smem_u32(sh.res), 0), 16);
    const uint32_t t0a = __shfl_sync(0xffffffffu, smem_u32(sh.t0), 0), t1a = __shfl_sync(0xffffffffu, smem_u32(sh.t1), 0);
    // Each batch is issued by one elected thread.  (An election and a 64-bit descriptor addition per MMA took about 60 cycles
    // an MMA, twice what the tensor core needs for it: 4265 cycles per tile pair of the forward.)
    auto issue_s = [&](int u, uint32_t col) {
        const uint32_t b0 = umma_desc_lo(t0a + (u % Cfg::kN0) * Cfg::kStr, 16);
        if (elect_one()) {
#pragma unroll
            for (int t = 0; t < 6; ++t)
#pragma unroll
                for (int kk = 0; kk < DP / 16; ++kk) {
                    const uint32_t b = b0 + ((term_b(t) * Cfg::kStrPart + (kk >> 2) * (kCols * 128) + (kk & 3) * 32) >> 4);
                    const uint32_t acc = (t > 0 || kk > 0) ? 1u : 0u;
                    if (kR0Tmem) umma_ts_one(tm + col, tm + Cfg::kR0 + term_a(t) * (DP / 2) + kk * 8, b, hi, idesc_s, acc);
                    else umma_ss_one(tm + col, res_lo + ((term_a(t) * Cfg::kResPart + (kk >> 2) * (kRows * 128) + (kk & 3) * 32) >> 4), b, hi, idesc_s, acc);
                }
        }
        __syncwarp();
    };
    auto issue_dp = [&](int u) {
        const uint32_t b0 = umma_desc_lo(t1a + (u % Cfg::kN1) * Cfg::kStr, 16);
        if (elect_one()) {
#pragma unroll
            for (int t = 0; t < 6; ++t)
#pragma unroll
                for (int kk = 0; kk < DP / 16; ++kk)
                    umma_ts_one(tm + Cfg::kDP, tm + Cfg::kR1 + term_a(t) * (DP / 2) + kk * 8,
                                b0 + ((term_b(t) * Cfg::kStrPart + (kk >> 2) * (kCols * 128) + (kk & 3) * 32) >> 4), hi, idesc_s,
                                (t > 0 || kk > 0) ? 1u : 0u);
        }
        __syncwarp();
    };
    auto issue_acc = [&](int u) {
        const uint32_t b0 = umma_desc_lo(kHasDP ? t0a + (u % Cfg::kN0) * Cfg::kStr : t1a + (u % Cfg::kN1) * Cfg::kStr, kCols * 128);
        if (elect_one()) {
#pragma unroll
            for (int t = 0; t < 6; ++t)
#pragma unroll
                for (int kk = 0; kk < kCols / 16; ++kk)
                    umma_ts_one(tm + Cfg::kAcc, tm + Cfg::kW + term_a(t) * Cfg::kWPart + kk * 8,
                                b0 + ((term_b(t) * Cfg::kStrPart + kk * 2048) >> 4), hi, idesc_acc, (t > 0 || kk > 0) ? 1u : 0u);
        }
        __syncwarp();
    };
    auto wait = [&](uint64_t* bar, uint32_t ph, int id, int it) {
        mbar_wait(bar, ph, ctx, id, it);
        __syncwarp();
        tc_fence_after();
    };
    if (w.n_it <= 0) return;
    auto start_s = [&](int u) {
        const int b = u & 1;
        wait(&sh.t0_full[u % Cfg::kN0], (u / Cfg::kN0) & 1, 20, u);
        if (u >= 2) wait(&sh.s_free[b], ((u >> 1) & 1) ^ 1, 22, u);   // S(u - 2) is in registers
        issue_s(u, Cfg::kS + (uint32_t)b * kCols);
        tc_commit(&sh.s_full[b]);
        if (!kHasDP) tc_commit(&sh.t0_empty[u % Cfg::kN0]);
    };
    auto start_dp = [&](int u) {
        wait(&sh.t1_full[u % Cfg::kN1], (u / Cfg::kN1) & 1, 24, u);
        issue_dp(u);
        tc_commit(sh.dp_full);
        tc_commit(&sh.t1_empty[u % Cfg::kN1]);
    };
    wait(sh.r0_full, 0, 26, 0);
    start_s(0);
    if (kHasDP) {
        wait(sh.r1_full, 0, 27, 0);
        start_dp(0);
    }
    for (int u = 0; u < w.n_it; ++u) {
        const bool more = u + 1 < w.n_it;
        if (more) start_s(u + 1);
        if (!kHasDP) wait(&sh.t1_full[u % Cfg::kN1], (u / Cfg::kN1) & 1, 25, u);
        wait(sh.w_full, u & 1, 28, u);
        issue_acc(u);
        tc_commit(sh.acc_full);
        tc_commit(kHasDP ? &sh.t0_empty[u % Cfg::kN0] : &sh.t1_empty[u % Cfg::kN1]);
        if (kHasDP && more) start_dp(u + 1);
    }
}

// ---------------------------------------------------------------------------- row threads
// This thread's values of P or dS -> their three bf16 parts in tensor memory.
template <int DP, int N>
__device__ __forceinline__ void store_parts(uint32_t taddr, const float (&x)[N]) {
    constexpr uint32_t kPart = F32Cfg<DP>::kWPart;
#pragma unroll
    for (int g = 0; g < N / 32; ++g) {
        uint32_t h[16], m[16], l[16];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] = x[g * 32 + i * 8 + e];
            uint4 a, b, c;
            split8(y, a, b, c);
            h[4 * i] = a.x; h[4 * i + 1] = a.y; h[4 * i + 2] = a.z; h[4 * i + 3] = a.w;
            m[4 * i] = b.x; m[4 * i + 1] = b.y; m[4 * i + 2] = b.z; m[4 * i + 3] = b.w;
            l[4 * i] = c.x; l[4 * i + 1] = c.y; l[4 * i + 2] = c.z; l[4 * i + 3] = c.w;
        }
        tmem_st16(taddr + g * 16, h);
        tmem_st16(taddr + kPart + g * 16, m);
        tmem_st16(taddr + 2 * kPart + g * 16, l);
    }
}
template <int N>
__device__ __forceinline__ void load_cols(uint32_t taddr, float (&x)[N]) {
    uint32_t a[N / 32][32];
#pragma unroll
    for (int g = 0; g < N / 32; ++g) tmem_ld32(taddr + g * 32, a[g]);
    tmem_wait_ld();
#pragma unroll
    for (int e = 0; e < N; ++e) x[e] = __uint_as_float(a[e / 32][e % 32]);
}

// One row of DP floats (zero past D, or everywhere if !ok) -> its bf16 parts at `taddr`, DP / 2 columns each.  Returns
// the largest magnitude.
template <int DP>
__device__ __forceinline__ float row_to_tmem(const float* src, bool ok, int D, uint32_t taddr) {
    float top = 0.f;
#pragma unroll 1
    for (int g = 0; g < DP / 32; ++g) {
        uint32_t h[16], m[16], l[16];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float y[8];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int d = g * 32 + i * 8 + e * 4;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (ok && d < D) v = __ldg(reinterpret_cast<const float4*>(src + d));
                y[4 * e] = v.x; y[4 * e + 1] = v.y; y[4 * e + 2] = v.z; y[4 * e + 3] = v.w;
                top = fmax3(fmax3(top, fabsf(v.x), fabsf(v.y)), fabsf(v.z), fabsf(v.w));
            }
            uint4 a, b, c;
            split8(y, a, b, c);
            h[4 * i] = a.x; h[4 * i + 1] = a.y; h[4 * i + 2] = a.z; h[4 * i + 3] = a.w;
            m[4 * i] = b.x; m[4 * i + 1] = b.y; m[4 * i + 2] = b.z; m[4 * i + 3] = b.w;
            l[4 * i] = c.x; l[4 * i + 1] = c.y; l[4 * i + 2] = c.z; l[4 * i + 3] = c.w;
        }
        __syncwarp();
        tmem_st16(taddr + g * 16, h);
        tmem_st16(taddr + DP / 2 + g * 16, m);
        tmem_st16(taddr + DP + g * 16, l);
    }
    tmem_wait_st();
    tc_fence_before();
    return top;
}

// Returns whether the row has to be computed again by plain arithmetic.
template <int DP, int MODE>
__device__ __forceinline__ bool f32_rows(const F32Params& p, const F32Item& w, const F32Shared& sh, const WaitCtx& ctx, int tid) {
    using Cfg = F32Cfg<DP>;
    constexpr int kCols = Cfg::kCols;
    constexpr bool kKeys = MODE == DV || MODE == DK, kHasDP = MODE == DK || MODE == DQ;
    const uint32_t lane_base = sh.tmem + ((uint32_t)(tid & ~31) << 16);
    const int row = w.r0 + tid, off = p.L - p.S;
    const int res_rows = kKeys ? w.Lv : p.S;
    const float c = p.scale_log2;

    // resident tiles: every thread its own row into tensor memory; R0 of DK / DQ at head dim 128 into shared memory
    constexpr bool kR0Tmem = DP == 64 || !kHasDP;
    const long long first = (long long)w.slice * (kKeys ? p.L : p.S) + w.r0;
    float top = 0.f;
    if (kR0Tmem) {
        top = row_to_tmem<DP>((kKeys ? p.k : p.q) + (first + tid) * p.D, row < res_rows, p.D, lane_base + Cfg::kR0);
        mbar_arrive(sh.r0_full);
    } else {
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {   // 64 rows at a time
            TileRegs<DP, 64> r;
            r.load((kKeys ? p.k : p.q) + (long long)w.slice * (kKeys ? p.L : p.S) * p.D, w.r0 + 64 * h, res_rows, p.D, tid);
            // rows 64h.. of a 128-row tile: same swizzle phase (64 is a multiple of 8), sub-blocks 128 rows apart
#pragma unroll
            for (int i = 0; i < TileRegs<DP, 64>::kSteps; ++i) {
                const int idx = i * 128 + tid, rr = idx / (DP / 8) + 64 * h, cc = idx % (DP / 8);
                unsigned char* q = sh.res + (cc >> 3) * (kRows * 128) + rr * 128 + (((cc & 7) ^ (rr & 7)) << 4);
                uint4 a, b, d;
                split8(r.x[i], a, b, d);
                *reinterpret_cast<uint4*>(q) = a;
                *reinterpret_cast<uint4*>(q + Cfg::kResPart) = b;
                *reinterpret_cast<uint4*>(q + 2 * Cfg::kResPart) = d;
#pragma unroll
                for (int e = 0; e < 8; e += 2) top = fmax3(top, fabsf(r.x[i][e]), fabsf(r.x[i][e + 1]));
            }
        }
        fence_proxy_async_smem();
        mbar_arrive(sh.r0_full);
    }
    if (kHasDP) {
        row_to_tmem<DP>((kKeys ? p.v : p.dout) + (first + tid) * p.D, row < res_rows, p.D, lane_base + Cfg::kR1);
        mbar_arrive(sh.r1_full);
    }
    if (top > kLarge) *sh.large = 1;
    uint64_t row_nlse = pack_f32x2(-INFINITY, -INFINITY), row_ndelta = 0;
    if (MODE == DQ && row < p.S) {
        const float nl = -p.lse[(long long)w.slice * p.S + row], nd = -p.delta[(long long)w.slice * p.S + row];
        row_nlse = pack_f32x2(nl, nl);
        row_ndelta = pack_f32x2(nd, nd);
    }

    float acc[DP];
#pragma unroll
    for (int d = 0; d < DP; ++d) acc[d] = 0.f;
    float m = -INFINITY, l = 0.f;
    auto wait_acc = [&](int u) {   // tile u is accumulated; its P / dS parts have been read
        mbar_wait(sh.acc_full, u & 1, ctx, 30, u);
        __syncwarp();
        tc_fence_after();
    };
    auto take_acc = [&](float mul) {   // acc = (acc + the tile's accumulator) * mul
#pragma unroll
        for (int g = 0; g < DP / 32; ++g) {
            uint32_t t[32];
            tmem_ld32(lane_base + Cfg::kAcc + g * 32, t);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 32; ++e) acc[g * 32 + e] = (acc[g * 32 + e] + __uint_as_float(t[e])) * mul;
        }
    };
    for (int u = 0; u < w.n_it; ++u) {
        const int b = u & 1;
        const int col0 = (w.t_begin + (kKeys ? u % w.nt : u)) * kCols;
        mbar_wait(&sh.s_full[b], (u >> 1) & 1, ctx, 32 + b, u);
        __syncwarp();
        tc_fence_after();
        float s[kCols];
        load_cols(lane_base + Cfg::kS + (uint32_t)b * kCols, s);
        tc_fence_before();
        mbar_arrive(&sh.s_free[b]);
        // visible columns [lo, hi) of this row
        int lo = 0, hi = kCols;
        if (kKeys) {
            if (p.causal) lo = row - off - col0;
        } else {
            hi = w.Lv - col0;
            if (p.causal) hi = min(hi, row + off + 1 - col0);
        }
        float corr = 1.f;
        if (MODE == FWD) {
            if (hi < kCols) {
#pragma unroll
                for (int e = 0; e < kCols; ++e) s[e] = e < hi ? s[e] : -INFINITY;
            }
            float x0 = m, x1 = s[0];
#pragma unroll
            for (int e = 0; e < kCols; e += 4) {
                x0 = fmax3(x0, s[e], s[e + 1]);
                x1 = fmax3(x1, s[e + 2], s[e + 3]);
            }
            const float m_new = fmaxf(x0, x1);   // raw scores: the scale is positive
            // exponents as (s - m) * c: the difference of two close floats is exact, where s * c - m * c would carry the
            // rounding of m * c into every probability
            const float mm = m_new == -INFINITY ? 0.f : m_new;   // nothing visible so far: P = exp2(-inf) = 0
            corr = ex2_approx((m - mm) * c);
            m = m_new;
            const uint64_t nm2 = pack_f32x2(-mm, -mm), c2 = pack_f32x2(c, c);
            uint64_t l0 = 0, l1 = 0;
#pragma unroll
            for (int e = 0; e < kCols; e += 4) {
                float y0, y1, y2, y3;
                unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(s[e], s[e + 1]), nm2), c2), y0, y1);
                unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(s[e + 2], s[e + 3]), nm2), c2), y2, y3);
                s[e] = ex2_approx(y0); s[e + 1] = ex2_approx(y1); s[e + 2] = ex2_approx(y2); s[e + 3] = ex2_approx(y3);
                l0 = add_f32x2(l0, pack_f32x2(s[e], s[e + 1]));
                l1 = add_f32x2(l1, pack_f32x2(s[e + 2], s[e + 3]));
            }
            float a0, a1;
            unpack_f32x2(add_f32x2(l0, l1), a0, a1);
            l = fmaf(l, corr, a0 + a1);
        } else {
            const float* st = sh.stat + (u & 7) * 128;
            const uint64_t sc2 = pack_f32x2(p.scale, p.scale), e2 = pack_f32x2(1.4426950408889634f, 1.4426950408889634f);
#pragma unroll
            for (int e = 0; e < kCols; e += 4) {
                ulonglong2 nl = make_ulonglong2(row_nlse, row_nlse);
                if (kKeys) nl = *reinterpret_cast<const ulonglong2*>(st + e);
                float y0, y1, y2, y3;
                unpack_f32x2(mul_f32x2(fma_f32x2(pack_f32x2(s[e], s[e + 1]), sc2, nl.x), e2), y0, y1);
                unpack_f32x2(mul_f32x2(fma_f32x2(pack_f32x2(s[e + 2], s[e + 3]), sc2, nl.y), e2), y2, y3);
                s[e] = ex2_approx(y0); s[e + 1] = ex2_approx(y1); s[e + 2] = ex2_approx(y2); s[e + 3] = ex2_approx(y3);
            }
            if (lo > 0 || hi < kCols) {
#pragma unroll
                for (int e = 0; e < kCols; ++e) s[e] = (e >= lo && e < hi) ? s[e] : 0.f;
            }
            if (kHasDP) {
                mbar_wait(sh.dp_full, u & 1, ctx, 35, u);
                __syncwarp();
                tc_fence_after();
                float dp[kCols];
                load_cols(lane_base + Cfg::kDP, dp);
                tc_fence_before();
#pragma unroll
                for (int e = 0; e < kCols; e += 4) {
                    ulonglong2 nd = make_ulonglong2(row_ndelta, row_ndelta);
                    if (kKeys) nd = *reinterpret_cast<const ulonglong2*>(st + kCols + e);
                    unpack_f32x2(mul_f32x2(pack_f32x2(s[e], s[e + 1]), add_f32x2(pack_f32x2(dp[e], dp[e + 1]), nd.x)), s[e], s[e + 1]);
                    unpack_f32x2(mul_f32x2(pack_f32x2(s[e + 2], s[e + 3]), add_f32x2(pack_f32x2(dp[e + 2], dp[e + 3]), nd.y)), s[e + 2], s[e + 3]);
                }
            }
        }
        __syncwarp();
        if (u > 0) wait_acc(u - 1);
        store_parts<DP>(lane_base + Cfg::kW, s);
        if (u > 0) take_acc(corr);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(sh.w_full);
    }
    if (w.n_it > 0) {
        wait_acc(w.n_it - 1);
        take_acc(1.f);
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");   // with the converters, for `large`
    float zero[4] = {MODE == FWD ? l * 0.f : 0.f, 0.f, 0.f, 0.f};   // NaN where something is not finite
#pragma unroll
    for (int d = 0; d < DP; ++d) zero[d & 3] = fmaf(acc[d], 0.f, zero[d & 3]);
    const bool finite = zero[0] + zero[1] + zero[2] + zero[3] == 0.f;

    const int n_rows = kKeys ? p.L : p.S;
    if (row < n_rows) {
        float mul = MODE == FWD ? 1.f / l : MODE == DV ? 1.f : p.scale;
        float* dst = (MODE == FWD ? p.out : MODE == DV ? p.dv : MODE == DK ? p.dk : p.dq) + ((long long)w.slice * n_rows + row) * p.D;
        const bool dead = kKeys && row >= w.Lv;   // gradients of padded keys are zero
#pragma unroll
        for (int d = 0; d < DP; d += 4)
            if (d < p.D)
                *reinterpret_cast<float4*>(dst + d) = dead ? make_float4(0.f, 0.f, 0.f, 0.f)
                                                           : make_float4(acc[d] * mul, acc[d + 1] * mul, acc[d + 2] * mul, acc[d + 3] * mul);
        if (MODE == FWD && p.lse_out != nullptr) p.lse_out[(long long)w.slice * p.S + row] = fmaf(m, p.scale, logf(l));
    }
    return w.n_it > 0 && row < res_rows && (*sh.large || !finite);
}

template <int DP, int MODE, int ROLE>
__device__ __forceinline__ bool f32_role(int idx, const F32Params& p, const F32Shared& sh, const WaitCtx& ctx) {
    const F32Item w = f32_item<MODE, F32Cfg<DP>::kCols>(idx, p);
    if (ROLE == 0) return f32_rows<DP, MODE>(p, w, sh, ctx, threadIdx.x);
    if (ROLE == 1) f32_convert<DP, MODE>(p, w, sh, ctx, threadIdx.x - 128);
    if (ROLE == 2) f32_issue<DP, MODE>(w, sh, ctx);
    return false;
}
template <int DP, bool kBwd, int ROLE>
__device__ __forceinline__ bool f32_run(const F32Params& p, const F32Shared& sh, const WaitCtx& ctx) {
    const int idx = blockIdx.x;
    if (!kBwd) return f32_role<DP, FWD, ROLE>(idx, p, sh, ctx);
    const int n_k = p.n_kt * p.kv_slices, n_q = p.n_qt * p.q_slices;
    if (idx < n_k) return f32_role<DP, DK, ROLE>(idx, p, sh, ctx);
    if (idx < n_k + n_q) return f32_role<DP, DQ, ROLE>(idx - n_k, p, sh, ctx);
    return f32_role<DP, DV, ROLE>(idx - n_k - n_q, p, sh, ctx);
}

// Row `tid` of this CTA's item with plain multiply-adds over the streamed rows that it sees, written like f32_rows does.  One
// form for all modes, behind everything else of the kernel: inside f32_rows its code alone cost [2,8,2048,64] 10 us of
// 300.  Streamed rows are the same for all lanes; the own rows R0, R1 are in shared memory (what the tiles took), rows
// 16 bytes apart modulo 128.
__device__ __forceinline__ float plain_dot(const float* a, const float* b, int D) {
    float s = 0.f;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
        const float4 x = *reinterpret_cast<const float4*>(a + d), y = __ldg(reinterpret_cast<const float4*>(b + d));
        s = fmaf(x.x, y.x, s); s = fmaf(x.y, y.y, s); s = fmaf(x.z, y.z, s); s = fmaf(x.w, y.w, s);
    }
    return s;
}
template <int DP, bool kBwd>
__device__ __forceinline__ void f32_plain_row(const F32Params& p, unsigned char* smem, int tid) {
    using Cfg = F32Cfg<DP>;
    constexpr int kCols = Cfg::kCols, kPlainPitch = DP + 4, kPlainCols = 32;
    static_assert(2 * kRows * kPlainPitch * 4 <= Cfg::kRes + (Cfg::kN0 + Cfg::kN1) * Cfg::kStr, "own rows take the tiles' place");
    const int n_k = p.n_kt * p.kv_slices, n_q = p.n_qt * p.q_slices, idx = blockIdx.x;
    const int mode = !kBwd ? FWD : idx < n_k ? DK : idx < n_k + n_q ? DQ : DV;
    const bool keys = mode == DK || mode == DV, has_dp = mode == DK || mode == DQ;
    const F32Item w = mode == FWD ? f32_item<FWD, kCols>(idx, p) : mode == DQ ? f32_item<DQ, kCols>(idx - n_k, p)
                                  : f32_item<DK, kCols>(mode == DK ? idx : idx - n_k - n_q, p);
    const int row = w.r0 + tid, off = p.L - p.S, own_rows = keys ? p.L : p.S, rows = keys ? p.S : p.L;
    const int lo = keys && p.causal ? max(0, row - off) : 0;
    const int hi = keys ? p.S : p.causal ? min(w.Lv, row + off + 1) : w.Lv;
    const long long own = (long long)w.slice * own_rows + row;
    const float *src0 = (keys ? p.k : p.q) + own * p.D, *src1 = has_dp ? (keys ? p.v : p.dout) + own * p.D : src0;
    float *r0 = reinterpret_cast<float*>(smem) + tid * kPlainPitch, *r1 = r0 + kRows * kPlainPitch;
    for (int d = 0; d < p.D; ++d) {
        r0[d] = src0[d];
        r1[d] = src1[d];
    }
    float m = -INFINITY;
    if (mode == FWD) {
        const float* t0 = p.k + (long long)(w.slice / p.group) * rows * p.D;
#pragma unroll 1
        for (int c = lo; c < hi; ++c) m = fmaxf(m, plain_dot(r0, t0 + (long long)c * p.D, p.D));
    }
    float* dst = (mode == FWD ? p.out : mode == DV ? p.dv : mode == DK ? p.dk : p.dq) + own * p.D;
#pragma unroll 1
    for (int d0 = 0; d0 < p.D; d0 += kPlainCols) {   // the weights again for each group of columns: no more registers than the rest
        float acc[kPlainCols] = {}, l = 0.f;
#pragma unroll 1
        for (int hh = 0; hh < (keys ? p.group : 1); ++hh) {
            const long long slice = keys ? (long long)w.slice * p.group + hh : w.slice / p.group;
            const float* t0 = (keys ? p.q : p.k) + slice * rows * p.D;
            const float* t1 = (keys ? p.dout : p.v) + slice * rows * p.D;
#pragma unroll 1
            for (int c = lo; c < hi; ++c) {
                const float s = plain_dot(r0, t0 + (long long)c * p.D, p.D);
                const long long q_row = keys ? slice * p.S + c : own;
                float x = mode == FWD ? expf((s - m) * p.scale) : expf(fmaf(s, p.scale, -p.lse[q_row]));
                l += x;
                if (has_dp) x *= plain_dot(r1, t1 + (long long)c * p.D, p.D) - p.delta[q_row];
                const float* t = (has_dp ? t0 : t1) + (long long)c * p.D + d0;
#pragma unroll
                for (int d = 0; d < kPlainCols; d += 4)
                    if (d0 + d < p.D) {
                        const float4 y = __ldg(reinterpret_cast<const float4*>(t + d));
                        acc[d] = fmaf(x, y.x, acc[d]); acc[d + 1] = fmaf(x, y.y, acc[d + 1]);
                        acc[d + 2] = fmaf(x, y.z, acc[d + 2]); acc[d + 3] = fmaf(x, y.w, acc[d + 3]);
                    }
            }
        }
        const float mul = mode == FWD ? 1.f / l : mode == DV ? 1.f : p.scale;
#pragma unroll
        for (int d = 0; d < kPlainCols; d += 4)
            if (d0 + d < p.D)
                *reinterpret_cast<float4*>(dst + d0 + d) = make_float4(acc[d] * mul, acc[d + 1] * mul, acc[d + 2] * mul, acc[d + 3] * mul);
        if (mode == FWD && d0 == 0 && p.lse_out != nullptr) p.lse_out[own] = fmaf(m, p.scale, logf(l));
    }
}

// kBwd: one launch holds the items of DK, DQ and DV one after the other.
template <int DP, bool kBwd>
__global__ void __launch_bounds__(kThreads, 1) attn_f32_sm100_kernel(const F32Params p) {
    using Cfg = F32Cfg<DP>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* aux = smem + Cfg::kRes + (Cfg::kN0 + Cfg::kN1) * Cfg::kStr;
    uint64_t* bars = reinterpret_cast<uint64_t*>(aux);
    F32Shared sh;
    sh.res = smem;
    sh.t0 = smem + Cfg::kRes;
    sh.t1 = sh.t0 + Cfg::kN0 * Cfg::kStr;
    sh.r0_full = bars;
    sh.r1_full = bars + 1;
    sh.dp_full = bars + 2;
    sh.w_full = bars + 3;
    sh.acc_full = bars + 4;
    sh.s_full = bars + 5;     // [2]
    sh.s_free = bars + 7;     // [2]
    sh.t0_full = bars + 9;    // [3]
    sh.t0_empty = bars + 12;  // [3]
    sh.t1_full = bars + 15;   // [2]
    sh.t1_empty = bars + 17;  // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint64_t* bar_next = bars + 24;   // for a CTA that has given up only: a CTA has one item
    uint4* response = reinterpret_cast<uint4*>(bars + 26);
    sh.large = abort_flag + 1;
    sh.stat = reinterpret_cast<float*>(aux + 1024);
    const int warp = uniform_warp_idx();
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        *sh.large = 0;
        mbar_init(bar_next, 1);
        for (int i = 0; i < 19; ++i) {
            const bool rows_or_converters = i == 0 || i == 1 || i == 3 || i == 7 || i == 8 || (i >= 9 && i < 12) || i == 15 || i == 16;
            mbar_init(&bars[i], rows_or_converters ? 128 : 1);
        }
        fence_barrier_init();
    }
    if (warp == 8) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    sh.tmem = *tmem_slot;
    WaitCtx ctx{p.status, abort_flag, warp};
    grid_let_next_start();
    grid_wait_for_previous();
    bool again = false;
    if (warp < 4) {
        setmaxnreg_inc<kRegsRows>();
        again = f32_run<DP, kBwd, 0>(p, sh, ctx);
    } else if (warp < 8) {
        setmaxnreg_dec<kRegsConvert>();   // (what the launch gave)
        f32_run<DP, kBwd, 1>(p, sh, ctx);
    } else {
        setmaxnreg_dec<kRegsIssue>();
        if (warp == 8) f32_run<DP, kBwd, 2>(p, sh, ctx);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(sh.tmem, 512);
        if (*abort_flag) {
            ItemStream rest{bar_next, response, (int)gridDim.x > p.first_wave};
            rest.drop_rest(ctx.budget);
        }
    }
    if (again && !*abort_flag) f32_plain_row<DP, kBwd>(p, smem, threadIdx.x);
}

// delta = rowsum(dO * O): 8 lanes share a row, four rows per warp and step; HBM-bound.
__global__ void __launch_bounds__(256) attn_f32_delta_kernel(const float* __restrict__ out, const float* __restrict__ dout,
                                                            float* __restrict__ delta, long long n_rows, int D) {
    grid_let_next_start();
    grid_wait_for_previous();
    const long long row = ((long long)blockIdx.x * 256 + threadIdx.x) >> 3;
    const int li = threadIdx.x & 7;
    float s = 0.f;
    if (row < n_rows) {
#pragma unroll 4
        for (int d = li * 4; d < D; d += 32) {
            const float4 x = __ldg(reinterpret_cast<const float4*>(out + row * D + d));
            const float4 y = __ldg(reinterpret_cast<const float4*>(dout + row * D + d));
            s = fmaf(x.x, y.x, s); s = fmaf(x.y, y.y, s); s = fmaf(x.z, y.z, s); s = fmaf(x.w, y.w, s);
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (li == 0 && row < n_rows) delta[row] = s;
}

F32Params f32_params(const AttnArgs& a) {
    F32Params p = {};
    p.q = (const float*)a.q; p.k = (const float*)a.k; p.v = (const float*)a.v; p.dout = (const float*)a.dout;
    p.out = (float*)a.out; p.dq = (float*)a.dq; p.dk = (float*)a.dk; p.dv = (float*)a.dv;
    p.S = a.S; p.L = a.L; p.D = a.D; p.causal = a.causal; p.group = a.group; p.H = a.H;
    p.scale = a.scale;
    p.scale_log2 = (float)((double)a.scale * 1.4426950408889634);
    p.kv_lens = a.kv_lens;
    p.n_qt = (a.S + kRows - 1) / kRows;
    p.n_kt = (a.L + kRows - 1) / kRows;
    p.q_slices = (int)a.BH;
    p.kv_slices = (int)(a.BH / a.group);
    p.first_wave = sm_count();
    p.status = device_status_word();
    // Few slices: the heaviest tiles of all slices first, so that the launch ends on light ones.  Many: slice by slice,
    // so that what runs at the same time shares a slice's tensors in L2 (the tail is then short beside the launch).
    p.rank_major = a.BH <= 2 * p.first_wave ? 1 : 0;
    return p;
}

template <int DP, bool kBwd>
cudaError_t f32_launch(const F32Params& p, long long items, cudaStream_t st) {
    const cudaError_t e = TT_ALLOW_SMEM((attn_f32_sm100_kernel<DP, kBwd>), F32Cfg<DP>::kSmem);
    if (e != cudaSuccess) return e;
    LaunchScope ls(kBwd ? K_BWD_F32 : K_FWD_F32, st);
    return launch_overlapped(attn_f32_sm100_kernel<DP, kBwd>, (unsigned)items, kThreads, F32Cfg<DP>::kSmem, st, p);
}

}  // namespace

// 16-byte rows of float tensors, head dims up to 128
bool attn_f32_sm100_supported(const AttnArgs& a, bool backward) {
    if (a.bf16 || a.D % 4 != 0 || a.D > 128) return false;
    uintptr_t bits = (uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.out;
    if (backward) bits |= (uintptr_t)a.dout | (uintptr_t)a.dq | (uintptr_t)a.dk | (uintptr_t)a.dv;
    if (bits & 15) return false;
    const long long tiles = a.BH * (long long)((std::max(a.S, a.L) + kRows - 1) / kRows);
    return 3 * tiles < (1LL << 31);
}
cudaError_t attn_fwd_f32_sm100(const AttnArgs& a, cudaStream_t st) {
    F32Params p = f32_params(a);
    p.lse_out = a.lse;
    const long long items = a.BH * p.n_qt;
    return a.D <= 64 ? f32_launch<64, false>(p, items, st) : f32_launch<128, false>(p, items, st);
}
cudaError_t attn_bwd_f32_sm100(const AttnArgs& a, float* delta, cudaStream_t st) {
    const long long n_rows = a.BH * (long long)a.S;
    {
        LaunchScope ls(K_BWD_SIMT_DELTA, st);
        const cudaError_t e = launch_overlapped(attn_f32_delta_kernel, (unsigned)((n_rows + 31) / 32), 256, 0, st, (const float*)a.out,
                                                (const float*)a.dout, delta, n_rows, a.D);
        if (e != cudaSuccess) return e;
    }
    F32Params p = f32_params(a);
    p.lse = a.lse;
    p.delta = delta;
    const long long items = 2LL * p.n_kt * p.kv_slices + (long long)p.n_qt * p.q_slices;
    return a.D <= 64 ? f32_launch<64, true>(p, items, st) : f32_launch<128, true>(p, items, st);
}

}  // namespace ttk
