// Row softmax, forward and backward, as HBM-bound kernels.
//
// Semantics of the reference's native SoftmaxForward (src/Layers.cu:324-349 of the reference
// project: softmax over the last axis, leading axes flattened to rows, row maximum subtracted;
// there it is five launches plus two host loops of per-row Thrust reductions) in ONE launch that
// reads every element once and writes it once.  The backward (the reference has none on the
// native side) is dx = y * (dy - sum(dy * y)).
//
// A row of up to 16384 values is held in registers by the smallest group of threads that takes it: 4 to 32 lanes or a
// CTA of 256 threads.  Longer rows are read twice, the second time mostly from L2 (clusters of CTAs that hold such a row
// in registers were slower for bf16: [5592, 24000] backward 612 us, against 137 now and 278 with three scalar passes).
//
// Loads and stores are 16-byte vectors at every pitch: the aligned vectors inside the row, and the fewer than 2 x 16
// bytes before and after them as one value each of the row's first threads.  That needs tensors that start on a
// 16-byte boundary; others take the same kernel with vectors of one value.
// Measured, forward / backward, with values of 2 or 4 bytes per load before: bf16 [131072, 1024] 145 / 182 -> 87 / 115 us (7.0
// TB/s), [130944, 1025] 248 / 184 -> 90 / 115, [10872, 12345] 282 / 260 -> 122 / 176; float [130944, 1025] 227 / 232 -> 157 / 230,
// [2048, 65536] 353 / 433 -> 225 / 382.
#include <type_traits>

#include "common.h"

namespace ttk {

__device__ __forceinline__ float sm_ld(const float* p) { return *p; }
__device__ __forceinline__ float sm_ld(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void sm_st(float* p, float v) { *p = v; }
__device__ __forceinline__ void sm_st(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// A vector as it is loaded: 16 bytes, or one value.  Unpacked only where it is used, so that loads are not separated by
// conversions and bf16 values wait in half the registers.
template <typename T, int kV> using Raw = std::conditional_t<kV == 1, T, uint4>;
__device__ __forceinline__ void unpack(float r, float (&x)[1]) { x[0] = r; }
__device__ __forceinline__ void unpack(__nv_bfloat16 r, float (&x)[1]) { x[0] = __bfloat162float(r); }
__device__ __forceinline__ void unpack(const uint4& r, float (&x)[4]) {
    x[0] = __uint_as_float(r.x); x[1] = __uint_as_float(r.y); x[2] = __uint_as_float(r.z); x[3] = __uint_as_float(r.w);
}
__device__ __forceinline__ void unpack(const uint4& r, float (&x)[8]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[2 * i] = __uint_as_float(w[i] << 16);
        x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ void sm_stv(float* p, const float (&x)[1]) { *p = x[0]; }
__device__ __forceinline__ void sm_stv(__nv_bfloat16* p, const float (&x)[1]) { sm_st(p, x[0]); }
__device__ __forceinline__ void sm_stv(float* p, const float (&x)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}
__device__ __forceinline__ void sm_stv(__nv_bfloat16* p, const float (&x)[8]) {
    __nv_bfloat162 h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<uint4*>(h);
}

// Reduction over the kThreads threads that hold a row: up to 32 neighbouring lanes, or the CTA.  A kernel reduces at most
// twice, `red` [2][kThreads / 32] shared, slot 0 and 1.
template <bool kMax>
__device__ __forceinline__ float sm_op(float a, float b) { return kMax ? fmaxf(a, b) : a + b; }
template <int kThreads, bool kMax>
__device__ __forceinline__ float row_reduce(float x, float* red, int slot) {
#pragma unroll
    for (int o = (kThreads < 32 ? kThreads : 32) / 2; o > 0; o >>= 1) x = sm_op<kMax>(x, __shfl_xor_sync(0xffffffffu, x, o));
    if (kThreads > 32) {
        constexpr int kWarps = kThreads / 32;
        if ((threadIdx.x & 31) == 0) red[slot * kWarps + (threadIdx.x >> 5)] = x;
        __syncthreads();
        x = red[slot * kWarps];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) x = sm_op<kMax>(x, red[slot * kWarps + w]);
    }
    return x;
}

// kBwd = false: out = softmax(a).   kBwd = true: out = a * (b - sum(a*b))  with a = y, b = dy.
// A row belongs to kThreads threads (kThreads <= 32: 256 / kThreads rows per CTA), kPer vectors of kV values each.
// kThreads >= 2 kV wherever a row can start between two vectors.  No branch lies between the loads: with a test of each
// vector for the row's ends they waited for one another (bf16 [131200, 1023] 358 us).
template <typename T, int kV, int kPer, int kThreads, bool kBwd>
__global__ void __launch_bounds__(256) softmax_rows_kernel(const T* a, const T* b, T* out, long long rows, int cols) {
    grid_let_next_start();
    grid_wait_for_previous();
    __shared__ float red[2 * 8];
    const int tid = kThreads > 32 ? (int)threadIdx.x : (int)threadIdx.x % kThreads;
    const long long row = kThreads > 32 ? (long long)blockIdx.x : (long long)blockIdx.x * (256 / kThreads) + threadIdx.x / kThreads;
    const bool live = row < rows;                       // (part of a warp may lie past the last row: it still shuffles)
    const long long base = (live ? row : 0) * cols;
    const int n = live ? cols : 0;
    const int head = min(n, (int)(-base & (kV - 1)));   // values before the first aligned vector
    const int nv = (n - head) / kV;
    const Raw<T, kV>* av = reinterpret_cast<const Raw<T, kV>*>(a + base + head);
    const Raw<T, kV>* bv = kBwd ? reinterpret_cast<const Raw<T, kV>*>(b + base + head) : nullptr;
    // this thread's single value: one of the head (threads 0 .. kV - 1) or of what follows the last vector
    const int at_one = tid < kV ? tid : head + nv * kV + tid - kV;
    const bool one = kV > 1 && (tid < kV ? tid < head : tid < 2 * kV && at_one < n);
    Raw<T, kV> ra[kPer], rb[kBwd ? kPer : 1];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int v = tid + i * kThreads;
        ra[i] = Raw<T, kV>{};
        if (v < nv) ra[i] = av[v];
        if (kBwd) {
            rb[i] = Raw<T, kV>{};
            if (v < nv) rb[i] = bv[v];
        }
    }
    float x1 = kBwd ? 0.f : -INFINITY, y1 = 0.f;
    if (one) {
        x1 = sm_ld(a + base + at_one);
        if (kBwd) y1 = sm_ld(b + base + at_one);
    }
    if (!kBwd) {
        float x[kPer][kV], m = x1;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            unpack(ra[i], x[i]);
#pragma unroll
            for (int e = 0; e < kV; ++e) {
                x[i][e] = tid + i * kThreads < nv ? x[i][e] : -INFINITY;
                m = fmaxf(m, x[i][e]);
            }
        }
        m = row_reduce<kThreads, true>(m, red, 0);
        x1 = __expf(x1 - m);
        float s = x1;
#pragma unroll
        for (int i = 0; i < kPer; ++i)
#pragma unroll
            for (int e = 0; e < kV; ++e) {
                x[i][e] = __expf(x[i][e] - m);
                s += x[i][e];
            }
        s = row_reduce<kThreads, false>(s, red, 1);
        const float inv = 1.0f / s;
        x1 *= inv;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
#pragma unroll
            for (int e = 0; e < kV; ++e) x[i][e] *= inv;
            if (tid + i * kThreads < nv) sm_stv(out + base + head + (tid + i * kThreads) * kV, x[i]);
        }
    } else {
        float d = x1 * y1;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            float x[kV], y[kV];
            unpack(ra[i], x);
            unpack(rb[i], y);
#pragma unroll
            for (int e = 0; e < kV; ++e) d = fmaf(x[e], y[e], d);
        }
        d = row_reduce<kThreads, false>(d, red, 0);
        x1 *= y1 - d;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            float x[kV], y[kV];
            unpack(ra[i], x);
            unpack(rb[i], y);
#pragma unroll
            for (int e = 0; e < kV; ++e) x[e] *= y[e] - d;
            if (tid + i * kThreads < nv) sm_stv(out + base + head + (tid + i * kThreads) * kV, x);
        }
    }
    if (one) sm_st(out + base + at_one, x1);
}

// Longer rows: one CTA of 1024 threads per row, read twice (forward: a running maximum and sum, then the values; backward:
// the product, then the values).  Two CTAs per SM at most, so that the rows in flight still lie in L2 when they are read
// again: 296 rows of 256 KB are 78 MB.
template <typename T, int kV, bool kBwd>
__global__ void __launch_bounds__(1024) softmax_rows_long_kernel(const T* a, const T* b, T* out, int cols) {
    grid_let_next_start();
    grid_wait_for_previous();
    __shared__ float red[2 * 32];
    const int tid = threadIdx.x;
    const long long base = (long long)blockIdx.x * cols;
    const int head = min(cols, (int)(-base & (kV - 1)));
    const int nv = (cols - head) / kV;
    const Raw<T, kV>* av = reinterpret_cast<const Raw<T, kV>*>(a + base + head);
    const Raw<T, kV>* bv = kBwd ? reinterpret_cast<const Raw<T, kV>*>(b + base + head) : nullptr;
    const int at_one = tid < kV ? tid : head + nv * kV + tid - kV;
    const bool one = kV > 1 && (tid < kV ? tid < head : tid < 2 * kV && at_one < cols);
    float x1 = kBwd ? 0.f : -INFINITY, y1 = 0.f;
    if (one) {
        x1 = sm_ld(a + base + at_one);
        if (kBwd) y1 = sm_ld(b + base + at_one);
    }
    if (!kBwd) {
        float m = x1, s = one ? __expf(x1 - x1) : 0.f;   // an infinity or NaN makes the sum NaN, as exp(x - max) does
        if (one && x1 == -INFINITY) s = 0.f;
#pragma unroll 4
        for (int v = tid; v < nv; v += 1024) {
            float x[kV];
            unpack(av[v], x);
            float mv = x[0];
#pragma unroll
            for (int e = 1; e < kV; ++e) mv = fmaxf(mv, x[e]);
            const float m_new = fmaxf(m, mv), ref = m_new == -INFINITY ? 0.f : m_new;   // nothing but -inf so far: sum 0
            s *= __expf(m - ref);
#pragma unroll
            for (int e = 0; e < kV; ++e) s += __expf(x[e] - ref);
            m = m_new;
        }
        const float top = row_reduce<1024, true>(m, red, 0);
        s = row_reduce<1024, false>(m == -INFINITY ? s : s * __expf(m - top), red, 1);
        const float inv = 1.0f / s;
#pragma unroll 4
        for (int v = tid; v < nv; v += 1024) {
            float x[kV];
            unpack(av[v], x);
#pragma unroll
            for (int e = 0; e < kV; ++e) x[e] = __expf(x[e] - top) * inv;
            sm_stv(out + base + head + v * kV, x);
        }
        if (one) sm_st(out + base + at_one, __expf(x1 - top) * inv);
    } else {
        float d = x1 * y1;
#pragma unroll 4
        for (int v = tid; v < nv; v += 1024) {
            float x[kV], y[kV];
            unpack(av[v], x);
            unpack(bv[v], y);
#pragma unroll
            for (int e = 0; e < kV; ++e) d = fmaf(x[e], y[e], d);
        }
        d = row_reduce<1024, false>(d, red, 0);
#pragma unroll 4
        for (int v = tid; v < nv; v += 1024) {
            float x[kV], y[kV];
            unpack(av[v], x);
            unpack(bv[v], y);
#pragma unroll
            for (int e = 0; e < kV; ++e) x[e] *= y[e] - d;
            sm_stv(out + base + head + v * kV, x);
        }
        if (one) sm_st(out + base + at_one, x1 * (y1 - d));
    }
}

template <typename T, int kV, bool kBwd>
static void launch_vectors(const T* a, const T* b, T* out, long long rows, int cols, cudaStream_t st) {
    const int nv = cols / kV;          // vectors inside a row at most
    const int odd = cols % kV != 0;    // rows that start between two vectors: at least 2 kV threads
    auto go = [&](auto per, auto threads) {
        constexpr int P = decltype(per)::value, N = decltype(threads)::value;
        const long long ctas = N > 32 ? rows : (rows + 256 / N - 1) / (256 / N);
        launch_overlapped(softmax_rows_kernel<T, kV, P, N, kBwd>, (unsigned)ctas, 256, 0, st, a, b, out, rows, cols);
    };
#define TT_SM_N(n) std::integral_constant<int, (n)>()
    // A warp takes a row up to 64 values per lane: no barrier, and each lane's loads are many.  (A CTA with a vector or two
    // per thread waits on its two reductions: float [130944, 1025] 225 us.)
    // kV = 1: rows off 16 bytes, and short ones at an odd pitch, a few values per lane.
    if (kV == 1 && nv <= 16) go(TT_SM_N(kV == 1 ? 4 : 1), TT_SM_N(4));
    else if (kV == 1 && nv <= 32) go(TT_SM_N(kV == 1 ? 8 : 1), TT_SM_N(4));
    else if (kV == 1 && nv <= 64) go(TT_SM_N(kV == 1 ? 8 : 1), TT_SM_N(8));
    else if (kV == 1 && nv <= 128) go(TT_SM_N(kV == 1 ? 8 : 1), TT_SM_N(16));
    else if (nv <= 4 && !odd) go(TT_SM_N(1), TT_SM_N(4));
    else if (nv <= 8 && !(odd && kV > 4)) go(TT_SM_N(1), TT_SM_N(8));
    else if (nv <= 16) go(TT_SM_N(1), TT_SM_N(16));
    else if (nv <= 32) go(TT_SM_N(1), TT_SM_N(32));
    else if (nv <= 64) go(TT_SM_N(2), TT_SM_N(32));
    else if (nv <= 128) go(TT_SM_N(4), TT_SM_N(32));
    else if (nv <= 256) go(TT_SM_N(8), TT_SM_N(32));
    else if (kV < 8 && nv <= 512) go(TT_SM_N(kV < 8 ? 16 : 8), TT_SM_N(32));
    else if (kV == 1 && nv <= 1024) go(TT_SM_N(kV == 1 ? 32 : 8), TT_SM_N(32));
    else if (kV > 1 && nv <= 512) go(TT_SM_N(2), TT_SM_N(256));
    else if (kV > 1 && nv <= 1024) go(TT_SM_N(4), TT_SM_N(256));
    else if (nv <= 2048) go(TT_SM_N(8), TT_SM_N(256));
    else if (kV < 8 && nv <= 4096) go(TT_SM_N(kV < 8 ? 16 : 8), TT_SM_N(256));
    else if (kV == 1 && nv <= 8192) go(TT_SM_N(kV == 1 ? 32 : 8), TT_SM_N(256));
    else if (kV == 1 && nv <= 16384) go(TT_SM_N(kV == 1 ? 64 : 8), TT_SM_N(256));
    else launch_overlapped(softmax_rows_long_kernel<T, kV, kBwd>, (unsigned)rows, 1024, 0, st, a, b, out, cols);
#undef TT_SM_N
}
template <typename T, bool kBwd>
static cudaError_t launch_softmax(const void* a, const void* b, void* out, long long rows, int cols, cudaStream_t st) {
    const T* pa = (const T*)a;
    const T* pb = (const T*)b;
    T* po = (T*)out;
    LaunchScope ls(kBwd ? K_SOFTMAX_BWD : K_SOFTMAX_FWD, st);
    const bool aligned = (((uintptr_t)a | (kBwd ? (uintptr_t)b : 0) | (uintptr_t)out) & 15) == 0;
    // Short rows that start between two vectors would be little else than the values around them: bf16 [262144, 13] 31 us on
    // vectors, 33 columns 30 us.
    const bool values = cols % (16 / (int)sizeof(T)) != 0 && cols <= (sizeof(T) == 2 ? 64 : 16);
    if (aligned && !values) launch_vectors<T, 16 / sizeof(T), kBwd>(pa, pb, po, rows, cols, st);
    else launch_vectors<T, 1, kBwd>(pa, pb, po, rows, cols, st);
    return cudaGetLastError();
}

cudaError_t softmax_rows_fwd(const void* in, void* out, long long rows, int cols, int bf16, cudaStream_t st) {
    return bf16 ? launch_softmax<__nv_bfloat16, false>(in, nullptr, out, rows, cols, st)
                : launch_softmax<float, false>(in, nullptr, out, rows, cols, st);
}
cudaError_t softmax_rows_bwd(const void* y, const void* dy, void* dx, long long rows, int cols, int bf16,
                             cudaStream_t st) {
    return bf16 ? launch_softmax<__nv_bfloat16, true>(y, dy, dx, rows, cols, st)
                : launch_softmax<float, true>(y, dy, dx, rows, cols, st);
}

}  // namespace ttk
