// Floats as three bf16 parts for the tensor cores, shared by the float attention and the float GEMM kernels.
#pragma once
#include "sm100_ptx.cuh"

namespace ttk {

// x[0..7] -> three 16-byte groups of bf16 whose sum is x, exactly from 2^-110 on (below, the last part falls under bf16's smallest
// subnormal, 2^-133) and for finite x.  The first part saturates: rounding a value next to
// the largest float up to infinity would leave a remainder of infinity, where the sum of the parts is finite.
__device__ __forceinline__ uint32_t pack_bf16x2_sat(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void split8(const float (&x)[8], uint4& h, uint4& m, uint4& l) {
    uint32_t hh[4], mm[4], ll[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a = x[2 * i], b = x[2 * i + 1];
        hh[i] = pack_bf16x2_sat(a, b);
        a -= __uint_as_float(hh[i] << 16);
        b -= __uint_as_float(hh[i] & 0xffff0000u);
        mm[i] = sm100::pack_bf16x2(a, b);
        a -= __uint_as_float(mm[i] << 16);
        b -= __uint_as_float(mm[i] & 0xffff0000u);
        ll[i] = sm100::pack_bf16x2(a, b);
    }
    h = make_uint4(hh[0], hh[1], hh[2], hh[3]);
    m = make_uint4(mm[0], mm[1], mm[2], mm[3]);
    l = make_uint4(ll[0], ll[1], ll[2], ll[3]);
}

// The kept products, smallest first: (part of A, part of B).
__host__ __device__ constexpr uint32_t term_a(int t) { return (0x001102u >> (4 * t)) & 3u; }
__host__ __device__ constexpr uint32_t term_b(int t) { return (0x010120u >> (4 * t)) & 3u; }

}  // namespace ttk
