// The exact cut of 32-bit values into three bfloat16 pieces, and what the kernels that multiply in pieces
// (linear_split_f32.cu, linear_batch_f32.cu, moe_split_f32.cu, attention_split_f32.cu) share: stores to tensor memory, register shares of warpgroups.
#pragma once
#include "tcgen05.cuh"

namespace tc {

template <int R> __device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R> __device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

// Two consecutive values -> their three pieces, packed (the first value in the lower half).  h is x rounded to the nearest
// bfloat16, m the rest rounded likewise, l what then remains.  Every subtraction is exact: with |x| in [2^e, 2^(e+1)) the
// rest after h is a multiple of 2^(e-23) of at most 2^(e-8), the rest after m one of at most 2^(e-17), which needs 7 of the
// 8 bits a bfloat16 has.  Rounding instead of cutting bits off keeps the dropped products of pieces (m l, l m, l l) below
// 2^-24 of the product (6e-8; cut off they reach 2^-21 and all have the product's sign, so that sums shrink by 4e-8), and
// they have either sign (tests/test_product_args.py has both cuts in numpy).  Values beyond the largest bfloat16 round to
// infinity: SPLIT_MAX is the limit that the kernels look for.  Below 2^-110 the last piece runs into the smallest bfloat16,
// 2^-133, and what lies under that is lost.
constexpr float SPLIT_MAX = 3.38953139e38f;

__device__ __forceinline__ uint32_t bf16x2_rn(float x0, float x1) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(x1), "f"(x0));
    return r;
}
__device__ __forceinline__ void cut2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = bf16x2_rn(x0, x1);
    const float r0 = x0 - __uint_as_float(h << 16), r1 = x1 - __uint_as_float(h & 0xffff0000u);
    m = bf16x2_rn(r0, r1);
    l = bf16x2_rn(r0 - __uint_as_float(m << 16), r1 - __uint_as_float(m & 0xffff0000u));
}

// 8 values -> the 16 bytes of each piece
__device__ __forceinline__ void cut8(const float4& x, const float4& y, uint4& h, uint4& m, uint4& l) {
    cut2(x.x, x.y, h.x, m.x, l.x);
    cut2(x.z, x.w, h.y, m.y, l.y);
    cut2(y.x, y.y, h.z, m.z, l.z);
    cut2(y.z, y.w, h.w, m.w, l.w);
}

// 8 columns of this warp's 32 lanes of tensor memory
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint4& a, const uint4& b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w));
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The plain sum of an element whose tensor-core sum is not finite; K a multiple of 4, both 16-byte aligned.
[[maybe_unused]] static __device__ __noinline__ float plain_dot(const float* a, const float* w, int K) {
    float s = 0.f;
    for (int k = 0; k < K && s == s; k += 4) {
        const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
        s = fmaf(x.x, y.x, s);
        s = fmaf(x.y, y.y, s);
        s = fmaf(x.z, y.z, s);
        s = fmaf(x.w, y.w, s);
    }
    return s;
}

}  // namespace tc
