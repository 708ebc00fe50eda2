// The exact cut of 32-bit values into three bfloat16 pieces, and what the kernels that multiply in pieces
// (linear_split_f32.cu, attention_split_f32.cu) share: stores to tensor memory, register shares of warpgroups.
#pragma once
#include "tcgen05.cuh"

namespace tc {

template <int R> __device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R> __device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

// Two consecutive values -> their three pieces, packed (the first value in the lower half).  Truncation keeps every
// subtraction exact, and the third piece needs no more than the 8 bits a bfloat16 has.
__device__ __forceinline__ void cut2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    const uint32_t u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
    h = __byte_perm(u0, u1, 0x7632);
    const float r0 = x0 - __uint_as_float(u0 & 0xffff0000u), r1 = x1 - __uint_as_float(u1 & 0xffff0000u);
    const uint32_t v0 = __float_as_uint(r0), v1 = __float_as_uint(r1);
    m = __byte_perm(v0, v1, 0x7632);
    const float s0 = r0 - __uint_as_float(v0 & 0xffff0000u), s1 = r1 - __uint_as_float(v1 & 0xffff0000u);
    l = __byte_perm(__float_as_uint(s0), __float_as_uint(s1), 0x7632);
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

}  // namespace tc
