// Device side of the rotation and the QK norm (rope.cu; the decode kernel applies them too, its quantising append included).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "kernels.hpp"

namespace cbkv {

// Two storage-type elements in one 32-bit word, with the non-fusing 2-wide instructions:
// each product and each sum is rounded on its own, never contracted into a multiply-add.
template <bool BF16> struct Pack;
template <> struct Pack<false> {
    using V2 = __half2;
    static __device__ __forceinline__ float2 up(uint32_t v) { return __half22float2(*reinterpret_cast<__half2*>(&v)); }
    static __device__ __forceinline__ float rt(float f) { return __half2float(__float2half_rn(f)); }
    static __device__ __forceinline__ uint32_t down(float a, float b) {
        __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<uint32_t*>(&h);
    }
};
template <> struct Pack<true> {
    using V2 = __nv_bfloat162;
    static __device__ __forceinline__ float2 up(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v)); }
    static __device__ __forceinline__ float rt(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }
    static __device__ __forceinline__ uint32_t down(float a, float b) {
        __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t*>(&h);
    }
};

// rope.rs:196-201 on two (i, i+half) pairs: out[i] = x1*cos + (-x2)*sin, out[i+half] = x2*cos + x1*sin.
template <bool BF16>
__device__ __forceinline__ void rotate2(uint32_t& x1, uint32_t& x2, uint32_t c, uint32_t s) {
    using V2 = typename Pack<BF16>::V2;
    const V2 a = *reinterpret_cast<V2*>(&x1), b = *reinterpret_cast<V2*>(&x2);
    const V2 cc = *reinterpret_cast<V2*>(&c), ss = *reinterpret_cast<V2*>(&s);
    V2 o1 = __hadd2_rn(__hmul2_rn(a, cc), __hmul2_rn(__hneg2(b), ss));
    V2 o2 = __hadd2_rn(__hmul2_rn(b, cc), __hmul2_rn(a, ss));
    x1 = *reinterpret_cast<uint32_t*>(&o1);
    x2 = *reinterpret_cast<uint32_t*>(&o2);
}

// y = x * inv_rms * w in f32, rounded once (norm.rs:27-28); gemma: w + 1 formed in the storage type.
template <bool BF16>
__device__ __forceinline__ uint32_t norm2(uint32_t x, uint32_t w, float inv_rms, bool gemma) {
    using P = Pack<BF16>;
    const float2 u = P::up(x);
    float2 wf = P::up(w);
    if (gemma) { wf.x = P::rt(__fadd_rn(wf.x, 1.f)); wf.y = P::rt(__fadd_rn(wf.y, 1.f)); }
    return P::down(__fmul_rn(__fmul_rn(u.x, inv_rms), wf.x), __fmul_rn(__fmul_rn(u.y, inv_rms), wf.y));
}

template <bool BF16>
__device__ __forceinline__ float sumsq2(uint32_t x) {
    const float2 u = Pack<BF16>::up(x);
    return __fadd_rn(__fmul_rn(u.x, u.x), __fmul_rn(u.y, u.y));
}

// 1 / rms of a row from the sum of its squares (norm.rs:22-27)
__device__ __forceinline__ float inv_rms_of(float ss, int d, float eps) {
    return __frcp_rn(__fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)d), eps)));
}

}  // namespace cbkv
