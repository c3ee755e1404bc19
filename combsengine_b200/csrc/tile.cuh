// Device helpers of the kernels that stream page tiles through a shared-memory ring and do their math with mma.sync
// (kernels.cu): barriers and copies, one tile against a block of query columns, int8 tiles, norm and rotation on the way.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "kernels.hpp"
#include "q8_unpack.cuh"
#include "rope.cuh"

namespace cbkv {

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
// Non-blocking look at a barrier phase (try_wait may suspend the thread for a while).
__device__ __forceinline__ uint32_t mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
// Bounded wait: gives up after `limit_ns` of wall time and returns false (the caller
// records it in the status word and stops consuming; nothing spins forever).
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, uint64_t limit_ns = 100000000ull) {
    for (int i = 0; i < 64; i++)
        if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > limit_ns) return false;
    return true;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if constexpr (BF16) {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    } else {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
}
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    if constexpr (BF16) {
        __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&v);
    } else {
        __half2 v = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&v);
    }
}
template <bool BF16>
__device__ __forceinline__ uint16_t to_elem(float x) {
    if constexpr (BF16) { __nv_bfloat16 v = __float2bfloat16_rn(x); return *reinterpret_cast<uint16_t*>(&v); }
    else { __half v = __float2half_rn(x); return *reinterpret_cast<uint16_t*>(&v); }
}
template <bool BF16>
__device__ __forceinline__ float from_elem(uint16_t x) {
    if constexpr (BF16) { return __bfloat162float(*reinterpret_cast<__nv_bfloat16*>(&x)); }
    else { return __half2float(*reinterpret_cast<__half*>(&x)); }
}

// Byte offset of (row, 16-byte chunk j) inside one swizzled 32-row x 128-byte block.
__device__ __forceinline__ uint32_t swz(uint32_t row, uint32_t j) { return row * 128u + ((j ^ (row & 7u)) << 4); }

// One 16-token tile against NT blocks of 8 query columns.
//   stage        shared address of the K|V tile ([D/64] blocks of 32 rows x 128 B)
//   qf           Q^T fragments (B operand), loaded once per work item
//   kpos0        absolute position of the tile's first token
//   qpos         absolute query position of this thread's two columns per block
template <int D, int NT, bool BF16>
__device__ __forceinline__ void attend_tile(uint32_t stage, const uint32_t (&qf)[NT][D / 16][2],
                                            float (&o)[NT][D / 16][4], float (&m)[NT][2], float (&l)[NT][2],
                                            int kpos0, const int (&qpos)[NT][2], int window, float scale_log2,
                                            bool need_mask, int lane) {
    const int g = lane >> 2;
    float s[NT][4], s2[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
        s2[nt][0] = s2[nt][1] = s2[nt][2] = s2[nt][3] = 0.f;
    }
    // ---- S^T = K . Q^T  (two accumulator chains, summed at the end)
    {
        const uint32_t row = (lane & 7) + ((lane >> 3) & 1) * 16;  // K slot (lane&7) + 8*((lane>>3)&1) -> its row
        const uint32_t jsel = lane >> 4;                           // which of the two 16-byte chunks
#pragma unroll
        for (int ks = 0; ks < D / 16; ks++) {
            uint32_t a[4];
            ldsm_x4(stage + (ks >> 2) * 4096u + swz(row, (ks & 3) * 2 + jsel), a);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                if (ks & 1) mma_16816<BF16>(s2[nt], a, qf[nt][ks][0], qf[nt][ks][1]);
                else mma_16816<BF16>(s[nt], a, qf[nt][ks][0], qf[nt][ks][1]);
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
#pragma unroll
            for (int i = 0; i < 4; i++) s[nt][i] += s2[nt][i];
        }
    }
    // ---- online softmax over the tile's 16 tokens (rows g and g+8 of the fragment)
    uint32_t pb[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
#pragma unroll
        for (int i = 0; i < 4; i++) s[nt][i] *= scale_log2;
        if (need_mask) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int kp = kpos0 + g + (i >> 1) * 8;
                int qp = qpos[nt][i & 1];
                bool ok = kp <= qp && (window <= 0 || kp + window > qp);  // keys in (p - w, p], kv.rs:252-257
                if (!ok) s[nt][i] = -INFINITY;
            }
        }
        float alpha[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            float mx = fmaxf(s[nt][j], s[nt][j + 2]);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
            float m_new = fmaxf(m[nt][j], mx);
            float m_use = (m_new == -INFINITY) ? 0.f : m_new;
            alpha[j] = exp2f(m[nt][j] - m_use);
            m[nt][j] = m_new;
            float p0 = exp2f(s[nt][j] - m_use);
            float p1 = exp2f(s[nt][j + 2] - m_use);
            s[nt][j] = p0;
            s[nt][j + 2] = p1;
            l[nt][j] = l[nt][j] * alpha[j] + p0 + p1;  // this thread's share; reduced over row groups at the end
        }
#pragma unroll
        for (int mt = 0; mt < D / 16; mt++) {
            o[nt][mt][0] *= alpha[0]; o[nt][mt][1] *= alpha[1];
            o[nt][mt][2] *= alpha[0]; o[nt][mt][3] *= alpha[1];
        }
        // P^T as the B operand: transpose the two 8x8 blocks across the warp
        pb[nt][0] = movmatrix_trans(pack2<BF16>(s[nt][0], s[nt][1]));
        pb[nt][1] = movmatrix_trans(pack2<BF16>(s[nt][2], s[nt][3]));
    }
    // ---- O^T += V^T . P^T   (V slots 0-7 are rows 8-15 of the block, slots 8-15 rows 24-31)
    {
        const uint32_t row = 8 + (lane & 7) + (lane >> 4) * 16;  // V slot (lane&7) + 8*(lane>>4) -> its row
        const uint32_t jsel = (lane >> 3) & 1;                   // d chunk
#pragma unroll
        for (int mt = 0; mt < D / 16; mt++) {
            uint32_t a[4];
            ldsm_x4_trans(stage + (mt >> 2) * 4096u + swz(row, (mt & 3) * 2 + jsel), a);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) mma_16816<BF16>(o[nt][mt], a, pb[nt][0], pb[nt][1]);
        }
    }
}

// ------------------------------------------------------------------ int8 pages (kv.rs:271-358)
// A quantised record (kernels.hpp, qrec_*) reaches shared memory as it lies in HBM, by one TMA box.  Values are
// converted in registers by a byte permute that puts a constant exponent byte over each value byte
// and one exact subtraction (q8_pair).  The group scales never touch the values: K's multiply the f32 score partial sums of their 32-wide group, V's multiply the
// probabilities of their token before the P.V product of that group's rows.
//
// The contraction index of an MMA may be permuted freely if both operands agree, and so may the
// output rows of O^T if the store undoes it; that is how a thread gets whole 4- and 8-byte words:
//   K (A operand, row = token): per group a thread takes bytes 8t..8t+7 of rows g and g+8; k-step s
//     contracts d = 32*grp + 8t + 4s + {0,1,2,3} against the Q fragment loaded in the same order.
//   V (A operand of O^T, row = d): per group a thread takes d = 4g..4g+3 of token pairs (2t, 2t+1)
//     and (2t+8, 2t+9), stored pair-interleaved so that one register is one 16-bit pick; m-tile
//     2*grp has rows d = 32*grp + 4g + {0 (row g), 1 (row g+8)}, m-tile 2*grp+1 the other two.
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.b16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}
// Byte -> number conversions (q8_fix, q8_pair, mul2): q8_unpack.cuh.
template <bool BF16>
__device__ __forceinline__ float2 up2(uint32_t v) {
    if constexpr (BF16) return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v));
    else return __half22float2(*reinterpret_cast<__half2*>(&v));
}
__device__ __forceinline__ float fast_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One 16-token quantised tile against the 8 query columns of the kv group (decode), in two steps:
// q8_load copies this thread's share of the record from shared memory to registers, after which the
// ring stage can go back to the producer; q8_attend does the math from registers.  The running
// maximum of a column moves only when the new one exceeds it by 2^8 (the exponentials stay far inside
// the f16 range), so most tiles skip the rescaling of the output accumulators.
template <int D>
struct Q8Tile {
    static constexpr int G = D / 32;
    uint2 kx[G], ky[G], va[G], vb[G];            // K bytes of rows g, g+8; V bytes of token pairs t, t+4
    uint32_t ks0[G / 2], ks1[G / 2], vs0[G], vs1[G];  // their scales
};

template <int D>
__device__ __forceinline__ void q8_load(uint32_t stage, int lane, Q8Tile<D>& r) {
    constexpr int G = D / 32;
    static_assert(G % 2 == 0, "scales are read two at a time");
    const int g = lane >> 2, t = lane & 3;
    const uint32_t kbase = stage, vbase = stage + 16u * D, ksc = stage + 32u * D, vsc = ksc + 16u * G * 2u;
    const int swz = qrec_swz(g, D);  // rows g and g+8 share it
    const uint32_t r0 = kbase + (uint32_t)g * D + 8u * t, r1 = r0 + 8u * D;
#pragma unroll
    for (int grp = 0; grp < G; grp++) {
        const uint32_t off = (uint32_t)((grp ^ swz) << 5);
        r.kx[grp] = lds64(r0 + off);
        r.ky[grp] = lds64(r1 + off);
    }
#pragma unroll
    for (int i = 0; i < G / 2; i++) {
        r.ks0[i] = lds32(ksc + (uint32_t)(g * G + 2 * i) * 2u);
        r.ks1[i] = lds32(ksc + (uint32_t)((g + 8) * G + 2 * i) * 2u);
    }
    // pair t and pair t+4 share the unit and chunk permutation (qrec_value_off)
    const uint32_t c0 = vbase + (uint32_t)t * 2u * D + (uint32_t)((g ^ (4 * ((t >> 1) & 1))) * 8);
#pragma unroll
    for (int grp = 0; grp < G; grp++) {
        const uint32_t off = (uint32_t)((grp ^ (t & 1)) * 64);
        r.va[grp] = lds64(c0 + off);
        r.vb[grp] = lds64(c0 + 8u * D + off);
        r.vs0[grp] = lds32(vsc + (uint32_t)(grp * 16 + 2 * t) * 2u);
        r.vs1[grp] = lds32(vsc + (uint32_t)(grp * 16 + 2 * t + 8) * 2u);
    }
}

template <int D, bool BF16>
__device__ __forceinline__ void q8_attend(const Q8Tile<D>& r, const uint32_t (&qf)[1][D / 16][2], float (&o)[1][D / 16][4],
                                          float (&m)[1][2], float (&l)[1][2], int kpos0, const int (&qpos)[1][2],
                                          int window, float scale_log2, bool need_mask, int lane, int dbg = 0) {
    (void)dbg;  // phase switches exist in the measurement build only
    constexpr int G = D / 32;
    const int g = lane >> 2;
    const uint2 (&kx)[G] = r.kx; const uint2 (&ky)[G] = r.ky; const uint2 (&va)[G] = r.va; const uint2 (&vb)[G] = r.vb;
    const uint32_t (&ks0)[G / 2] = r.ks0; const uint32_t (&ks1)[G / 2] = r.ks1;
    const uint32_t (&vs0)[G] = r.vs0; const uint32_t (&vs1)[G] = r.vs1;
    // ---- S^T = sum over groups of scale_K[token][grp] * (Kq . Q^T)
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#ifdef CBKV_MEASURE
    if (!(dbg & 32))  // skip the score phase
#endif
#pragma unroll
    for (int grp = 0; grp < G; grp++) {
        const uint32_t x0 = q8_fix<BF16>(kx[grp].x), x1 = q8_fix<BF16>(kx[grp].y);
        const uint32_t y0 = q8_fix<BF16>(ky[grp].x), y1 = q8_fix<BF16>(ky[grp].y);
        float sg[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t a[4];
        a[0] = q8_pair<BF16>(x0, SEL_LO); a[1] = q8_pair<BF16>(y0, SEL_LO);
        a[2] = q8_pair<BF16>(x0, SEL_HI); a[3] = q8_pair<BF16>(y0, SEL_HI);
        mma_16816<BF16>(sg, a, qf[0][2 * grp][0], qf[0][2 * grp][1]);
        a[0] = q8_pair<BF16>(x1, SEL_LO); a[1] = q8_pair<BF16>(y1, SEL_LO);
        a[2] = q8_pair<BF16>(x1, SEL_HI); a[3] = q8_pair<BF16>(y1, SEL_HI);
        mma_16816<BF16>(sg, a, qf[0][2 * grp + 1][0], qf[0][2 * grp + 1][1]);
        const float2 f0 = up2<BF16>(ks0[grp >> 1]), f1 = up2<BF16>(ks1[grp >> 1]);
        const float k0 = (grp & 1) ? f0.y : f0.x, k1 = (grp & 1) ? f1.y : f1.x;
        s[0] += sg[0] * k0; s[1] += sg[1] * k0; s[2] += sg[2] * k1; s[3] += sg[3] * k1;
    }
    // ---- online softmax over the tile's 16 tokens (rows g and g+8 of the fragment)
#pragma unroll
    for (int i = 0; i < 4; i++) s[i] *= scale_log2;
    if (need_mask) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int kp = kpos0 + g + (i >> 1) * 8, qp = qpos[0][i & 1];
            const bool ok = kp <= qp && (window <= 0 || kp + window > qp);
            if (!ok) s[i] = -INFINITY;
        }
    }
    float alpha[2] = {1.f, 1.f};
    bool moved = false;
#ifdef CBKV_MEASURE
    if (!(dbg & 64))  // skip the softmax
#endif
#pragma unroll
    for (int j = 0; j < 2; j++) {
        float mx = fmaxf(s[j], s[j + 2]);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        if (mx > m[0][j] + 8.f) {  // also the first finite maximum (m starts at -inf)
            alpha[j] = fast_ex2(m[0][j] - mx);
            m[0][j] = mx;
            moved = true;
        }
        const float m_use = (m[0][j] == -INFINITY) ? 0.f : m[0][j];
        const float p0 = fast_ex2(s[j] - m_use), p1 = fast_ex2(s[j + 2] - m_use);
        s[j] = p0; s[j + 2] = p1;
        l[0][j] = l[0][j] * alpha[j] + p0 + p1;
    }
    if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
        for (int mt = 0; mt < D / 16; mt++) {
            o[0][mt][0] *= alpha[0]; o[0][mt][1] *= alpha[1];
            o[0][mt][2] *= alpha[0]; o[0][mt][3] *= alpha[1];
        }
    }
    uint32_t pb0 = pack2<BF16>(s[0], s[1]), pb1 = pack2<BF16>(s[2], s[3]);
    pb0 = movmatrix_trans(pb0);  // tokens 2t, 2t+1 of column g
    pb1 = movmatrix_trans(pb1);  // tokens 2t+8, 2t+9
    // ---- O^T += sum over groups of Vq^T . (P^T * scale_V[token][grp])
#ifdef CBKV_MEASURE
    if (!(dbg & 128))  // skip the output phase
#endif
#pragma unroll
    for (int grp = 0; grp < G; grp++) {
        const uint32_t a0 = q8_fix<BF16>(va[grp].x), a1 = q8_fix<BF16>(va[grp].y);  // d 4g, 4g+1 | 4g+2, 4g+3 of tokens 2t, 2t+1
        const uint32_t c0 = q8_fix<BF16>(vb[grp].x), c1 = q8_fix<BF16>(vb[grp].y);  // the same of tokens 2t+8, 2t+9
        const uint32_t b0 = mul2<BF16>(pb0, vs0[grp]), b1 = mul2<BF16>(pb1, vs1[grp]);
        uint32_t a[4];
        a[0] = q8_pair<BF16>(a0, SEL_LO); a[1] = q8_pair<BF16>(a0, SEL_HI);
        a[2] = q8_pair<BF16>(c0, SEL_LO); a[3] = q8_pair<BF16>(c0, SEL_HI);
        mma_16816<BF16>(o[0][2 * grp], a, b0, b1);
        a[0] = q8_pair<BF16>(a1, SEL_LO); a[1] = q8_pair<BF16>(a1, SEL_HI);
        a[2] = q8_pair<BF16>(c1, SEL_LO); a[3] = q8_pair<BF16>(c1, SEL_HI);
        mma_16816<BF16>(o[0][2 * grp + 1], a, b0, b1);
    }
}

// ------------------------------------------------------------------ norm and rotation on the way
// A thread's query fragments hold both elements of a pair (d, d + D/2): k-steps ks and ks + D/32.  The cosine and sine
// words of its pairs:
template <int D, bool Q8>
__device__ __forceinline__ int q_word(int ks, int i, int t) {  // 32-bit word of the row behind fragment register [ks][i]
    return Q8 ? 16 * (ks >> 1) + 4 * t + 2 * (ks & 1) + i : ks * 8 + i * 4 + t;
}
template <int D>
__device__ __forceinline__ const uint32_t* rope_row(const RopeDev& r, int pos) {
    const int64_t p = pos < r.max_position ? pos : r.max_position - 1;  // the host refuses a step past the table
    return reinterpret_cast<const uint32_t*>(r.table) + p * (D / 2);
}
template <int D, bool Q8>
__device__ __forceinline__ void load_rope_words(const RopeDev& r, int pos, int t, uint32_t (&cs)[D / 32][2], uint32_t (&sn)[D / 32][2]) {
    const uint32_t* row = rope_row<D>(r, pos);
#pragma unroll
    for (int ks = 0; ks < D / 32; ks++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            cs[ks][i] = __ldg(row + q_word<D, Q8>(ks, i, t));
            sn[ks][i] = __ldg(row + D / 4 + q_word<D, Q8>(ks, i, t));
        }
}
template <int D, bool BF16, bool Q8>
__device__ __forceinline__ void rope_q_frags(const RopeDev& r, int t, bool live, const uint32_t (&cs)[D / 32][2], const uint32_t (&sn)[D / 32][2],
                                             uint32_t (&qf)[1][D / 16][2]) {
    if (r.q_weight) {
        float ss = 0.f;
#pragma unroll
        for (int ks = 0; ks < D / 16; ks++) ss = __fadd_rn(ss, __fadd_rn(sumsq2<BF16>(qf[0][ks][0]), sumsq2<BF16>(qf[0][ks][1])));
        ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, 1));  // the row is spread over the four lanes of a quad
        ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, 2));
        const float inv_rms = inv_rms_of(ss, D, r.eps);
        const uint32_t* w = reinterpret_cast<const uint32_t*>(r.q_weight);
        if (live) {
#pragma unroll
            for (int ks = 0; ks < D / 16; ks++)
#pragma unroll
                for (int i = 0; i < 2; i++) qf[0][ks][i] = norm2<BF16>(qf[0][ks][i], __ldg(w + q_word<D, Q8>(ks, i, t)), inv_rms, r.gemma != 0);
        }
    }
#pragma unroll
    for (int ks = 0; ks < D / 32; ks++)
#pragma unroll
        for (int i = 0; i < 2; i++) rotate2<BF16>(qf[0][ks][i], qf[0][ks + D / 32][i], cs[ks][i], sn[ks][i]);
}
// Sum of squares of a row, in every lane of the warp.
template <int D, bool BF16>
__device__ __forceinline__ float row_sumsq(const uint16_t* row, int lane) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(row);
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < D / 2; c += 32) ss = __fadd_rn(ss, c + lane < D / 2 ? sumsq2<BF16>(w[c + lane]) : 0.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));
    return ss;
}
// Words w, w + 1, ... of a K row (32-bit words, N of them, all in one half), normed and rotated.
template <int D, bool BF16, int N>
__device__ __forceinline__ void rope_k_words(const RopeDev& r, const uint32_t* row, int w, int pos, float inv_rms, uint32_t (&out)[N]) {
    const int lo = w % (D / 4);  // the words of the pairs in the first half
    const uint32_t* tr = rope_row<D>(r, pos);
    const uint32_t* wt = reinterpret_cast<const uint32_t*>(r.k_weight);
#pragma unroll
    for (int i = 0; i < N; i++) {
        uint32_t a = row[lo + i], b = row[D / 4 + lo + i];
        if (wt) {
            a = norm2<BF16>(a, __ldg(wt + lo + i), inv_rms, r.gemma != 0);
            b = norm2<BF16>(b, __ldg(wt + D / 4 + lo + i), inv_rms, r.gemma != 0);
        }
        rotate2<BF16>(a, b, __ldg(tr + lo + i), __ldg(tr + D / 4 + lo + i));
        out[i] = w < D / 4 ? a : b;
    }
}
template <int D, bool BF16>
__device__ __forceinline__ uint2 rope_k4(const RopeDev& r, const uint2* row, int c, int pos, float inv_rms) {
    uint32_t o[2];
    rope_k_words<D, BF16, 2>(r, reinterpret_cast<const uint32_t*>(row), 2 * c, pos, inv_rms, o);
    return make_uint2(o[0], o[1]);
}

// Fused append for int8 pages: kv_quantize (kv.rs:284-313) of the step's new K and V rows of one
// (sequence, kv head), written into the tile that was just fetched and into its record in HBM.
// Lane c owns values 4c..4c+3 (a 32-value group = 8 lanes); head_dim <= 128 per round.
template <int D, bool BF16, bool ROPE>
__device__ __forceinline__ void q8_append_row(uint32_t stage, uint8_t* recp, const uint16_t* krow, const uint16_t* vrow,
                                              int slot, int lane, const RopeDev& rope, int pos) {
    float inv_rms = 0.f;
    if constexpr (ROPE) { if (rope.k_weight) inv_rms = inv_rms_of(row_sumsq<D, BF16>(krow, lane), D, rope.eps); }
#pragma unroll
    for (int is_v = 0; is_v < 2; is_v++) {
        const uint2* src = reinterpret_cast<const uint2*>(is_v ? vrow : krow);
#pragma unroll
        for (int c0 = 0; c0 < D / 4; c0 += 32) {
            const int c = c0 + lane;
            const bool live = c < D / 4;
            float x[4] = {0.f, 0.f, 0.f, 0.f};
            if (live) {
                const uint2 raw = ROPE && !is_v ? rope_k4<D, BF16>(rope, src, c, pos, inv_rms) : src[c];
                x[0] = from_elem<BF16>((uint16_t)(raw.x & 0xffff)); x[1] = from_elem<BF16>((uint16_t)(raw.x >> 16));
                x[2] = from_elem<BF16>((uint16_t)(raw.y & 0xffff)); x[3] = from_elem<BF16>((uint16_t)(raw.y >> 16));
            }
            float amax = fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fmaxf(fabsf(x[2]), fabsf(x[3])));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
            const float scale = fmaxf(__fdiv_rn(amax, 127.0f), 1e-8f);
            if (live) {
                uint32_t word = 0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    float q = roundf(__fdiv_rn(x[i], scale));
                    q = fminf(fmaxf(q, -127.f), 127.f);
                    word |= (uint32_t)((int)q + 128) << (8 * i);
                }
                if (!is_v) {
                    const uint32_t off = (uint32_t)qrec_value_off(0, slot, 4 * c, 16, D);
                    asm volatile("st.shared.b32 [%0], %1;" ::"r"(stage + off), "r"(word) : "memory");
                    *reinterpret_cast<uint32_t*>(recp + off) = word;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const uint32_t off = (uint32_t)qrec_value_off(1, slot, 4 * c + i, 16, D);
                        const uint32_t b = (word >> (8 * i)) & 0xffu;
                        asm volatile("st.shared.u8 [%0], %1;" ::"r"(stage + off), "r"(b) : "memory");
                        recp[off] = (uint8_t)b;
                    }
                }
                if ((c & 7) == 0) {
                    const uint32_t off = (uint32_t)qrec_scale_off(is_v, slot, c >> 3, 16, D);
                    const uint32_t sv = to_elem<BF16>(scale);
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(stage + off), "h"((uint16_t)sv) : "memory");
                    *reinterpret_cast<uint16_t*>(recp + off) = (uint16_t)sv;
                }
            }
        }
    }
}

// Issue the TMA copies for one (page, kv head) tile: D/64 boxes of 32 rows x 64 elems.
template <int D>
__device__ __forceinline__ void issue_tile(const CUtensorMap* map, uint32_t stage, uint32_t bar, int row0) {
    mbar_expect_tx(bar, 32u * D * 2u);
#pragma unroll
    for (int x = 0; x < D / 64; x++) tma_load_2d(stage + x * 4096u, map, x * 64, row0, bar);
}

}  // namespace cbkv
