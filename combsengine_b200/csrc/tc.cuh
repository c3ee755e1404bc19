// Device helpers of the tcgen05 chunk kernels (prefill_tc.cu, chunk_pair.cu): barriers, copies, tensor-memory access, the
// work record of a CTA, and the partial rows of items cut along K/V.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "kernels.hpp"

namespace cbkv {

namespace {

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
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded: gives up after a wall-clock limit (the caller records it and winds down).
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, uint64_t limit_ns = 200000000ull) {
    for (int i = 0; i < 64; i++)
        if (mbar_try_wait(bar, parity)) return true;
    // the timer is slow to read, and a read in flight would hold up the return: look at it once per 64 polls
    const uint64_t t0 = global_ns();
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}
// The same in a role's loop: gives up as well when another role of the CTA has (looked at only while the barrier is not there).
__device__ __forceinline__ bool mbar_wait_unless(uint32_t bar, uint32_t parity, volatile int* failed) {
    for (int i = 0; i < 64; i++)
        if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (mbar_try_wait(bar, parity)) return true;
        if (*failed || global_ns() - t0 > 200000000ull) return false;
    }
}
// 16 bytes to shared memory without a register in between; zeros if not `there` (src is valid either way)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// K or V of one page of one kv head (LayerArena::map_page): all its column blocks in one copy
__device__ __forceinline__ void tma_load_page(uint32_t dst, const CUtensorMap* map, int is_v, int row16, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(0), "r"(is_v), "r"(row16), "r"(bar) : "memory");
}
// Non-blocking look at a barrier phase.
__device__ __forceinline__ uint32_t mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor (tcgen05): start address, leading / stride byte
// offsets (all >> 4), descriptor version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // version
    d |= (uint64_t)2 << 61;  // SWIZZLE_128B
    return d;
}
// Instruction descriptor, kind::f16: f32 accumulate, A/B f16 or bf16, M x N, operand majors.
__device__ __forceinline__ uint32_t instr_desc(bool bf16, int M, int N, bool b_mn_major) {
    uint32_t d = 0;
    d |= 1u << 4;                       // D format: f32
    d |= (bf16 ? 1u : 0u) << 7;         // A format
    d |= (bf16 ? 1u : 0u) << 10;        // B format
    d |= 0u << 15;                      // A: K-major
    d |= (b_mn_major ? 1u : 0u) << 16;  // B: K-major or MN-major
    d |= (uint32_t)(N >> 3) << 17;
    d |= (uint32_t)(M >> 4) << 24;
    return d;
}
// MMAs and commits are written for a converged warp: all lanes carry the operands, one elected lane issues.  Issued by one
// lane of a divergent branch instead, each operand is moved to the uniform registers that the instruction reads one by one
// and a 128 x 128 x 16 MMA, 64 cycles of the tensor pipe, took 83 (A in tensor memory) to 107 to issue.  With neither copies nor
// softmax (512 items of 62 K/V tiles at head_dim 128) the two-tile kernel takes 379 us this way, 438 the other, pairs of SMs 357 and 518.
__device__ __forceinline__ void umma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
          "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
          "r"(r[30]), "r"(r[31])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ float ex2_approx(float x) {  // one MUFU op; -inf -> 0
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
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

// Cycle counters per role, 16 slots per CTA: measurement build only (-DCBKV_MEASURE).
#ifdef CBKV_MEASURE
#define TC_NOW() clock64()
#define TC_ACC(var) do { if (a.dbg_buf) { const long long t1__ = clock64(); var += t1__ - tprev; tprev = t1__; } } while (0)
#define TC_DUMP(...) do { if (a.dbg_buf) { __VA_ARGS__ } } while (0)
#else
#define TC_NOW() 0ll
#define TC_ACC(var) do { (void)var; (void)tprev; } while (0)
#define TC_DUMP(...) do { } while (0)
#endif

constexpr int kTmemCols = 512;
constexpr int kPageCap = 2560;   // block-table entries staged in shared memory (40960 tokens); longer ranges read the rest from global memory

// The CTA's work: one TileItem, and what follows from it (both kernels; X counts the item's query tiles).
struct CtaWork {
    SeqMeta sm;
    int seq, h, qt, t0, t1, part, parts, slot_base, cut;
};
__device__ __forceinline__ CtaWork load_work(const ChunkArgs& a) {
    const int4* p = reinterpret_cast<const int4*>(a.tiles + blockIdx.x);
    const int4 x = __ldg(p), y = __ldg(p + 1);
    CtaWork w;
    w.seq = x.x; w.h = x.y; w.qt = x.z; w.t0 = x.w;
    w.t1 = y.x; w.part = y.y & 0xffff; w.parts = y.y >> 16; w.slot_base = y.z; w.cut = y.w;
    w.sm = a.step.seq_meta[w.seq];
    return w;
}

// Two runs of 32 columns of this thread's lane, both loads in flight before the wait
__device__ __forceinline__ void tmem_ld32x2(uint32_t first, uint32_t second, uint32_t (&r)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%64];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%65];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]),
          "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15]),
          "=&r"(r[16]), "=&r"(r[17]), "=&r"(r[18]), "=&r"(r[19]), "=&r"(r[20]), "=&r"(r[21]), "=&r"(r[22]), "=&r"(r[23]),
          "=&r"(r[24]), "=&r"(r[25]), "=&r"(r[26]), "=&r"(r[27]), "=&r"(r[28]), "=&r"(r[29]), "=&r"(r[30]), "=&r"(r[31]),
          "=&r"(r[32]), "=&r"(r[33]), "=&r"(r[34]), "=&r"(r[35]), "=&r"(r[36]), "=&r"(r[37]), "=&r"(r[38]), "=&r"(r[39]),
          "=&r"(r[40]), "=&r"(r[41]), "=&r"(r[42]), "=&r"(r[43]), "=&r"(r[44]), "=&r"(r[45]), "=&r"(r[46]), "=&r"(r[47]),
          "=&r"(r[48]), "=&r"(r[49]), "=&r"(r[50]), "=&r"(r[51]), "=&r"(r[52]), "=&r"(r[53]), "=&r"(r[54]), "=&r"(r[55]),
          "=&r"(r[56]), "=&r"(r[57]), "=&r"(r[58]), "=&r"(r[59]), "=&r"(r[60]), "=&r"(r[61]), "=&r"(r[62]), "=&r"(r[63])
        : "r"(first), "r"(second) : "memory");
}
// N consecutive columns of this thread's lane
template <int N>
__device__ __forceinline__ void tmem_ld_row(uint32_t taddr, uint32_t (&r)[N]) {
    static_assert(N == 32 || N == 64, "half a KV tile: 32 or 64 tokens");
    if constexpr (N == 32) tmem_ld32(taddr, r);
    else tmem_ld32x2(taddr, taddr + 32, r);
}
__device__ __forceinline__ float max3(float x, float y, float z) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(x), "f"(y), "f"(z));
    return r;
}
template <int N>
__device__ __forceinline__ float max_of(const uint32_t (&v)[N]) {
    float m[4] = {__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), __uint_as_float(v[3])};  // four chains
#pragma unroll
    for (int e = 4; e + 8 <= N; e += 8) {
#pragma unroll
        for (int c = 0; c < 4; c++) m[c] = max3(m[c], __uint_as_float(v[e + 2 * c]), __uint_as_float(v[e + 2 * c + 1]));
    }
    static_assert(N % 8 == 0, "the last four");
    return max3(max3(m[0], __uint_as_float(v[N - 4]), __uint_as_float(v[N - 3])), max3(m[1], __uint_as_float(v[N - 2]), __uint_as_float(v[N - 1])), fmaxf(m[2], m[3]));
}
// A pair of 32-bit numbers in one register pair: fma.rn.f32x2 and add.rn.f32x2 do two per issue slot.
__device__ __forceinline__ uint64_t f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t f32x2_bits(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ float2 f32x2_split(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t x, uint64_t y, uint64_t z) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t x, uint64_t y) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
// 2^(s * scale - ref) of N scores, packed in pairs in the order of the scores (out may be sv); adds them to `sum` (two pairs of chains).
template <int N, bool BF16>
__device__ __forceinline__ void exp_pack(const uint32_t* sv, uint64_t scale2, uint64_t neg_ref2, uint64_t (&sum)[2], uint32_t* out) {
#pragma unroll
    for (int e = 0; e < N; e += 2) {
        const float2 x = f32x2_split(fma2(f32x2_bits(sv[e], sv[e + 1]), scale2, neg_ref2));
        const float p0 = ex2_approx(x.x), p1 = ex2_approx(x.y);
        sum[(e >> 1) & 1] = add2(sum[(e >> 1) & 1], f32x2(p0, p1));
        out[e >> 1] = pack2<BF16>(p0, p1);
    }
}
__device__ __forceinline__ float sum_of(const uint64_t (&sum)[2]) {
    const float2 x = f32x2_split(add2(sum[0], sum[1]));
    return x.x + x.y;
}
// 16 packed columns of this thread's lane (the caller waits)
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
          "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
// A operand from tensor memory
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
// the same; whether x held in any of the threads
__device__ __forceinline__ bool bar_any(int id, int threads, bool x) {
    uint32_t any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(any) : "r"((uint32_t)x), "r"(id), "r"(threads) : "memory");
    return any != 0;
}

// 32 columns of one output row
template <bool BF16>
__device__ __forceinline__ void store_row32(uint16_t* dst, const float (&v)[32], float inv) {
#pragma unroll
    for (int u = 0; u < 4; u++) {
        uint4 w;
        w.x = pack2<BF16>(v[u * 8 + 0] * inv, v[u * 8 + 1] * inv);
        w.y = pack2<BF16>(v[u * 8 + 2] * inv, v[u * 8 + 3] * inv);
        w.z = pack2<BF16>(v[u * 8 + 4] * inv, v[u * 8 + 5] * inv);
        w.w = pack2<BF16>(v[u * 8 + 6] * inv, v[u * 8 + 7] * inv);
        *reinterpret_cast<uint4*>(dst + u * 8) = w;
    }
}

// ---- items cut along K/V.  A slice's rows go to memory un-normalised, with each row's (reference exponent, sum);
// only the rows that exist are written, packed (row = q head * valid tokens + token), the row being the fast index:
// a warp's accesses are contiguous, and a few tokens' rows cost a few KB, not the whole tile.
template <int D>
__device__ __forceinline__ float4* slice_rows(const ChunkArgs& a, int slot, int n_x, int X) {
    return reinterpret_cast<float4*>(a.split_o) + ((size_t)slot * n_x + X) * (D / 4) * 128;
}
// Adds the slices of query tile X up: `rows` packed rows of `nv` tokens per q head, first token r0x.  Every thread of
// `threads` takes (row, 8 columns) items; the loads of four slices travel together, so an item costs one round trip to
// L2 per four slices however few rows there are.
template <int D, bool BF16>
__device__ __forceinline__ void merge_slices(const ChunkArgs& a, const CtaWork& wk, int n_x, int X, int nv, int r0x, int r, int threads) {
    const int rows = a.geo.n_rep * nv, n_rep = a.geo.n_rep;
    for (int idx = r; idx < rows * (D / 8); idx += threads) {
        const int c8 = idx / rows, row = idx - c8 * rows;
        float M = -INFINITY, L = 0.f;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
#pragma unroll 1
        for (int p0 = 0; p0 < wk.parts; p0 += 4) {
            float2 ml[4];
            float4 u[4], v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const bool ok = p0 + q < wk.parts;
                const int slot = wk.slot_base + p0 + (ok ? q : 0);
                ml[q] = __ldcg(a.split_ml + ((size_t)slot * n_x + X) * 128 + row);
                const float4* src = slice_rows<D>(a, slot, n_x, X) + row;
                u[q] = __ldcg(src + (size_t)(2 * c8) * 128);
                v[q] = __ldcg(src + (size_t)(2 * c8 + 1) * 128);
                if (!ok) ml[q] = make_float2(-INFINITY, 0.f);
            }
            float Mn = M;
#pragma unroll
            for (int q = 0; q < 4; q++) Mn = fmaxf(Mn, ml[q].x);
            const float so = M == -INFINITY ? 0.f : exp2f(M - Mn);
            x.x *= so; x.y *= so; x.z *= so; x.w *= so; y.x *= so; y.y *= so; y.z *= so; y.w *= so; L *= so;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (ml[q].x == -INFINITY) continue;  // keys this row does not see
                const float f = exp2f(ml[q].x - Mn);
                x.x += f * u[q].x; x.y += f * u[q].y; x.z += f * u[q].z; x.w += f * u[q].w;
                y.x += f * v[q].x; y.y += f * v[q].y; y.z += f * v[q].z; y.w += f * v[q].w;
                L += f * ml[q].y;
            }
            M = Mn;
        }
        const float inv = 1.f / L;
        uint4 w;
        w.x = pack2<BF16>(x.x * inv, x.y * inv); w.y = pack2<BF16>(x.z * inv, x.w * inv);
        w.z = pack2<BF16>(y.x * inv, y.y * inv); w.w = pack2<BF16>(y.z * inv, y.w * inv);
        const int rep = row / nv, tok = r0x + row - rep * nv;
        uint16_t* orow = reinterpret_cast<uint16_t*>(a.out) + ((size_t)wk.sm.tok_off * a.geo.n_q + (size_t)(wk.h * n_rep + rep) * wk.sm.snew + tok) * D;
        *reinterpret_cast<uint4*>(orow + c8 * 8) = w;
    }
}
// The CTA's slices are written: draw the item's ticket.  True in every one of the `threads` calling threads (named
// barrier `bar`, thread `first` among them) when it was the last one.  No CTA waits for another.
__device__ __forceinline__ bool last_slice(const ChunkArgs& a, const CtaWork& wk, int bar, int threads, bool first, int* s_ticket) {
    __threadfence();
    bar_sync(bar, threads);
    if (first) {
        const int tk = atomicAdd(a.split_counter + wk.cut, 1);
        if (tk == wk.parts - 1) a.split_counter[wk.cut] = 0;  // ready for the next launch
        *s_ticket = tk;
        __threadfence();
    }
    bar_sync(bar, threads);
    return *s_ticket == wk.parts - 1;
}

}  // namespace

}  // namespace cbkv
