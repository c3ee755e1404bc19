// Chunk (prefill) attention on the 5th-generation tensor cores: tcgen05.mma with
// accumulators in tensor memory, operands staged in shared memory by TMA.
// Reference math: attend() with seq > 1, kv.rs:243-268 — scores = q k^T * scale, causal
// mask aligned to the chunk's position (kv.rs:247-251), optional window (kv.rs:252-257),
// softmax over keys, P V — here as a flash-style loop over 128-token KV tiles.
//
// One CTA = one (sequence, kv head, tile of query tokens).  The 128 rows of the MMA are
// "columns" of the problem: row m = rep * TPT + i is q head `rep` of the kv group at
// the tile's i-th token (TPT = 128 / RS tokens, RS = n_rep rounded up to a power of
// two), so the K/V tiles are shared by the whole q-head group.
//
//   warp 0        TMA producer: one copy per page and operand
//   warp 1        converged, one elected lane issues tcgen05.mma: S = Q K^T (two S buffers), O += P V,
//                 whichever has its operands first
//   warps 2..9    softmax: two threads per TMEM lane (row), one for each half of a tile's keys; P goes back to
//                 tensor memory over its S columns (16-bit pairs) and is the A operand of P V; O rescaled in
//                 TMEM when a row max moves
//
// KV tiles hold KT tokens: 128 for head_dim 64 and 128; 64 for head_dim 256, where two S buffers of 128 columns, Q
// (128) and O (256) would be more than the 512 columns of tensor memory, and three K and three V buffers of 64 KB more
// than shared memory (S = Q K^T is then 128 x 64 and O += P V one 128 x 256 MMA per 16 keys).
//
// Tensor memory: S0 [0,KT), S1 [KT, 2 KT), Q [2 KT, 2 KT + D / 2) packed, O [512 - D, 512) -> 512 columns allocated.
// Shared memory: kTcBufs K and V buffers each, [page][8-token group][column block][8 rows x 128 bytes]:
// the five-dimensional view of a layer (LayerArena::map_page) takes K or V of a page out of the arena's
// [K 0-7][V 0-7][K 8-15][V 8-15] order in one copy.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "kernels.hpp"
#include "pdl.cuh"
#include "q8_unpack.cuh"
#include "tc.cuh"

namespace cbkv {

namespace {

constexpr int kThreads = 320;

constexpr int kTcBufs = 3;       // K buffers and V buffers of the one-tile kernel

template <int D>
struct TcKeys { static constexpr int value = D == 256 ? 64 : 128; };  // tokens per KV tile

template <int D>
constexpr int tc_smem_bytes() {
    // K and V buffers of KT tokens x D, barriers, the staged block table and the half-row exchange; at least 120 KB
    // so that two CTAs never share an SM (each allocates all 512 tensor-memory columns)
    constexpr int need = 2 * kTcBufs * TcKeys<D>::value * D * 2 + 256 + kPageCap * 4 + 2 * 128 * 2 * 4 + 64;
    return need < 120 * 1024 ? 120 * 1024 : need;
}

}  // namespace

template <int D, bool BF16>
__global__ void __launch_bounds__(kThreads) chunk_tc_kernel(const __grid_constant__ CUtensorMap tmap, const ChunkArgs a) {
    constexpr int XB = D / 64;                 // column blocks per row
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int KT = TcKeys<D>::value;       // tokens per KV tile
    constexpr int HK = KT / 2;                 // keys of a softmax thread
    constexpr int PPT = KT / 16;               // pages per KV tile
    constexpr uint32_t KVB = (uint32_t)KT * D * 2u;  // K or V of KT tokens: [page][8-token group][column block][8 rows of 128 bytes]
    constexpr uint32_t PGB = 16u * D * 2u;           // one page of it
    constexpr int NB = kTcBufs;
    uint8_t* sK = smem;                 // NB K buffers, NB V buffers: K is free again once its scores are computed
    uint8_t* sV = sK + NB * KVB;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + NB * KVB);
    const uint32_t b_k_full = smem_u32(bars + 0), b_k_empty = smem_u32(bars + NB), b_v_full = smem_u32(bars + 2 * NB), b_v_empty = smem_u32(bars + 3 * NB);
    const uint32_t b_s_full = smem_u32(bars + 4 * NB), b_p_full = smem_u32(bars + 4 * NB + 2), b_o_done = smem_u32(bars + 4 * NB + 4);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4 * NB + 5);
    volatile int* failed = reinterpret_cast<volatile int*>(bars + 4 * NB + 6);
    int* s_ticket = reinterpret_cast<int*>(bars + 4 * NB + 7);
    int* s_asked = reinterpret_cast<int*>(bars + 4 * NB + 8);  // K and V buffers whose copies have been announced
    const uint32_t b_drain = smem_u32(bars + 4 * NB + 9);
    static_assert(4 * NB + 10 <= 32, "barriers");
    int* s_pages = reinterpret_cast<int*>(bars + 32);   // [kPageCap] physical pages of the KV range
    float* s_xch = reinterpret_cast<float*>(s_pages + kPageCap);  // [2 buffers][128 rows][2 halves]
    int* s_pair = reinterpret_cast<int*>(s_xch + 2 * 128 * 2);    // [4 pairs of warps][tile parity] a wait ran out

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if ((smem_u32(smem) & 1023u) != 0) {
        if (tid == 0) atomicOr(a.status, ST_SMEM_ALIGN);
        return;
    }
    // ---- which (sequence, kv head, query tile), which slice of its K/V tiles
    const CtaWork wk = load_work(a);
    const SeqMeta sm = wk.sm;
    const int Hkv = a.geo.n_kv, n_rep = a.geo.n_rep, RS = a.rep_slots, TPT = 128 / RS, h = wk.h;
    const int r0 = wk.qt * TPT;                            // first new token of the tile
    const int nv = min(TPT, sm.snew - r0);                 // tokens of it
    const int q_min = sm.pos + r0, q_max = q_min + nv - 1;
    const int lo_key = a.window > 0 ? max(0, q_min - a.window + 1) : 0;
    const int p_lo = (lo_key >> 4) + wk.t0 * PPT, p_hi = min(q_max >> 4, (lo_key >> 4) + wk.t1 * PPT - 1);
    const int n_tiles = wk.t1 - wk.t0;
    const int k0 = p_lo * 16;                               // absolute position of key 0 of tile 0

    if (tid == 0) {
        for (int i = 0; i < NB; i++) {
            mbar_init(b_k_full + i * 8, 1); mbar_init(b_k_empty + i * 8, 1); mbar_init(b_v_full + i * 8, 1); mbar_init(b_v_empty + i * 8, 1);
        }
        for (int i = 0; i < 2; i++) { mbar_init(b_s_full + i * 8, 1); mbar_init(b_p_full + i * 8, D == 64 ? 8 : 256); }
        mbar_init(b_o_done, 1);
        mbar_init(b_drain, 1);
        *failed = 0;
        for (int i = 0; i < 8; i++) s_pair[i] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap) : "memory");
    }
    if (warp == 0) {  // tensor memory for this CTA
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i <= p_hi - p_lo && i < kPageCap; i += kThreads) s_pages[i] = a.step.tables[sm.tbl_off + p_lo + i];
    tc_fence_before();
    __syncthreads();  // barriers and block table are ready: the producer starts while the other warps bring Q
    tc_fence_after();
    // q, the pages and the partial-result buffers belong to earlier launches until here; everything above (barriers,
    // tensor memory, the work record and the block table, which came with the step's upload) runs under their tail
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t tS0 = tmem, tQ = tmem + 2 * KT, tO = tmem + 512 - D;
    static_assert(2 * KT + D / 2 + D <= 512, "tensor memory");
    // ---- Q goes to tensor memory (the A operand of S, packed pairs like P): from shared memory the 128-row A and the
    // K tile together would need more than the 128 bytes a cycle that it delivers.  Row m = rep * TPT + i; each of a
    // row's two softmax threads brings half of it; rows past the data are zero.
    if (warp >= 2) {
        const int m = (warp & 3) * 32 + lane, H = (warp - 2) >> 2, rep = m / TPT, i = m - rep * TPT;
        const bool row_ok = rep < n_rep && i < nv;
        const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(a.q) + (size_t)sm.tok_off * a.geo.n_q * D +
                                                          ((size_t)(h * n_rep + (row_ok ? rep : 0)) * sm.snew + r0 + (row_ok ? i : 0)) * D + H * (D / 2));
#pragma unroll
        for (int c = 0; c < D / 64; c++) {  // 32 elements: 16 packed columns
            uint32_t w[16];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint4 v = row_ok ? src[c * 4 + u] : make_uint4(0, 0, 0, 0);
                w[u * 4] = v.x; w[u * 4 + 1] = v.y; w[u * 4 + 2] = v.z; w[u * 4 + 3] = v.w;
            }
            tmem_st16(tQ + ((uint32_t)(warp & 3) << 21) + H * (D / 4) + c * 16, w);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    if (warp >= 1) bar_sync(10, kThreads - 32);  // every warp but the producer
    tc_fence_after();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        // The block-table entries of the whole KV range were staged in shared memory by all threads; one copy per
        // page brings its K, another its V, each issued by the page's lane.
        bool ok = true;
        int asked[2] = {0, 0};
        long long tprev = TC_NOW(), c_wait = 0, c_issue = 0;
#pragma unroll 1
        for (int j = 0; j < n_tiles && ok; j++) {
            const int st = j % NB;
            // pages past the last visible one repeat it: finite data that the causal mask hides
            int phys = 0;
            if (lane < PPT) {
                const int idx = min(j * PPT + lane, p_hi - p_lo);
                phys = idx < kPageCap ? s_pages[idx] : a.step.tables[sm.tbl_off + p_lo + idx];
                if (phys < 0 || phys >= a.geo.num_pages) { atomicOr(a.status, ST_BAD_PAGE); phys = 0; }
            }
#pragma unroll
            for (int is_v = 0; is_v < 2 && ok; is_v++) {
                const uint32_t full = (is_v ? b_v_full : b_k_full) + st * 8, empty = (is_v ? b_v_empty : b_k_empty) + st * 8;
                if (lane == 0) {
                    if (j >= NB && !mbar_wait_bounded(empty, (j / NB - 1) & 1)) ok = false;
                    TC_ACC(c_wait);
                    if (*failed) ok = false;
                    if (ok) { mbar_expect_tx(full, KVB); asked[is_v]++; }
                    else { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (ok && lane < PPT && (j != a.fault_tile || blockIdx.x != 0))
                    tma_load_page(smem_u32((is_v ? sV : sK) + st * KVB + lane * PGB), &tmap, is_v, (phys * Hkv + h) * 2, full);
                if (lane == 0) TC_ACC(c_issue);
            }
        }
        if (lane == 0) { s_asked[0] = asked[0]; s_asked[1] = asked[1]; }
        TC_DUMP(if (lane == 0) { a.dbg_buf[(size_t)blockIdx.x * 16 + 0] = c_wait; a.dbg_buf[(size_t)blockIdx.x * 16 + 1] = c_issue; a.dbg_buf[(size_t)blockIdx.x * 16 + 15] = n_tiles; });
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        {
            const uint32_t id_qk = instr_desc(BF16, 128, KT, false);
            const uint32_t id_pv = instr_desc(BF16, 128, D, true);
            // descriptors differ only in the start address field (bits 0-13, address >> 4); 8-token groups of K and V
            // are XB * 1024 bytes apart, 64-wide column blocks 1024
            const uint64_t dk = smem_desc(smem_u32(sK), 16, XB * 1024), dv = smem_desc(smem_u32(sV), 1024, XB * 1024);
            auto issue_qk = [&](int j) {
                const uint64_t kst = (uint64_t)((uint32_t)(j % NB) * KVB >> 4);
#pragma unroll
                for (int ks = 0; ks < D / 16; ks++)  // 16 elements = 32 bytes inside the swizzled row, four steps per 64-column block
                    umma_ts(tS0 + (j & 1) * KT, tQ + ks * 8, dk + kst + (uint64_t)(((ks >> 2) * 1024 + (ks & 3) * 32) >> 4), id_qk, ks > 0);
                umma_commit(b_s_full + (j & 1) * 8);
                umma_commit(b_k_empty + (j % NB) * 8);
            };
            long long tprev = TC_NOW(), c_wkv = 0, c_wp = 0, c_iss = 0;
            bool ok = true;
            int next_qk = 0;  // scores issued so far
#pragma unroll 1
            for (int j = 0; ok && j < n_tiles; j++) {
                // Until this tile's P is there: the scores of the next tile as soon as its K has landed.  They go to the
                // other S buffer, whose P the previous P V (issued before) was the last to read.  Neither waits for the
                // other: a P V held up by a K that is still on its way would hold up the V buffer it frees.
                uint64_t t0 = 0;
                for (int n = 0;; n++) {
                    if (next_qk <= j + 1 && next_qk < n_tiles && __all_sync(0xffffffffu, mbar_test_wait(b_k_full + (next_qk % NB) * 8, (next_qk / NB) & 1))) {
                        TC_ACC(c_wkv);
                        tc_fence_after();
                        issue_qk(next_qk++);
                        TC_ACC(c_iss);
                    }
                    if (next_qk > j && __all_sync(0xffffffffu, mbar_test_wait(b_p_full + (j & 1) * 8, (j >> 1) & 1))) break;
                    if ((n & 63) == 63) {
                        if (*failed) ok = false;
                        if (t0 == 0) t0 = global_ns();
                        else if (global_ns() - t0 > 200000000ull) ok = false;
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                    }
                }
                TC_ACC(c_wp);
                if (ok) ok = __all_sync(0xffffffffu, mbar_wait_bounded(b_v_full + (j % NB) * 8, (j / NB) & 1) && !*failed);
                TC_ACC(c_wkv);
                if (!ok) break;
                tc_fence_after();
                const int st = j % NB;
                const uint64_t vst = (uint64_t)((st * KVB) >> 4);
#pragma unroll
                for (int ks = 0; ks < PPT; ks++)  // 16 keys per step = one page; P: 8 packed columns, V: MN-major
                    umma_ts(tO, tS0 + (j & 1) * KT + ks * 8, dv + vst + (uint64_t)((ks * PGB) >> 4), id_pv, (j > 0 || ks > 0));
                umma_commit(b_v_empty + st * 8);
                umma_commit(b_o_done);
                TC_ACC(c_iss);
            }
            if (!ok) {
                if (lane == 0) { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                umma_commit(b_drain);  // waited for below
            }
            TC_DUMP(if (lane == 0) { a.dbg_buf[(size_t)blockIdx.x * 16 + 2] = c_wkv; a.dbg_buf[(size_t)blockIdx.x * 16 + 3] = c_wp; a.dbg_buf[(size_t)blockIdx.x * 16 + 4] = c_iss; });
        }
    } else {
        // ------------------------------------------------------------ softmax + epilogue: two threads per row
        // The warps come in pairs that may touch the same quarter of the tensor-memory lanes; H = 0 takes the first
        // half of a tile's keys and of the O columns, H = 1 the second.
        const int H = (warp - 2) >> 2;
        const int lane_base = (warp & 3) * 32;             // the TMEM lanes this warp may touch
        const int m = lane_base + lane;                    // row of the tile
        const int rep = m / TPT, i = m - rep * TPT;
        const bool row_ok = rep < n_rep && i < nv;
        const int q_pos = q_min + min(i, nv - 1);          // rows past the data mimic the last token
        const uint32_t lane_addr = (uint32_t)lane_base << 16;
        const int pair_bar = 1 + (warp & 3);
        // A named barrier has no time limit, so the two warps of a pair must leave the loop in the same
        // iteration: whichever sees a wait run out says so before the pair's barrier, both read it after.  Two flags
        // in turn: a warp may be at the next tile before the other has read this one's.
        // Exponents are taken against a reference maximum that is only moved when a row's maximum
        // exceeds it by more than 8 (a factor 256): probabilities then stay below 256, exact enough in
        // f16/bf16 with f32 sums, and O needs rescaling only on those rare moves.
        float m_ref = -INFINITY, l_run = 0.f;              // l_run: this half's share of the row sum
        bool ok = true;
        long long tprev = TC_NOW(), c_ws = 0, c_ld = 0, c_exp = 0, c_wo = 0, c_st = 0;
        const long long tstart = tprev;
#pragma unroll 1
        for (int j = 0; j < n_tiles; j++) {
            ok = D == 64 ? mbar_wait_unless(b_s_full + (j & 1) * 8, (j >> 1) & 1, failed) : mbar_wait_bounded(b_s_full + (j & 1) * 8, (j >> 1) & 1) && !*failed;
            ok = __all_sync(0xffffffffu, ok);
            TC_ACC(c_ws);
            volatile int* pair_failed = s_pair + (warp & 3) * 2 + (j & 1);
            if (!ok && lane == 0) *pair_failed = 1;  // the loads below then read stale columns: harmless, nothing is kept
            tc_fence_after();
            const uint32_t tS = tS0 + (j & 1) * KT + lane_addr;
            const int kbase = k0 + j * KT + H * HK;
            const bool need_mask = (kbase + HK - 1 > q_min) || (a.window > 0 && kbase + a.window <= q_max);
            uint32_t sv[HK];
            tmem_ld_row<HK>(tS + H * HK, sv);
            if (need_mask) {
#pragma unroll
                for (int e = 0; e < HK; e++) {
                    const int kp = kbase + e;
                    if (!(kp <= q_pos && (a.window <= 0 || kp + a.window > q_pos))) sv[e] = 0xff800000u;  // -inf
                }
            }
            float mx;
            if constexpr (D == 64) {
                mx = max_of(sv);
            } else {
                float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
                for (int e = 0; e < HK; e += 4) {
                    m0 = fmaxf(m0, __uint_as_float(sv[e])); m1 = fmaxf(m1, __uint_as_float(sv[e + 1]));
                    m2 = fmaxf(m2, __uint_as_float(sv[e + 2])); m3 = fmaxf(m3, __uint_as_float(sv[e + 3]));
                }
                mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
            }
            float* xrow = s_xch + ((j & 1) * 128 + m) * 2;
            xrow[H] = mx;
            bar_sync(pair_bar, 64);  // also: both warps have their S columns in registers, so P may overwrite them
            mx = fmaxf(mx, xrow[H ^ 1]) * a.scale_log2;  // scale > 0: the maximum commutes with the scaling
            if (*pair_failed) { ok = false; break; }     // both warps of the pair, in the same iteration
            TC_ACC(c_ld);
            float alpha = 1.f;
            if (mx > m_ref + 8.f || m_ref == -INFINITY) {  // both halves see the same mx: the same decision
                alpha = (m_ref == -INFINITY) ? 0.f : exp2f(m_ref - mx);
                m_ref = mx;
            }
            const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
            float sum_all;
            if constexpr (D == 64) {
                uint64_t sum[2] = {0ull, 0ull};
                exp_pack<HK, BF16>(sv, f32x2(a.scale_log2, a.scale_log2), f32x2(-m_use, -m_use), sum, sv);  // a pair reuses a register whose score is consumed
                sum_all = sum_of(sum);
            } else {  // (two at a time, and maxima of three above, spill at head_dim 256: verification there was 2 % slower with
                      // them; 128 comes here only when asked for, 4 % slower on long prompts, 600 / 576 us, and equal on short steps)
                float sum = 0.f, sum2 = 0.f;
#pragma unroll
                for (int e = 0; e < HK; e += 2) {
                    const float p0 = ex2_approx(fmaf(__uint_as_float(sv[e]), a.scale_log2, -m_use));
                    const float p1 = ex2_approx(fmaf(__uint_as_float(sv[e + 1]), a.scale_log2, -m_use));
                    if (e & 2) sum2 += p0 + p1; else sum += p0 + p1;  // two chains
                    sv[e >> 1] = pack2<BF16>(p0, p1);
                }
                sum_all = sum + sum2;
            }
#pragma unroll
            for (int c = 0; c < HK / 32; c++) tmem_st16(tS + H * (HK / 2) + c * 16, sv + c * 16);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            l_run = l_run * alpha + sum_all;
            TC_ACC(c_exp);
            // O may be rescaled once the previous P V is complete.  A parity wait cannot tell a phase from the one two
            // before it, so it holds only where the phase before the awaited one is known to be complete.  Here: the
            // scores of tile j were issued after P V of tile j - 2, so S being full says that phase j - 2 is.
            if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                bool done = mbar_wait_bounded(b_o_done, (j - 1) & 1) && !*failed;
                done = __all_sync(0xffffffffu, done);
                TC_ACC(c_wo);
                if (!done) {
                    if (lane == 0) { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                } else {
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < D / 64; c++) {
                        uint32_t v[32];
                        tmem_ld32(tO + lane_addr + H * (D / 2) + c * 32, v);
#pragma unroll
                        for (int e = 0; e < 32; e++) v[e] = __float_as_uint(__uint_as_float(v[e]) * alpha);
                        tmem_st32(tO + lane_addr + H * (D / 2) + c * 32, v);
                    }
                }
            }
            tc_fence_before();     // the tensor-memory traffic above is ordered before the hand-over
            if constexpr (D == 64) {
                __syncwarp();
                if (lane == 0) mbar_arrive(b_p_full + (j & 1) * 8);
            } else {
                mbar_arrive(b_p_full + (j & 1) * 8);
            }
            TC_ACC(c_st);
        }
        TC_DUMP(if (tid == 64) {
            unsigned long long* b = a.dbg_buf + (size_t)blockIdx.x * 16;
            b[5] = c_ws; b[6] = c_ld; b[7] = c_exp; b[8] = c_wo; b[9] = c_st; b[10] = TC_NOW() - tstart;
        });
        (void)tstart; (void)c_wo;
        // ---- epilogue: O / l -> out, or a slice's partial rows.  The last scores say that P V of tile n - 3 is complete
        // and no more, so phase n - 2 is waited for before n - 1: asked for n - 1 alone, a barrier still in phase n - 2
        // would answer with phase n - 3, of the same parity (with n = 2, with none at all).
        if (ok && n_tiles > 1) ok = mbar_wait_bounded(b_o_done, (n_tiles - 2) & 1);
        if (ok) ok = mbar_wait_bounded(b_o_done, (n_tiles - 1) & 1) && !*failed;
        ok = __all_sync(0xffffffffu, ok);
        float* xrow = s_xch + ((n_tiles & 1) * 128 + m) * 2;
        xrow[H] = l_run;
        bar_sync(pair_bar, 64);
        const float l_row = l_run + xrow[H ^ 1];
        if (!ok && lane == 0) {
            *failed = 1;
            atomicOr(a.status, ST_WAIT_TIMEOUT);
        }
        tc_fence_after();
        if (wk.parts == 1) {
            if (ok) {
                const float inv = 1.f / l_row;
                uint16_t* orow = reinterpret_cast<uint16_t*>(a.out) +
                                 ((size_t)sm.tok_off * a.geo.n_q + (size_t)(h * n_rep + (row_ok ? rep : 0)) * sm.snew + (row_ok ? r0 + i : 0)) * D;
#pragma unroll 1
                for (int c = H * (D / 64); c < (H + 1) * (D / 64); c++) {
                    uint32_t v[32];
                    tmem_ld32(tO + lane_addr + c * 32, v);
                    float f[32];
#pragma unroll
                    for (int e = 0; e < 32; e++) f[e] = __uint_as_float(v[e]);
                    if (row_ok) store_row32<BF16>(orow + c * 32, f, inv);
                }
            }
        } else {
            const int slot = wk.slot_base + wk.part, prow = rep * nv + i;
            if (ok) {
                float4* rows = slice_rows<D>(a, slot, 1, 0) + prow;
#pragma unroll 1
                for (int c = H * (D / 64); c < (H + 1) * (D / 64); c++) {
                    uint32_t v[32];
                    tmem_ld32(tO + lane_addr + c * 32, v);
                    if (row_ok) {
#pragma unroll
                        for (int u = 0; u < 8; u++)
                            rows[(size_t)(c * 8 + u) * 128] = make_float4(__uint_as_float(v[u * 4]), __uint_as_float(v[u * 4 + 1]),
                                                                          __uint_as_float(v[u * 4 + 2]), __uint_as_float(v[u * 4 + 3]));
                    }
                }
                if (H == 0 && row_ok) a.split_ml[(size_t)slot * 128 + prow] = make_float2(m_ref, l_row);
            }
            // every softmax warp passes the barriers whatever happened to its waits
            if (last_slice(a, wk, 9, 256, tid == 64, s_ticket) && !*failed)
                merge_slices<D, BF16>(a, wk, 1, 0, nv, r0, tid - 64, 256);
        }
    }
    // ---- wind down: everybody meets, then the allocating warp frees the tensor memory
    tc_fence_before();
    __syncthreads();
    // Never leave with a product or a copy in flight if somebody gave up (a copy's barrier is in the phase announced last, or
    // past it).  If the issuer was not the one, its last product has the limit of the first wait to end.
    if (tid == 0 && *failed) {
        mbar_wait_bounded(b_drain, 0);
        for (int is_v = 0; is_v < 2; is_v++)
            for (int i = max(0, s_asked[is_v] - NB); i < s_asked[is_v]; i++) mbar_wait_bounded((is_v ? b_v_full : b_k_full) + (i % NB) * 8, (i / NB) & 1);
    }
    __syncwarp();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

template <int D, bool BF16>
static cudaError_t launch_tc(const CUtensorMap& map, const ChunkArgs& a, bool overlap, cudaStream_t st) {
    if (a.n_items <= 0) return cudaSuccess;
    return launch_pdl(overlap, chunk_tc_kernel<D, BF16>, a.n_items, kThreads, tc_smem_bytes<D>(), st, map, a);
}


// ------------------------------------------------------------------ two query tiles per CTA
// The second-generation kernel: each CTA works on two 128-row query tiles (A and B) that
// share every K/V tile, which halves the shared-memory fill per FLOP, and keeps P in tensor
// memory (it overwrites the first 64 columns of its S tile as packed 16-bit pairs and is the
// A operand of the P V product), so no shared memory is spent on P.
//
//   warp 0        TMA producer: two K and two V buffers, one copy per page of each
//   warp 1        MMA issuer:  QK_A, QK_B, then per K/V tile  PV_A, QK_A', PV_B, QK_B'
//   warps 2..9    softmax of tile A        warps 10..17  softmax of tile B
//
// A tile's softmax is the longest link of the chain QK -> softmax -> PV, and that chain sets the pace.  Two threads share
// a row: the warps of a tile come in pairs that may touch the same quarter of the tensor-memory lanes; H = 0 takes keys
// 0-31 and 64-95 of the tile, H = 1 the others (and, when the row maximum moves, the matching half of the O columns).
// They exchange their maxima through shared memory once per tile and their sums once at the end.  P is handed over in two
// halves, so that P V of keys 0-63 runs under the exponentials of keys 64-127 and only 256 of its 512 cycles are part of the chain.
//
// K and V have buffers of their own: K of the tile after next is asked for when the scores of this one are computed, and so has
// one and a half tiles of time to arrive; in one buffer with V, which is read last, it had half of one (without softmax a
// launch of 512 items of 62 K/V tiles took 546 us with copies, 379 without).  The same launch, softmax and all: 630 us with one
// buffer, one lane issuing, P handed over whole and a load of the scores at a time, 518 now (1028 TFLOP/s; a chain of 3600 cycles
// per tile, 2048 of them MMA; without the exponentials 485, without copies 508, with neither 465).  Verification of drafts, 8 sequences x 5 tokens after 512 to 6144, 28 layers: 1642 -> 1461 us.
//
// Tensor memory: S_A [0,128), S_B [128,256), O_A [256,384), O_B [384,512).
constexpr int kThreads2 = 576;

template <int D>
constexpr int tc2_smem_bytes() {
    return 2 * 128 * D * 2 /* Q_A, Q_B */ + 2 * 2 * 128 * D * 2 /* two K and two V buffers */ + 256 + kPageCap * 4 +
           2 * 2 * 128 * 2 * 4 /* half-row maxima of both tiles, double-buffered */;
}

// Q8: the layer holds int8 records (kernels.hpp, qrec_*) and the kernel converts them itself
// (cbkv_set_chunk_kernel mode 4; by default int8 layers go through a float copy, which is faster so far).
// Two warps after the softmax warps take the TMA producer's place, one for K and one for V.  Each keeps a
// ring of raw half-records (a record's K bytes and K scales, or its V bytes and V scales: two boxes of
// the layer's byte tensor maps) in flight, turns a landed half-record into q * scale in registers
// (q8_unpack.cuh: kv_dequantize, kv.rs:319-358), stores that where the tensor pipe reads it, and refills
// the slot itself.  Shared memory is cut differently from the float kernel: K is double-buffered as there
// (the scores of the next tile are issued a tile ahead), V has one buffer (P.V of a tile is the last thing
// that reads it), and the 32 KB this frees plus the tail of the allocation hold 8 K and 14 V half-records.
// Measured on 8 prompts x 8192 tokens: 2.4 times the float-copy route's time.  The V buffer can only be
// refilled between the last P.V of a tile and the first of the next, and one warp needs about 1400 cycles
// per half-record there (wait, convert, refill), eight times per tile; 640 threads at 96 registers leave no
// room for more converting warps, and 227 KB no room for a second V buffer beside the raw rings.
constexpr int kLoaders2 = 2;
constexpr int kThreads2Q8 = kThreads2 + kLoaders2 * 32;
constexpr int kRawK = 8, kRawV = 14;       // half-records per ring
constexpr int kRawVInStage = 7;            // V slots that fit behind the K ring in the freed stage quarter
template <int D>
constexpr int tc2_half_rec() { return 16 * D + 16 * (D / 32) * 2; }  // values + scales of K or of V
template <int D>
constexpr int tc2_smem_bytes_q8() { static_assert(kPageCap % 32 == 0, "128-byte aligned slots"); return tc2_smem_bytes<D>() + (kRawV - kRawVInStage) * tc2_half_rec<D>() + (kRawK + kRawV + 2) * 8; }

template <int D, bool BF16, bool Q8>
__global__ void __launch_bounds__(Q8 ? kThreads2Q8 : kThreads2) chunk_tc2_kernel(const __grid_constant__ CUtensorMap tmap32, const __grid_constant__ CUtensorMap tmap_sc, const ChunkArgs a) {
    static_assert(D == 128, "two-tile kernel: head_dim 128");
    constexpr uint32_t TILE = 128u * D * 2u;   // one Q tile
    constexpr uint32_t BLK = 128u * 128u;      // 64-column block of a Q tile
    constexpr int XB = D / 64, NV = Q8 ? 1 : 2;  // column blocks of a row, V buffers
    constexpr uint32_t KVB = 128u * D * 2u;    // a K or V buffer
    constexpr uint32_t PGB = 16u * D * 2u;     // a page in it
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;                 // Q_A then Q_B
    uint8_t* sKV = sQ + 2 * TILE;       // two K buffers, two V buffers: [page][8-token group][column block][8 rows of 128 bytes]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + 4 * KVB);
    const uint32_t b_k_full = smem_u32(bars + 0), b_k_empty = smem_u32(bars + 2), b_v_full = smem_u32(bars + 4), b_v_empty = smem_u32(bars + 6);
    const uint32_t b_s_full = smem_u32(bars + 8), b_p_full = smem_u32(bars + 10) /* [tile][half of the keys] */, b_o_done = smem_u32(bars + 14);
    const uint32_t b_q_full = smem_u32(bars + 16);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
    volatile int* failed = reinterpret_cast<volatile int*>(bars + 18);  // and the ticket
    int* s_asked = reinterpret_cast<int*>(bars + 19);  // K and V buffers whose copies have been announced (float layers)
    const uint32_t b_drain = smem_u32(bars + 20);
    int* s_pages = reinterpret_cast<int*>(bars + 32);
    float* s_xch = reinterpret_cast<float*>(s_pages + kPageCap);  // [2 buffers][2 tiles][128 rows][2 halves]
    // Q8 layout of the stage area: K buffers [0, 64 KB), V buffer [64, 96 KB), raw K ring and the first raw V
    // slots [96, 128 KB); the other raw V slots and the Q8 barriers follow the exchange area.  A K or V buffer
    // is [64-column block][page][8-token group][8 rows of 128 bytes], 128-byte swizzle.
    constexpr uint32_t REC = 2u * 16u * D + 2u * 16u * (D / 32) * 2u;  // an int8 record
    constexpr uint32_t HALF = 16u * D + 16u * (D / 32) * 2u;              // a record's K or V values with their scales
    static_assert(HALF == (uint32_t)(REC / 2), "half a record");
    constexpr uint32_t QBUF = 128u * D * 2u, QBLK = QBUF / 2;          // one K or V buffer, one 64-column block of it
    static_assert(!Q8 || kRawK * HALF + kRawVInStage * HALF <= 4 * KVB - 3 * QBUF, "raw rings in the freed quarter");
    uint8_t* sRawK = sKV + 3 * QBUF;
    uint8_t* sRawV0 = sRawK + kRawK * HALF;
    uint8_t* sRawV1 = reinterpret_cast<uint8_t*>(s_xch + 2 * 2 * 128 * 2);  // 128-byte aligned, as every slot is
    const uint32_t b_q8 = smem_u32(sRawV1 + (kRawV - kRawVInStage) * HALF);
    const uint32_t b_rawk = b_q8, b_rawv = b_rawk + kRawK * 8;
    (void)sRawK; (void)sRawV0; (void)sRawV1; (void)b_rawk; (void)b_rawv; (void)REC;

    const long long t_entry = TC_NOW();
    (void)t_entry;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if ((smem_u32(smem) & 1023u) != 0) {
        if (tid == 0) atomicOr(a.status, ST_SMEM_ALIGN);
        return;
    }
    // ---- which (sequence, kv head, pair of query tiles), which slice of its K/V tiles
    const CtaWork wk = load_work(a);
    const SeqMeta sm = wk.sm;
    const int Hkv = a.geo.n_kv, n_rep = a.geo.n_rep, RS = a.rep_slots, TPT = 128 / RS, h = wk.h;
    const int r0 = wk.qt * 2 * TPT;                               // first new token of tile A
    const int q_first = sm.pos + r0, q_last = sm.pos + min(r0 + 2 * TPT, sm.snew) - 1;
    // With no more tokens than one tile holds (verifying a draft, the decoding sequences of a mixed step), tile B is
    // left out altogether: the chain of one tile is then shorter than the time its K/V takes to arrive.
    const bool two = sm.snew - r0 > TPT;
    const int lo_key = a.window > 0 ? max(0, q_first - a.window + 1) : 0;
    const int p_lo = (lo_key >> 4) + 8 * wk.t0, p_hi = min(q_last >> 4, (lo_key >> 4) + 8 * wk.t1 - 1);
    const int n_tiles = wk.t1 - wk.t0;
    const int k0 = p_lo * 16;

    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            mbar_init(b_k_full + i * 8, 1); mbar_init(b_k_empty + i * 8, 1); mbar_init(b_v_full + i * 8, 1); mbar_init(b_v_empty + i * 8, 1);
            mbar_init(b_s_full + i * 8, 1); mbar_init(b_p_full + i * 16, 8); mbar_init(b_p_full + i * 16 + 8, 8); mbar_init(b_o_done + i * 8, 1);
        }
        mbar_init(b_q_full, 16);
        mbar_init(b_drain, 1);
        if constexpr (Q8)
            for (int i = 0; i < kRawK + kRawV; i++) mbar_init(b_rawk + i * 8, 1);
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap32) : "memory");
        if constexpr (Q8) asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_sc) : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i <= p_hi - p_lo && i < kPageCap; i += (int)blockDim.x) s_pages[i] = a.step.tables[sm.tbl_off + p_lo + i];
    tc_fence_before();
    __syncthreads();  // barriers and block table are ready: the producer starts while the softmax warps bring Q
    tc_fence_after();
    // q, the pages and the partial-result buffers belong to earlier launches until here; everything above (barriers,
    // tensor memory, the work record and the block table, which came with the step's upload) runs under their tail
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    // ---- Q tiles: row m of tile X is q head (m / TPT) at token r0 + X TPT + m % TPT
    if (warp >= 2 && warp < 18) {
        const uint16_t* qbase = reinterpret_cast<const uint16_t*>(a.q) + (size_t)sm.tok_off * a.geo.n_q * D;
#pragma unroll
        for (int u = 0; u < 2 * (D / 32); u++) {  // all of a thread's copies are in flight together
            const int X = u / (D / 32), c = tid - 64 + (u - X * (D / 32)) * 512, m = c / (D / 8), j = c - m * (D / 8), rep = m / TPT, r = r0 + X * TPT + (m - rep * TPT);
            if (X == 1 && !two) break;
            const bool there = rep < n_rep && r < sm.snew;
            cp_async16(smem_u32(sQ) + X * TILE + (j >> 3) * BLK + m * 128u + (((j & 7) ^ (m & 7)) << 4),
                       there ? qbase + ((size_t)(h * n_rep + rep) * sm.snew + r) * D + j * 8 : qbase, there);
        }
        cp_async_wait_all();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(b_q_full);
    }

    if (Q8 && warp >= 18) {
        // ------------------------------------------------------------ int8 layer: warp 18 feeds K, warp 19 feeds V
        const bool is_v = warp == 19;
        const int n_slots = is_v ? kRawV : kRawK;
        const uint32_t b_raw = is_v ? b_rawv : b_rawk;
        auto slot_ptr = [&](int sl) -> uint8_t* {
            if (!is_v) return sRawK + sl * HALF;
            return sl < kRawVInStage ? sRawV0 + sl * HALF : sRawV1 + (sl - kRawVInStage) * HALF;
        };
        const int n_recs = 8 * n_tiles;
        // lane 0: the half-record of page n of the CTA's range into its slot (values, then scales behind them).
        // Two boxes of the layer's byte tensor maps (128-byte rows, REC / 128 rows per record: K values, V values,
        // one row of K scales, one of V scales); plain bulk copies of the same bytes cost the issuing thread about
        // a thousand cycles per record, tensor-map copies a few dozen.
        auto issue = [&](int n, int sl) {
            const int idx = min(n, p_hi - p_lo);  // pages past the end repeat the last one (masked)
            int phys = idx < kPageCap ? s_pages[idx] : a.step.tables[sm.tbl_off + p_lo + idx];
            if (phys < 0 || phys >= a.geo.num_pages) { atomicOr(a.status, ST_BAD_PAGE); phys = 0; }
            const int row0 = (phys * Hkv + h) * (int)(REC / 128u);
            const uint32_t dst = smem_u32(slot_ptr(sl)), bar = b_raw + sl * 8;
            mbar_expect_tx(bar, HALF);
            if (n >> 3 == a.fault_tile && blockIdx.x == 0) return;
            tma_load_2d(dst, &tmap32, 0, row0 + (is_v ? 16 : 0), bar);
            tma_load_2d(dst + 16u * D, &tmap_sc, 0, row0 + 32 + (is_v ? 1 : 0), bar);
        };
        // Lane l takes the 16-byte pieces l, l + 32, l + 64, l + 96 of a half-record's 2048 value bytes.
        // K: 16 consecutive d of token l / 8 + 4 i, one scale group.  V: 8 consecutive d of token pair
        // l / 16 + 2 i.  Both permutations of qrec_value_off repeat every eight tokens, so piece i + 2 lands
        // one 8-token group (1024 bytes) after piece i, and pieces i = 0, 1 differ by four rows.
        uint32_t src_sc, d0[2], d1[2];  // scale offset of piece 0; where the piece's two 16-byte results go (i even, i odd)
        if (!is_v) {
            const int s0 = lane >> 3, grp = ((lane & 7) >> 1) ^ (s0 & 3), j0 = grp * 32 + (lane & 1) * 16, cc = (j0 & 63) >> 3;
            src_sc = 16u * D + (uint32_t)(s0 * (D / 32) + grp) * 2u;  // + 4 i tokens = + 4 i (D / 32) * 2 bytes
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int row = s0 + 4 * e;
                const uint32_t base = (uint32_t)(j0 >> 6) * QBLK + (uint32_t)row * 128u;
                d0[e] = base + (uint32_t)((cc ^ row) << 4); d1[e] = base + (uint32_t)(((cc + 1) ^ row) << 4);
            }
        } else {
            const int p0 = lane >> 4, grp = ((lane & 15) >> 2) ^ (p0 & 1);
            src_sc = 16u * D + (uint32_t)(grp * 8 + p0) * 4u;          // + 2 i pairs = + 8 i bytes
#pragma unroll
            for (int e = 0; e < 2; e++) {  // pair p0 + 2 i: (pair >> 1) & 1 = i & 1
                const int chunk = (2 * (lane & 3)) ^ (4 * e), j0 = grp * 32 + chunk * 4, cc = (j0 & 63) >> 3;
                const int t0 = 2 * p0 + 4 * e, t1 = t0 + 1;            // rows inside the 8-token group
                const uint32_t base = (uint32_t)(j0 >> 6) * QBLK;
                d0[e] = base + (uint32_t)t0 * 128u + (uint32_t)((cc ^ t0) << 4); d1[e] = base + (uint32_t)t1 * 128u + (uint32_t)((cc ^ t1) << 4);
            }
        }
        int issued = 0;
        if (lane == 0)
            for (; issued < n_slots && issued < n_recs; issued++) issue(issued, issued);
        issued = __shfl_sync(0xffffffffu, issued, 0);
        bool ok = true;
        int n = 0, sl = 0, ph = 0;  // record, its slot, the slot's phase
        long long tprev = TC_NOW(), c_wait = 0, c_issue = 0, c_conv = 0, c_meet = 0;
#pragma unroll 1
        for (; n < n_recs; n++) {
            const int j = n >> 3, pg = n & 7;
            if (lane == 0) {
                if (pg == 0) {  // the buffer this tile goes to must have been read to the end
                    if (!is_v && j >= 2 && !mbar_wait_bounded(b_k_empty + (j & 1) * 8, ((j >> 1) - 1) & 1)) ok = false;
                    if (is_v && j >= 1 && !mbar_wait_bounded(b_v_empty, (j - 1) & 1)) ok = false;
                }
                if (ok && !mbar_wait_bounded(b_raw + sl * 8, ph)) ok = false;
                if (*failed) ok = false;
                if (!ok) { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                TC_ACC(c_wait);
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            const uint8_t* rp = slot_ptr(sl);
            uint8_t* out = sKV + (is_v ? 2 * QBUF : (uint32_t)(j & 1) * QBUF) + (uint32_t)pg * 2048u;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 raw = *reinterpret_cast<const uint4*>(rp + lane * 16 + i * 512);
                uint8_t* o = out + (i >> 1) * 1024;
                uint4 x, y;
                if (!is_v) {
                    const uint32_t sc = *reinterpret_cast<const uint16_t*>(rp + src_sc + i * (4 * (D / 32) * 2));
                    q8_unpack_k16<BF16>(raw, sc | (sc << 16), x, y);
                } else {
                    const uint32_t sc = *reinterpret_cast<const uint32_t*>(rp + src_sc + i * 8);
                    q8_unpack_v8x2<BF16>(raw, sc, x, y);
                }
                *reinterpret_cast<uint4*>(o + d0[i & 1]) = x;
                *reinterpret_cast<uint4*>(o + d1[i & 1]) = y;
            }
            // A finished tile goes to the tensor pipe's proxy.  The slot's next copy needs no fence: every lane's
            // loads from the slot have returned their values (the stores above used them) before the warp meets.
            if (lane == 0) TC_ACC(c_conv);
            if (pg == 7) fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                TC_ACC(c_meet);
                if (issued < n_recs) issue(issued, sl);
                if (pg == 7) mbar_arrive(is_v ? b_v_full : b_k_full + (j & 1) * 8);
                TC_ACC(c_issue);
            }
            if (issued < n_recs) issued++;
            if (++sl == n_slots) { sl = 0; ph ^= 1; }
        }
        // never leave with a copy in flight: the records n .. issued - 1 have been asked for and not taken
        if (lane == 0)
            for (; n < issued; n++) {
                if (!mbar_wait_bounded(b_raw + sl * 8, ph)) { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                if (++sl == n_slots) { sl = 0; ph ^= 1; }
            }
        TC_DUMP(if (tid == 18 * 32) { unsigned long long* b = a.dbg_buf + (size_t)blockIdx.x * 16; b[0] = c_wait; b[1] = c_issue + c_conv + c_meet; b[12] = c_conv; b[13] = c_meet; b[14] = c_issue; b[15] = n_tiles; });
        (void)c_wait; (void)c_issue; (void)c_conv; (void)c_meet; (void)tprev;
    } else if (!Q8 && warp == 0) {
        // ------------------------------------------------------------ TMA producer
        bool ok = true;
        int asked[2] = {0, 0};
        long long tprev = TC_NOW(), c_wait = 0, c_issue = 0;
#pragma unroll 1
        for (int j = 0; j < n_tiles && ok; j++) {
            const int st = j & 1;
            // pages past the last visible one repeat it: finite data that the causal mask hides
            int phys = 0;
            if (lane < 8) {
                const int idx = min(j * 8 + lane, p_hi - p_lo);
                phys = idx < kPageCap ? s_pages[idx] : a.step.tables[sm.tbl_off + p_lo + idx];
                if (phys < 0 || phys >= a.geo.num_pages) { atomicOr(a.status, ST_BAD_PAGE); phys = 0; }
            }
#pragma unroll
            for (int is_v = 0; is_v < 2 && ok; is_v++) {
                const uint32_t full = (is_v ? b_v_full : b_k_full) + st * 8, empty = (is_v ? b_v_empty : b_k_empty) + st * 8;
                if (lane == 0) {
                    if (j >= 2 && !mbar_wait_bounded(empty, ((j >> 1) - 1) & 1)) ok = false;
                    TC_ACC(c_wait);
                    if (*failed) ok = false;
                    if (ok) { mbar_expect_tx(full, KVB); asked[is_v]++; }
                    else { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (ok && lane < 8 && (j != a.fault_tile || blockIdx.x != 0)) tma_load_page(smem_u32(sKV + (2 * is_v + st) * KVB + lane * PGB), &tmap32, is_v, (phys * Hkv + h) * 2, full);
                if (lane == 0) TC_ACC(c_issue);
            }
        }
        if (lane == 0) { s_asked[0] = asked[0]; s_asked[1] = asked[1]; }
        TC_DUMP(if (lane == 0) { a.dbg_buf[(size_t)blockIdx.x * 16 + 0] = c_wait; a.dbg_buf[(size_t)blockIdx.x * 16 + 1] = c_issue; a.dbg_buf[(size_t)blockIdx.x * 16 + 15] = n_tiles; });
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        {
            const uint32_t id_qk = instr_desc(BF16, 128, 128, false);
            const uint32_t id_pv = instr_desc(BF16, 128, D, true);
            // 8-token groups of K and V, their 64-wide column blocks, and a page of V are this far apart in a buffer
            constexpr uint32_t GRP = Q8 ? 1024u : XB * 1024u, CBLK = Q8 ? QBLK : 1024u, VPAGE = Q8 ? 2048u : PGB;
            const uint64_t dq = smem_desc(smem_u32(sQ), 16, 1024), dk = smem_desc(smem_u32(sKV), 16, GRP);
            const uint64_t dv = smem_desc(smem_u32(sKV) + 2 * KVB, CBLK, GRP);
            const int last_x = two ? 1 : 0;
            auto wait = [&](uint32_t bar, int parity) -> bool { return __all_sync(0xffffffffu, mbar_wait_unless(bar, parity, failed)); };
            auto issue_qk = [&](int X, int j) {
                const uint64_t kst = (uint64_t)(((j & 1) * KVB) >> 4), qst = (uint64_t)((X * TILE) >> 4);
#pragma unroll
                for (int ks = 0; ks < D / 16; ks++) {
                    const uint64_t qoff = (uint64_t)(((ks >> 2) * BLK + (ks & 3) * 32) >> 4);
                    const uint64_t koff = (uint64_t)(((ks >> 2) * CBLK + (ks & 3) * 32) >> 4);
                    umma(tmem + X * 128, dq + qst + qoff, dk + kst + koff, id_qk, ks > 0);
                }
                umma_commit(b_s_full + X * 8);
                if (X == last_x) umma_commit(b_k_empty + (j & 1) * 8);  // all scores of this K buffer have been issued
            };
            long long tprev = TC_NOW(), c_wkv = 0, c_wp = 0, c_iss = 0, c_pv = 0;
            bool ok = wait(b_q_full, 0) && wait(b_k_full, 0);
            if (ok) { tc_fence_after(); issue_qk(0, 0); if (two) issue_qk(1, 0); }
#pragma unroll 1
            for (int j = 0; ok && j < n_tiles; j++) {
                TC_ACC(c_iss);
                const int vs = NV == 2 ? (j & 1) : 0;
                const uint64_t vst = (uint64_t)((vs * KVB) >> 4);
                ok = wait(b_v_full + vs * 8, NV == 2 ? (j >> 1) & 1 : j & 1);
                TC_ACC(c_wkv);
#pragma unroll
                for (int X = 0; X < 2; X++) {
                    if (X > last_x || !ok) break;
#pragma unroll
                    for (int half = 0; half < 2; half++) {  // P of the tile's first 64 keys, of the others
                        if (ok) ok = wait(b_p_full + X * 16 + half * 8, j & 1);
                        TC_ACC(c_wp);
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll
                        for (int ks = half * 4; ks < half * 4 + 4; ks++)  // 16 keys = one page per step; P: 8 packed columns per step
                            umma_ts(tmem + 256 + X * 128, tmem + X * 128 + ks * 8, dv + vst + (uint64_t)((ks * VPAGE) >> 4), id_pv, (j > 0 || ks > 0));
                        TC_ACC(c_pv);
                    }
                    if (!ok) break;
                    if (X == last_x) umma_commit(b_v_empty + vs * 8);  // every read of this V buffer has been issued
                    if (j + 1 == n_tiles) { umma_commit(b_o_done + X * 8); continue; }
                    if (X == 0) {
                        ok = wait(b_k_full + ((j + 1) & 1) * 8, ((j + 1) >> 1) & 1);
                        TC_ACC(c_wkv);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    issue_qk(X, j + 1);
                    TC_ACC(c_iss);
                }
            }
            if (!ok) {
                if (lane == 0) { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                umma_commit(b_drain);  // waited for below
            }
            (void)c_pv;
            TC_DUMP(if (lane == 0) { a.dbg_buf[(size_t)blockIdx.x * 16 + 2] = c_wkv; a.dbg_buf[(size_t)blockIdx.x * 16 + 3] = c_wp; a.dbg_buf[(size_t)blockIdx.x * 16 + 4] = c_iss;
                    a.dbg_buf[(size_t)blockIdx.x * 16 + 11] = c_pv; });
        }
    } else if (warp >= 2 && warp < (two ? 18 : 10)) {
        // ------------------------------------------------------------ softmax + epilogue of tile X, half H of the keys
        const int X = (warp - 2) >> 3, H = ((warp - 2) >> 2) & 1;
        const int lane_base = (warp & 3) * 32;  // the quarter of the tensor-memory lanes this warp may touch
        const int m = lane_base + lane;
        const int rep = m / TPT, r = r0 + X * TPT + (m - rep * TPT);
        const bool row_ok = rep < n_rep && r < sm.snew;
        const int q_pos = sm.pos + min(r, sm.snew - 1);
        const int qx_min = sm.pos + min(r0 + X * TPT, sm.snew - 1), qx_max = sm.pos + min(r0 + (X + 1) * TPT, sm.snew) - 1;
        const uint32_t lane_addr = (uint32_t)lane_base << 16;
        const uint32_t tS = tmem + X * 128 + lane_addr, tO = tmem + 256 + X * 128 + lane_addr;
        const int pair_bar = 1 + X * 4 + (warp & 3);  // named barrier of the two warps that share this quarter of tile X
        // A named barrier has no time limit, so the two warps of a pair must leave the loop in the same iteration.  Whether
        // one saw a wait run out travels with the pair's barrier: a flag in shared memory could be raised for the next tile
        // (once another role has given up, that wait ends at once) before the other has read it for this one, and two
        // flags in turn cost 0.4 to 1.2 % (26 sequences of a mixed step 4626 us, this way 4496; one flag 4586).
        float m_ref = -INFINITY, l_run = 0.f;  // l_run: this half's share of the row sum
        bool ok = true;
        long long tprev = TC_NOW(), c_ws = 0, c_ld = 0, c_exp = 0, c_wo = 0, c_st = 0;
        const long long tstart = tprev;
#pragma unroll 1
        for (int j = 0; j < n_tiles; j++) {
            ok = mbar_wait_unless(b_s_full + X * 8, j & 1, failed);
            ok = __all_sync(0xffffffffu, ok);
            TC_ACC(c_ws);
            tc_fence_after();  // (without the scores the loads below read stale columns: harmless, nothing is kept)
            // this thread's keys: 32 H .. 32 H + 31 of the tile's first 64 and of its last 64
            const int kbase = k0 + j * 128 + H * 32;
            const bool need_mask = (kbase + 95 > qx_min) || (a.window > 0 && kbase + a.window <= max(qx_max, qx_min));
            uint32_t sv[64];
            tmem_ld32x2(tS + H * 32, tS + 64 + H * 32, sv);
            if (need_mask) {
#pragma unroll
                for (int e = 0; e < 64; e++) {
                    const int kp = kbase + e + (e & 32);
                    if (!(kp <= q_pos && (a.window <= 0 || kp + a.window > q_pos))) sv[e] = 0xff800000u;  // -inf
                }
            }
            float mx = max_of(sv);
            // the other half's maximum (double-buffered by tile parity: the partner may still be reading the
            // previous tile's entry when this one is written only if it were two tiles behind, which the
            // barrier of the tile in between rules out)
            float* xrow = s_xch + (((j & 1) * 2 + X) * 128 + m) * 2;
            xrow[H] = mx;
            const bool gave_up = bar_any(pair_bar, 64, !ok);  // also: both warps have their S columns in registers, so P may overwrite them
            mx = fmaxf(mx, xrow[H ^ 1]) * a.scale_log2;
            if (gave_up) { ok = false; break; }  // both warps of the pair, in the same iteration
            TC_ACC(c_ld);
            float alpha = 1.f;
            if (mx > m_ref + 8.f || m_ref == -INFINITY) {  // both halves see the same mx: the same decision
                alpha = (m_ref == -INFINITY) ? 0.f : exp2f(m_ref - mx);
                m_ref = mx;
            }
            const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
            const uint64_t scale2 = f32x2(a.scale_log2, a.scale_log2), neg_ref2 = f32x2(-m_use, -m_use);
            uint64_t sum[2] = {0ull, 0ull};
            uint32_t pk[16];
            exp_pack<32, BF16>(sv, scale2, neg_ref2, sum, pk);
            tmem_st16(tS + H * 16, pk);  // P of keys 32 H .. : packed columns 16 H ..
            // S_X being full means P V_X of the previous tile has completed (the tensor pipe runs in
            // order), so O_X may be rescaled now: this warp takes the O columns 64 H .. 64 H + 63
            if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
                for (int c = 0; c < 2; c++) {
                    uint32_t ov[32];
                    tmem_ld32(tO + H * 64 + c * 32, ov);
#pragma unroll
                    for (int e = 0; e < 32; e++) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * alpha);
                    tmem_st32(tO + H * 64 + c * 32, ov);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(b_p_full + X * 16);  // P V of the first 64 keys runs under the others' exponentials
            TC_ACC(c_exp);
            exp_pack<32, BF16>(sv + 32, scale2, neg_ref2, sum, pk);
            tmem_st16(tS + 32 + H * 16, pk);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            l_run = l_run * alpha + sum_of(sum);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(b_p_full + X * 16 + 8);
            TC_ACC(c_st);
        }
        TC_DUMP(if (tid == 64) {
            unsigned long long* b = a.dbg_buf + (size_t)blockIdx.x * 16;
            b[5] = c_ws; b[6] = c_ld; b[7] = c_exp; b[8] = c_wo; b[9] = c_st; b[10] = TC_NOW() - tstart;
            if (!Q8) { b[12] = 0x7c2; b[13] = tstart - t_entry; }  // float layer: cycles in front of the softmax loop
        });
        const long long t_loop_end = TC_NOW();
        (void)tstart; (void)c_wo; (void)t_loop_end;
        if (ok) ok = mbar_wait_bounded(b_o_done + X * 8, 0) && !*failed;
        ok = __all_sync(0xffffffffu, ok);
        // the row sum is the two halves' sums (exchanged whether or not the wait succeeded: the pair must
        // meet at its barrier the same number of times)
        float* xrow = s_xch + ((n_tiles & 1) * 2 + X) * 256 + m * 2;
        xrow[H] = l_run;
        bar_sync(pair_bar, 64);
        const float l_row = l_run + xrow[H ^ 1];
        if (!ok && lane == 0) {
            *failed = 1;
            atomicOr(a.status, ST_WAIT_TIMEOUT);
        }
        uint16_t* orow = reinterpret_cast<uint16_t*>(a.out) +
                         ((size_t)sm.tok_off * a.geo.n_q + (size_t)(h * n_rep + (row_ok ? rep : 0)) * sm.snew + (row_ok ? r : 0)) * D;
        if (wk.parts == 1) {
            if (ok) {
                tc_fence_after();
                const float inv = 1.f / l_row;
#pragma unroll 1
                for (int c = 2 * H; c < 2 * H + 2; c++) {  // this warp writes the output columns 64 H .. 64 H + 63
                    uint32_t v[32];
                    tmem_ld32(tO + c * 32, v);
                    float f[32];
#pragma unroll
                    for (int e = 0; e < 32; e++) f[e] = __uint_as_float(v[e]);
                    if (row_ok) store_row32<BF16>(orow + c * 32, f, inv);
                }
            }
        } else {
            // ---- a slice of a cut item: un-normalised rows and their (reference exponent, sum) go to memory, the
            // CTA draws a ticket, and the CTA that draws the item's last one adds the slices up.  No CTA waits
            // for another; every softmax warp passes both barriers whatever happened to its waits.
            const int slot = wk.slot_base + wk.part;
            const int nv = min(TPT, sm.snew - r0 - X * TPT), prow = rep * nv + (m - rep * TPT);
            if (ok) {
                tc_fence_after();
                float4* rows = slice_rows<D>(a, slot, 2, X) + prow;
#pragma unroll 1
                for (int c = 2 * H; c < 2 * H + 2; c++) {
                    uint32_t v[32];
                    tmem_ld32(tO + c * 32, v);
                    if (row_ok) {
#pragma unroll
                        for (int u = 0; u < 8; u++)
                            rows[(size_t)(c * 8 + u) * 128] = make_float4(__uint_as_float(v[u * 4]), __uint_as_float(v[u * 4 + 1]),
                                                                          __uint_as_float(v[u * 4 + 2]), __uint_as_float(v[u * 4 + 3]));
                    }
                }
                if (H == 0 && row_ok) a.split_ml[((size_t)slot * 2 + X) * 128 + prow] = make_float2(m_ref, l_row);
            }
            int* s_ticket = reinterpret_cast<int*>(const_cast<int*>(failed)) + 1;
            if (last_slice(a, wk, 9, two ? 512 : 256, tid == 64, s_ticket) && !*failed)
                merge_slices<D, BF16>(a, wk, 2, X, nv, r0 + X * TPT, (tid - 64) & 255, 256);
        }
        TC_DUMP(if (tid == 64 && !Q8) { a.dbg_buf[(size_t)blockIdx.x * 16 + 14] = TC_NOW() - t_loop_end; });
    }
    tc_fence_before();
    __syncthreads();
    // never leave with a product or a copy in flight if somebody gave up (as above)
    if (tid == 0 && *failed) {
        mbar_wait_bounded(b_drain, 0);
        for (int is_v = 0; is_v < 2 && !Q8; is_v++)
            for (int i = max(0, s_asked[is_v] - 2); i < s_asked[is_v]; i++) mbar_wait_bounded((is_v ? b_v_full : b_k_full) + (i & 1) * 8, (i >> 1) & 1);
    }
    __syncwarp();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

template <bool BF16>
static cudaError_t launch_tc2(const CUtensorMap& map32, const CUtensorMap& map_sc, const ChunkArgs& a, bool overlap, cudaStream_t st) {
    if (a.n_items <= 0) return cudaSuccess;
    if (a.q8_arena) return launch_pdl(overlap, chunk_tc2_kernel<128, BF16, true>, a.n_items, kThreads2Q8, tc2_smem_bytes_q8<128>(), st, map32, map_sc, a);
    return launch_pdl(overlap, chunk_tc2_kernel<128, BF16, false>, a.n_items, kThreads2, tc2_smem_bytes<128>(), st, map32, map_sc, a);
}

bool chunk_tc2_supported(int d) { return d == 128; }

// Two query tiles per CTA (head_dim 128): the work list has one item per pair of tiles.
cudaError_t launch_chunk_tc2(const CUtensorMap& map32, const CUtensorMap& map_sc, const ChunkArgs& a, bool bf16, bool overlap, cudaStream_t st) {
    if (a.geo.d != 128) return cudaErrorInvalidValue;
    return bf16 ? launch_tc2<true>(map32, map_sc, a, overlap, st) : launch_tc2<false>(map32, map_sc, a, overlap, st);
}

bool chunk_tc_supported(int d) { return d == 64 || d == 128 || d == 256; }

cudaError_t chunk_tc_init() {
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(chunk_tc_kernel<64, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem_bytes<64>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_tc_kernel<64, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem_bytes<64>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_tc_kernel<128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem_bytes<128>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_tc_kernel<128, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem_bytes<128>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_tc_kernel<256, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem_bytes<256>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_tc_kernel<256, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem_bytes<256>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_tc2_kernel<128, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc2_smem_bytes<128>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_tc2_kernel<128, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc2_smem_bytes<128>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_tc2_kernel<128, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc2_smem_bytes_q8<128>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_tc2_kernel<128, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc2_smem_bytes_q8<128>())) != cudaSuccess) return e;
    return cudaSuccess;
}

// `map`: the layer's map_page (K or V of a page per copy).
cudaError_t launch_chunk_tc(const CUtensorMap& map, const ChunkArgs& a, bool bf16, bool overlap, cudaStream_t st) {
    switch (a.geo.d) {
        case 64: return bf16 ? launch_tc<64, true>(map, a, overlap, st) : launch_tc<64, false>(map, a, overlap, st);
        case 128: return bf16 ? launch_tc<128, true>(map, a, overlap, st) : launch_tc<128, false>(map, a, overlap, st);
        case 256: return bf16 ? launch_tc<256, true>(map, a, overlap, st) : launch_tc<256, false>(map, a, overlap, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace cbkv
