// Chunk (prefill) attention on pairs of SMs: the one-tile kernel of prefill_tc.cu with cta_group::2.
// Reference math: attend() with seq > 1, kv.rs:243-268.
//
// What bounds the one-SM kernels: an MMA of 16 deep takes the tensor pipe 64 cycles at N = 128, 128 at N = 256, and hardly
// less than 50 with a smaller N (measured, back to back, either cta_group, A in shared or tensor memory); and shared
// memory delivers 128 bytes a cycle, which two query tiles of head_dim 128 use up (128-row Q and 128 keys per MMA, and the
// copies), while at head_dim 256 K, V and Q leave room for KV tiles of 64 keys only, at that price.  A pair of CTAs,
// one query tile each, runs M = 256 MMAs for which each CTA holds half of K and half of V: half of the operand bytes, half
// of the L2 reads per query tile, and KV tiles of 128 keys at both head_dims.
//
// A cluster of two CTAs = one (sequence, kv head, two tiles of query tokens); rank 0 and rank 1 take a tile each.  Row
// m = rep * TPT + i of a tile is q head `rep` of the kv group at the tile's i-th token.  KV tiles of KT tokens:
//   K: rank r holds keys [r KT / 2, (r + 1) KT / 2) of the tile, all of head_dim
//   V: rank r holds all keys, columns [r D / 2, (r + 1) D / 2)
//
//   warp 0        TMA producer of this CTA's halves; the bytes of both CTAs are counted by rank 0's barriers
//   warp 1        rank 0 only: one thread issues tcgen05.mma for the pair: S = Q K^T (two S buffers), O += P V
//   warps 2..9    softmax of the even KV tiles (S buffer 0)       warps 10..17  of the odd ones (S buffer 1)
//
// With eight warps the exponentials of a tile would wait for its scores' load and maximum; with sixteen, two tiles are in
// work, and the special function unit (1024 cycles for the 128 x 128 exponentials of a tile) has something to do nearly
// always.  Two threads share a row, one for each half of a tile's keys.  The reference exponent of a row passes from tile
// to tile through shared memory: it needs a tile's maximum only, not its exponentials.
//
// Tensor memory: S0 [0,128), S1 [128,256); head_dim 128: P0 [256,320), P1 [320,384), O [384,512), so that S is free for the
// scores after next as soon as it is in registers; head_dim 256: O [256,512), P over the first half of its S.
#include <algorithm>

#include "kernels.hpp"
#include "pdl.cuh"
#include "tc.cuh"

namespace cbkv {

namespace {

constexpr int kPairThreads = 576;
constexpr int kPairKeys = 128;  // tokens per KV tile
template <int D>
struct PairBufs { static constexpr int value = D == 256 ? 2 : 5; };  // K buffers and V buffers (32 or 16 KB each)
constexpr int kPairBufs = 5;

// barriers, each 8 bytes
constexpr int kBKFull = 0, kBVFull = kBKFull + kPairBufs, kBKEmpty = kBVFull + kPairBufs, kBVEmpty = kBKEmpty + kPairBufs;
constexpr int kBSFull = kBVEmpty + kPairBufs, kBPFull = kBSFull + 2, kBODone = kBPFull + 2, kBQFull = kBODone + 2;
constexpr int kPairWords = 4 + 8;  // 8-byte words after the barriers: tensor memory, failed, ticket, the issuer's last barrier, then the 16 flags of the pairs of warps
constexpr int kBSFree = kBQFull + 1, kBRef = kBSFree + 2 /* [2 buffers][4 quarters] */, kBCount = kBRef + 8;

template <int D>
constexpr int pair_smem_bytes() {
    return 128 * D * 2 /* Q */ + 2 * PairBufs<D>::value * (kPairKeys / 2) * D * 2 + (kBCount + kPairWords) * 8 + kPageCap * 4 +
           (2 * 2 * 2 * 128 /* half-row maxima */ + 2 * 128 /* reference exponents */ + 4 * 128 /* row sums */) * 4;
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t at_rank0(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
// Only tensor memory passes between the CTAs through these barriers (P and O stored, S loaded by the threads that arrive;
// the MMAs issued behind the wait).  The memory model's release and acquire are about generic memory; tensor-memory
// operations are ordered by tcgen05.fence::before_thread_sync and ::after_thread_sync around whatever orders the
// execution of the two threads (PTX, tcgen05 memory consistency), and an arrival that a wait has observed does that in
// any scope.  A cluster-scope release and acquire would cost every tile a memory barrier: a launch at head_dim 128 took 786
// us with them, 620 without.
__device__ __forceinline__ void arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// the same with cluster scope, for Q, which the threads write to shared memory
__device__ __forceinline__ void arrive_cluster_release(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ uint32_t test_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
// K or V of one page of one kv head, from column block x on; the bytes are counted by a barrier of rank 0
__device__ __forceinline__ void load_page_pair(uint32_t dst, const CUtensorMap* map, int x, int is_v, int row16, uint32_t bar_rank0) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(0), "r"(x), "r"(is_v), "r"(row16), "r"(bar_rank0) : "memory");
}
__device__ __forceinline__ void umma_pair_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier at this offset in both CTAs when everything issued before is complete
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// the same on this CTA's barrier alone
__device__ __forceinline__ void commit_own(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}

}  // namespace

template <int D, bool BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads) chunk_pair_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const ChunkArgs a) {
    constexpr int KT = kPairKeys;              // tokens per KV tile
    constexpr int HK = KT / 2;                 // keys of a softmax thread, and of this CTA's half of K
    constexpr int PPT = KT / 16;               // pages per KV tile
    constexpr int XB = D / 64, XBV = D / 128;  // 64-wide column blocks of K rows, of this CTA's half of V rows
    constexpr uint32_t HALF = (uint32_t)HK * D * 2u;                  // a K or V buffer
    constexpr uint32_t PGK = 16u * D * 2u, PGV = 16u * D;             // a page in it
    constexpr int NB = PairBufs<D>::value;
    constexpr bool OWN_P = D == 128;           // P in columns of its own
    constexpr uint32_t QBLK = 128u * 128u;     // 64-column block of the Q tile
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;                 // [64-column block][128 rows of 128 bytes], 128-byte swizzle
    uint8_t* sK = sQ + 128 * D * 2;     // [page][8-token group][column block][8 rows of 128 bytes]
    uint8_t* sV = sK + NB * HALF;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + NB * HALF);
    auto bar = [&](int i) -> uint32_t { return smem_u32(bars + i); };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBCount);
    volatile int* failed = reinterpret_cast<volatile int*>(bars + kBCount + 1);
    int* s_ticket = reinterpret_cast<int*>(bars + kBCount + 2);
    const uint32_t b_drain = bar(kBCount + 3);
    int* s_pair = reinterpret_cast<int*>(bars + kBCount + 4);      // [8 pairs of warps][parity of the group's tile] a wait ran out
    int* s_pages = reinterpret_cast<int*>(bars + kBCount + kPairWords);  // [kPageCap] physical pages of the KV range
    float* s_xch = reinterpret_cast<float*>(s_pages + kPageCap);   // [S buffer][parity of the group's tile][128 rows][2 halves]
    float* s_ref = s_xch + 2 * 2 * 2 * 128;                        // [S buffer][128 rows]
    float* s_sum = s_ref + 2 * 128;                                // [group][half][128 rows]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_rank();
    if ((smem_u32(smem) & 1023u) != 0) {  // the same in both CTAs
        if (tid == 0) atomicOr(a.status, ST_SMEM_ALIGN);
        return;
    }
    // ---- which (sequence, kv head, pair of query tiles), which slice of its K/V tiles
    CtaWork wk;
    {
        const int4* p = reinterpret_cast<const int4*>(a.tiles + (blockIdx.x >> 1));
        const int4 x = __ldg(p), y = __ldg(p + 1);
        wk.seq = x.x; wk.h = x.y; wk.qt = x.z; wk.t0 = x.w;
        wk.t1 = y.x; wk.part = y.y & 0xffff; wk.parts = y.y >> 16; wk.slot_base = y.z;
        wk.cut = 2 * y.w + rank;  // each tile's slices are added up on their own
        wk.sm = a.step.seq_meta[wk.seq];
    }
    const SeqMeta sm = wk.sm;
    const int Hkv = a.geo.n_kv, n_rep = a.geo.n_rep, RS = a.rep_slots, TPT = 128 / RS, h = wk.h;
    const int ri = wk.qt * 2 * TPT;                                   // first new token of the pair
    const int r0 = ri + rank * TPT;                                   // of this CTA's tile
    const int nv = max(0, min(TPT, sm.snew - r0));                    // tokens of it (rank 1 may have none)
    const int q_first = sm.pos + ri, q_last = sm.pos + min(ri + 2 * TPT, sm.snew) - 1;
    const int q_min = min(sm.pos + r0, q_last), q_max = max(q_min, sm.pos + r0 + nv - 1);
    const int lo_key = a.window > 0 ? max(0, q_first - a.window + 1) : 0;
    const int p_lo = (lo_key >> 4) + wk.t0 * PPT, p_hi = min(q_last >> 4, (lo_key >> 4) + wk.t1 * PPT - 1);
    const int n_tiles = wk.t1 - wk.t0;
    const int k0 = p_lo * 16;                                         // absolute position of key 0 of tile 0

    if (tid == 0) {
        for (int i = 0; i < NB; i++) {
            mbar_init(bar(kBKFull + i), 1); mbar_init(bar(kBVFull + i), 1); mbar_init(bar(kBKEmpty + i), 1); mbar_init(bar(kBVEmpty + i), 1);
        }
        for (int i = 0; i < 2; i++) { mbar_init(bar(kBSFull + i), 1); mbar_init(bar(kBPFull + i), 16); mbar_init(bar(kBODone + i), 1); }
        mbar_init(bar(kBQFull), 32);
        for (int i = 0; i < 2; i++) mbar_init(bar(kBSFree + i), 16);
        for (int i = 0; i < 8; i++) mbar_init(bar(kBRef + i), 1);
        mbar_init(b_drain, 1);
        *failed = 0;
        for (int i = 0; i < 16; i++) s_pair[i] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_k) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_v) : "memory");
    }
    if (warp == 0) {  // tensor memory of both CTAs
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i <= p_hi - p_lo && i < kPageCap; i += kPairThreads) s_pages[i] = a.step.tables[sm.tbl_off + p_lo + i];
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers and tensor memory are there
    tc_fence_after();
    // q, the pages and the partial-result buffers belong to earlier launches until here; everything above runs under their tail
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t tS0 = tmem, tP0 = OWN_P ? tmem + 2 * KT : tmem, tO = tmem + 512 - D;
    constexpr uint32_t PSTRIDE = OWN_P ? KT / 2 : KT;
    static_assert(2 * KT + (OWN_P ? KT : 0) + D <= 512, "tensor memory");

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        bool ok = true;
        const int withheld = blockIdx.x == 0 ? a.fault_tile : -1;  // announced and not made
        int asked[2] = {0, 0};  // K and V buffers that this CTA has asked copies for
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
                const uint32_t full = bar((is_v ? kBVFull : kBKFull) + st), empty = bar((is_v ? kBVEmpty : kBKEmpty) + st);
                if (lane == 0) {
                    if (j >= NB && !mbar_wait_bounded(empty, (j / NB - 1) & 1)) ok = false;
                    if (*failed) ok = false;
                    if (!ok) { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                    else if (rank == 0) mbar_expect_tx(full, 2 * HALF);  // this CTA's copies and the other's
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (!ok) break;
                asked[is_v]++;
                const uint32_t full0 = at_rank0(full);
                if (is_v) {
                    if (lane < PPT && j != withheld) load_page_pair(smem_u32(sV + st * HALF) + lane * PGV, &tmap_v, rank * XBV, 1, (phys * Hkv + h) * 2, full0);
                } else if (lane >= rank * (PPT / 2) && lane < (rank + 1) * (PPT / 2) && j != withheld) {
                    load_page_pair(smem_u32(sK + st * HALF) + (lane - rank * (PPT / 2)) * PGK, &tmap_k, 0, 0, (phys * Hkv + h) * 2, full0);
                }
            }
        }
        // Leave last: every buffer's final use is over, so no copy and no arrival is on its way to this CTA any more.  If
        // somebody gave up that use may never come; the wait for it is then a hundred milliseconds in which the copies land.
#pragma unroll
        for (int is_v = 0; is_v < 2; is_v++)
            for (int i = max(0, asked[is_v] - NB) + lane; i < asked[is_v]; i += 32)
                if (!mbar_wait_bounded(bar((is_v ? kBVEmpty : kBKEmpty) + i % NB), (i / NB) & 1)) ok = false;
        if (!ok) { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (rank == 0) {
            const uint32_t id_qk = instr_desc(BF16, 256, KT, false);
            const uint32_t id_pv = instr_desc(BF16, 256, D, true);
            const uint64_t dq = smem_desc(smem_u32(sQ), 16, 1024), dk = smem_desc(smem_u32(sK), 16, XB * 1024), dv = smem_desc(smem_u32(sV), 1024, XBV * 1024);
            bool ok = true;
            // until f() holds, within the limit
            auto wait_for = [&](auto&& f) {
                uint64_t t0 = 0;
                for (int n = 0; ok; n++) {
                    if (__all_sync(0xffffffffu, f())) return;
                    if ((n & 63) == 63) {
                        if (*failed) ok = false;
                        if (t0 == 0) t0 = global_ns();
                        else if (global_ns() - t0 > 200000000ull) ok = false;
                        ok = __all_sync(0xffffffffu, ok);
                    }
                }
            };
            auto issue_qk = [&](int j) {
                const uint64_t kst = (uint64_t)((uint32_t)(j % NB) * HALF >> 4);
                tc_fence_after();
#pragma unroll
                for (int ks = 0; ks < D / 16; ks++)  // 16 elements = 32 bytes inside the swizzled row, four steps per 64-column block
                    umma_pair_ss(tS0 + (j & 1) * KT, dq + (uint64_t)(((ks >> 2) * QBLK + (ks & 3) * 32) >> 4), dk + kst + (uint64_t)(((ks >> 2) * 1024 + (ks & 3) * 32) >> 4), id_qk, ks > 0);
                commit_pair(bar(kBSFull + (j & 1)));
                commit_pair(bar(kBKEmpty + j % NB));
            };
            wait_for([&] { return test_wait_cluster(bar(kBQFull), 0) != 0; });
            int next_qk = 0;  // scores issued so far
#pragma unroll 1
            for (int j = 0; ok && j < n_tiles; j++) {
                // Until this tile's P is there: the scores of the next tiles as soon as their K has landed and their S buffer
                // is free: in both CTAs' registers, or, with P over it, read by a P V issued before.
                wait_for([&] {
                    if (next_qk < n_tiles && next_qk <= j + (OWN_P ? 2 : 1) &&
                        __all_sync(0xffffffffu, (!OWN_P || next_qk < 2 || mbar_test_wait(bar(kBSFree + (next_qk & 1)), ((next_qk - 2) >> 1) & 1)) &&
                        mbar_test_wait(bar(kBKFull + next_qk % NB), (next_qk / NB) & 1)))
                        issue_qk(next_qk++);
                    return next_qk > j && mbar_test_wait(bar(kBPFull + (j & 1)), (j >> 1) & 1);
                });
                const int st = j % NB;
                if (ok) wait_for([&] { return mbar_test_wait(bar(kBVFull + st), (j / NB) & 1) != 0; });
                if (!ok) break;
                tc_fence_after();
                const uint64_t vst = (uint64_t)((st * HALF) >> 4);
#pragma unroll
                for (int ks = 0; ks < PPT; ks++)  // 16 keys per step = one page; P: 8 packed columns, V: MN-major
                    umma_pair(tO, tP0 + (j & 1) * PSTRIDE + ks * 8, dv + vst + (uint64_t)((ks * PGV) >> 4), id_pv, (j > 0 || ks > 0));
                commit_pair(bar(kBVEmpty + st));
                commit_pair(bar(kBODone + (j & 1)));
            }
            if (!ok) {  // what has been issued ends before the tensor memory is given back
                if (lane == 0) { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                commit_own(b_drain);
                mbar_wait_bounded(b_drain, 0);
            }
        }
    } else {
        // ------------------------------------------------------------ softmax + epilogue
        const int sw = warp - 2, X = sw >> 3, H = (sw >> 2) & 1, quarter = warp & 3;  // group (S buffer), half of the keys
        const int m = quarter * 32 + lane;                 // row of the tile, TMEM lane
        const int rep = m / TPT, i = m - rep * TPT;
        const bool row_ok = rep < n_rep && i < nv;
        const int q_pos = min(q_min + i, q_max);           // rows past the data mimic the last token
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        const int pair_id = X * 4 + quarter;               // the two warps with the same rows and tiles
        // ---- Q to shared memory, rows past the data are zero
        {
            const uint16_t* qbase = reinterpret_cast<const uint16_t*>(a.q) + (size_t)sm.tok_off * a.geo.n_q * D;
#pragma unroll
            for (int u = 0; u < D / 32; u++) {  // all of a thread's copies are in flight together
                const int c = tid - 64 + u * 512, mm = c / (D / 8), jj = c - mm * (D / 8), rr = mm / TPT, ii = mm - rr * TPT;
                const bool there = rr < n_rep && ii < nv;
                cp_async16(smem_u32(sQ) + (jj >> 3) * QBLK + mm * 128u + (((jj & 7) ^ (mm & 7)) << 4),
                           there ? qbase + ((size_t)(h * n_rep + rr) * sm.snew + r0 + ii) * D + jj * 8 : qbase, there);
            }
            cp_async_wait_all();
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) arrive_cluster_release(at_rank0(bar(kBQFull)));
        }
        // A named barrier has no time limit, so the two warps of a pair must leave the loop in the same
        // iteration: whichever sees a wait run out says so before the pair's barrier, both read it after.  Flags and
        // half-row maxima have two places each, taken in turn: a warp may pass the barrier, and with P in columns of its
        // own find its next scores there and write again, before the other has read what it wrote for this tile.  It
        // cannot come back to the same place without the barrier in between, which the other reaches after that read.
        const uint32_t tS = tS0 + X * KT + lane_addr, tP = tP0 + X * PSTRIDE + lane_addr;
        const uint32_t p_full0 = at_rank0(bar(kBPFull + X)), s_free0 = at_rank0(bar(kBSFree + X));
        // Exponents are taken against a reference that is only moved when a row's maximum exceeds it by more than 8 (a
        // factor 256): probabilities then stay below 256, exact enough in f16/bf16 with f32 sums, and O is rescaled rarely.
        float m_own = -INFINITY, l_run = 0.f;              // reference of this thread's last tile, its share of the row sum against that
        bool ok = true;
#pragma unroll 1
        for (int j = X; j < n_tiles; j += 2) {
            ok = mbar_wait_unless(bar(kBSFull + X), (j >> 1) & 1, failed);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            const int kbase = k0 + j * KT + H * HK;
            const bool need_mask = (kbase + HK - 1 > q_min) || (a.window > 0 && kbase + a.window <= q_max);
            uint32_t sv[HK];
            tmem_ld_row<HK>(tS + H * HK, sv);
            if constexpr (OWN_P) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_cluster(s_free0);
            }
            if (need_mask) {
#pragma unroll
                for (int e = 0; e < HK; e++) {
                    const int kp = kbase + e;
                    if (!(kp <= q_pos && (a.window <= 0 || kp + a.window > q_pos))) sv[e] = 0xff800000u;  // -inf
                }
            }
            float mx = max_of(sv);
            const int turn = (j >> 1) & 1;
            volatile int* pair_failed = s_pair + pair_id * 2 + turn;
            float* xrow = s_xch + ((X * 2 + turn) * 128 + m) * 2;
            xrow[H] = mx;
            // the reference that the tile before left; read before the pair's barrier, after which its place may be reused
            float m_ref = -INFINITY;
            if (j > 0) {
                if (ok) ok = mbar_wait_bounded(bar(kBRef + (X ^ 1) * 4 + quarter), ((j - 1) >> 1) & 1);
                ok = __all_sync(0xffffffffu, ok);
                m_ref = s_ref[(X ^ 1) * 128 + m];
            }
            if (!ok && lane == 0) *pair_failed = 1;
            bar_sync(1 + pair_id, 64);  // also: both warps have their S columns in registers, where P may overwrite them
            mx = fmaxf(mx, xrow[H ^ 1]) * a.scale_log2;  // scale > 0: the maximum commutes with the scaling
            if (*pair_failed) { ok = false; break; }     // both warps of the pair, in the same iteration
            float alpha = 1.f;
            if (mx > m_ref + 8.f || (m_ref == -INFINITY && mx > -INFINITY)) {  // both halves see the same values: the same decision
                if (m_ref != -INFINITY) alpha = exp2f(m_ref - mx);  // else O holds zeros for this row
                m_ref = mx;
            }
            if (H == 0) {
                s_ref[X * 128 + m] = m_ref;
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(kBRef + X * 4 + quarter));
            }
            const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
            float sum = 0.f, sum2 = 0.f;
#pragma unroll
            for (int e = 0; e < HK; e += 2) {
                const float p0 = ex2_approx(fmaf(__uint_as_float(sv[e]), a.scale_log2, -m_use));
                const float p1 = ex2_approx(fmaf(__uint_as_float(sv[e + 1]), a.scale_log2, -m_use));
                if (e & 2) sum2 += p0 + p1; else sum += p0 + p1;  // two chains
                sv[e >> 1] = pack2<BF16>(p0, p1);  // P pair e/2 reuses a register whose score is already consumed
            }
            // the P V that read this P buffer last, two tiles ago, is complete
            if (j > 1) {
                bool done = mbar_wait_unless(bar(kBODone + X), ((j - 2) >> 1) & 1, failed);
                if (!__all_sync(0xffffffffu, done) && lane == 0) { *failed = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
                tc_fence_after();
            }
#pragma unroll
            for (int c = 0; c < HK / 32; c++) tmem_st16(tP + H * (HK / 2) + c * 16, sv + c * 16);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            l_run = (m_own != m_ref && m_own != -INFINITY ? l_run * exp2f(m_own - m_ref) : l_run) + (sum + sum2);
            m_own = m_ref;
            // O may be rescaled once the previous P V is complete.  A parity wait cannot tell a phase from the one two
            // before it, so the phase before the awaited one has to be known to be complete: the barriers alternate between
            // tiles, and P V of tile j - 2, waited for above, was issued after that of tile j - 3.
            if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                bool done = mbar_wait_bounded(bar(kBODone + (X ^ 1)), ((j - 1) >> 1) & 1) && !*failed;
                done = __all_sync(0xffffffffu, done);
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
            __syncwarp();
            if (lane == 0) arrive_cluster(p_full0);
        }
        // ---- epilogue: O / l -> out, or a slice's partial rows.  The group that did not have the last tile waits for the
        // P V of its own last one first, so that both are one phase ahead at most when they wait for the last.
        const int lt = n_tiles - 1;
        if (ok && X != (lt & 1)) {
            if (lt > 0) ok = mbar_wait_bounded(bar(kBODone + X), ((lt - 1) >> 1) & 1);
            if (ok) ok = mbar_wait_bounded(bar(kBRef + (lt & 1) * 4 + quarter), (lt >> 1) & 1);
        }
        if (ok) ok = mbar_wait_bounded(bar(kBODone + (lt & 1)), (lt >> 1) & 1) && !*failed;
        ok = __all_sync(0xffffffffu, ok);
        const float m_ref = X == (lt & 1) ? m_own : s_ref[(lt & 1) * 128 + m];
        s_sum[(X * 2 + H) * 128 + m] = m_own == -INFINITY ? 0.f : l_run * exp2f(m_own - m_ref);
        bar_sync(9 + quarter, 128);  // the four warps that share these rows
        const float l_row = (s_sum[m] + s_sum[128 + m]) + (s_sum[256 + m] + s_sum[384 + m]);
        if (!ok && lane == 0) {
            *failed = 1;
            atomicOr(a.status, ST_WAIT_TIMEOUT);
        }
        tc_fence_after();
        const int part = X * 2 + H;                        // this warp's quarter of the O columns
        if (wk.parts == 1) {
            if (ok) {
                const float inv = 1.f / l_row;
                uint16_t* orow = reinterpret_cast<uint16_t*>(a.out) +
                                 ((size_t)sm.tok_off * a.geo.n_q + (size_t)(h * n_rep + (row_ok ? rep : 0)) * sm.snew + (row_ok ? r0 + i : 0)) * D;
#pragma unroll 1
                for (int c = part * (D / 128); c < (part + 1) * (D / 128); c++) {
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
                float4* rows = slice_rows<D>(a, slot, 2, rank) + prow;
#pragma unroll 1
                for (int c = part * (D / 128); c < (part + 1) * (D / 128); c++) {
                    uint32_t v[32];
                    tmem_ld32(tO + lane_addr + c * 32, v);
                    if (row_ok) {
#pragma unroll
                        for (int u = 0; u < 8; u++)
                            rows[(size_t)(c * 8 + u) * 128] = make_float4(__uint_as_float(v[u * 4]), __uint_as_float(v[u * 4 + 1]),
                                                                          __uint_as_float(v[u * 4 + 2]), __uint_as_float(v[u * 4 + 3]));
                    }
                }
                if (part == 0 && row_ok) a.split_ml[((size_t)slot * 2 + rank) * 128 + prow] = make_float2(m_ref, l_row);
            }
            // every softmax warp passes the barriers whatever happened to its waits
            if (last_slice(a, wk, 13, 512, tid == 64, s_ticket) && !*failed && nv > 0)
                merge_slices<D, BF16>(a, wk, 2, rank, nv, r0, tid - 64, 512);
        }
    }
    // ---- wind down: both CTAs meet (nothing is on its way to either any more), then the tensor memory is freed
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    cluster_sync();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

bool chunk_pair_supported(int d) { return d == 128 || d == 256; }

cudaError_t chunk_pair_init() {
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(chunk_pair_kernel<128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_smem_bytes<128>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_pair_kernel<128, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_smem_bytes<128>())) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(chunk_pair_kernel<256, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_smem_bytes<256>())) != cudaSuccess) return e;
    return cudaFuncSetAttribute(chunk_pair_kernel<256, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_smem_bytes<256>());
}

cudaError_t launch_chunk_pair(const CUtensorMap& map_k, const CUtensorMap& map_v, const ChunkArgs& a, bool bf16, bool overlap, cudaStream_t st) {
    if (a.n_items <= 0) return cudaSuccess;
    switch (a.geo.d) {
        case 128: return bf16 ? launch_pdl(overlap, chunk_pair_kernel<128, true>, 2 * a.n_items, kPairThreads, pair_smem_bytes<128>(), st, map_k, map_v, a)
                              : launch_pdl(overlap, chunk_pair_kernel<128, false>, 2 * a.n_items, kPairThreads, pair_smem_bytes<128>(), st, map_k, map_v, a);
        case 256: return bf16 ? launch_pdl(overlap, chunk_pair_kernel<256, true>, 2 * a.n_items, kPairThreads, pair_smem_bytes<256>(), st, map_k, map_v, a)
                              : launch_pdl(overlap, chunk_pair_kernel<256, false>, 2 * a.n_items, kPairThreads, pair_smem_bytes<256>(), st, map_k, map_v, a);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace cbkv
