// CUDA kernels of the paged KV path, written for sm_100a.
//
//   append_kernel   scatter of a step's new K/V rows into page slots
//                   (reference: the slice_assign loop, kv.rs:721-734)
//   decode_kernel   GQA decode attention read in place from the pages, with the
//                   append fused in: no gather copy (kv.rs:611-636), no repeat_kv
//                   (kv.rs:177-187), no f32 upcast pass (kv.rs:213-215)
//   chunk_kernel    attention of a chunk of new tokens over paged prefix + chunk
//                   (causal, bottom-right aligned, optional window; kv.rs:243-268)
//   generic_kernel  any page size / head_dim; one warp per query row
//
// Layout of one layer in HBM: pages [num_pages][n_kv][32 rows][d] (f16/bf16).  The 32
// rows of one (page, kv head) are [K slots 0-7][V slots 0-7][K slots 8-15][V slots 8-15]
// (page_row() in kernels.hpp).
// A tile reaches shared memory through one TMA box per 64-element column block
// (32 rows x 128 B, 128-byte swizzle), so ldmatrix reads are bank-conflict free.
//
// Math per tile (16 tokens) in a warp, all in registers:
//   S^T[16 tok x 8 col] = K[16 x d] . Q^T[d x 8 col]      mma.m16n8k16, f32 accumulate
//   online softmax over tokens: warp shuffles across the 8 row groups
//   O^T[d x 8 col]     += V^T[d x 16 tok] . P^T[16 tok x 8 col]
// A "column" is one (query token, q head of the kv group): for decode the 8 columns
// are the q heads that share the kv head, so K/V are read once for the whole group.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "kernels.hpp"
#include "pdl.cuh"
#include "tile.cuh"

namespace cbkv {


// ------------------------------------------------------------------ append
template <typename T>
__global__ void append_kernel(const AppendArgs a) {
    const int D8 = a.geo.d / 8;
    const int64_t total = (int64_t)a.step.n_tokens * a.geo.n_kv * 2 * D8, stride = (int64_t)gridDim.x * blockDim.x;
    // where 16 bytes go, in vectors of the arena; -1: the table entry is not a page
    auto place_of = [&](int64_t idx) -> int64_t {
        const int64_t rem = idx / D8;
        const int kv = (int)(rem & 1), c = (int)(idx - rem * D8);
        int64_t row = rem >> 1;  // packed row: sequence blocks of [n_kv][snew] rows
        int lo = 0, hi = a.step.n_seqs - 1;  // last sequence whose first row is <= row
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if ((int64_t)a.step.seq_meta[mid].tok_off * a.geo.n_kv <= row) lo = mid; else hi = mid - 1;
        }
        const SeqMeta sm = a.step.seq_meta[lo];
        int64_t local = row - (int64_t)sm.tok_off * a.geo.n_kv;
        int h = (int)(local / sm.snew), r = (int)(local % sm.snew);
        int gpos = sm.pos + r;                         // global = pos + written, kv.rs:725
        int phys = a.step.tables[sm.tbl_off + gpos / a.geo.page_size];  // kv.rs:728
        int slot = gpos % a.geo.page_size;             // kv.rs:726
        if (phys < 0 || phys >= a.geo.num_pages) { atomicOr(a.status, ST_BAD_PAGE); return -1; }
        return (((int64_t)phys * a.geo.n_kv + h) * 2 * a.geo.page_size + page_row(kv, slot, a.geo.page_size, a.geo.tiled != 0)) * D8 + c;
    };
    // The first look-up, a chain of loads, runs under the tail of the launch before: the records and block tables came with
    // the step's upload, which no kernel overlaps.
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t to = idx < total ? place_of(idx) : -1;
    pdl_wait();
    pdl_launch_dependents();
    while (idx < total) {
        const int64_t rem = idx / D8;
        if (to >= 0) reinterpret_cast<uint4*>(a.arena)[to] = *(reinterpret_cast<const uint4*>((rem & 1) ? a.v : a.k) + (rem >> 1) * D8 + (idx - rem * D8));
        idx += stride;
        if (idx < total) to = place_of(idx);
    }
}

// ------------------------------------------------------------------ decode
// The launch's (sequence, kv head, page) units are cut into work items (manager.hpp): CTA c
// starts with item c and then claims further items from a device counter, larger ones first,
// so CTAs on SMs that stream more slowly take fewer of them and all finish together.  An item
// may cover the tail of one segment, whole segments and the head of another ("pieces").
//
// Warp 0 is the producer: it claims items two ahead, publishes them to the other warps
// through a small queue in shared memory, reads each tile's record index from the per-step
// unit_row array (one coalesced load per 32 tiles) and issues the TMA copies into a CTA-wide
// ring of NS stages.  The next C warps consume: tile n of the CTA (counted across items)
// lives in stage n % NS and belongs to consumer warp n % C, and NS is a multiple of C, so
// every stage has one producer and one consumer that visit it in order (an mbarrier parity
// wait is only unambiguous for a waiter at most one phase ahead).  Each consumer keeps a
// running (max, sum, numerator) state in registers; when a piece ends the states go to
// shared memory and the last warp (merger) combines them off the consumers' path.  A segment
// cut across items leaves partials in global scratch; whoever draws the segment's last ticket
// merges them (nobody waits for another CTA).
//
// Every wait is bounded; a warp that gives up records it in the status word, raises the CTA's
// failure flag and falls through the remaining barriers without computing.  The producer
// leaves last, after every copy it issued has landed.
constexpr int QN = 8;          // slots of the item queue (a power of two)
constexpr int DEFER_CAP = 20;  // segments a CTA can leave to its cooperative merge at the end

struct Piece {
    int sb, se;  // unit range of the segment
    int h;
    int q_pos, page_lo, page_last, tok_off, nparts, part_base;
};

__device__ __forceinline__ Piece load_piece(const DecodeArgs& a, int seg) {
    // this segment's record and the first word of the next one (the array has n_segs + 1 entries)
    const int4* p = reinterpret_cast<const int4*>(a.segs + seg);
    const int4 x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2);
    Piece pc;
    pc.sb = x.x; pc.page_lo = x.y; pc.q_pos = x.z; pc.tok_off = x.w;
    pc.nparts = y.x; pc.part_base = y.y;
    pc.se = z.x;
    pc.h = seg % a.geo.n_kv;
    pc.page_last = pc.q_pos >> 4;  // decode: the one new token, at the end of the window
    return pc;
}

template <int D>
__device__ __forceinline__ void load_q_frags(const DecodeArgs& a, const Piece& p, int g, int t, uint32_t (&qf)[1][D / 16][2]) {
    // Q^T fragments of the kv group's q heads (columns >= n_rep are zero)
    const int n_rep = a.geo.n_rep;
    const uint32_t* qrow = reinterpret_cast<const uint32_t*>(
        reinterpret_cast<const uint16_t*>(a.q) + ((size_t)p.tok_off * a.geo.n_q + (size_t)p.h * n_rep + (g < n_rep ? g : 0)) * D);
#pragma unroll
    for (int ks = 0; ks < D / 16; ks++) {
        qf[0][ks][0] = g < n_rep ? __ldg(qrow + ks * 8 + t) : 0u;
        qf[0][ks][1] = g < n_rep ? __ldg(qrow + ks * 8 + 4 + t) : 0u;
    }
}

// The same fragments in the contraction order of the quantised K tiles (see q8_attend).
template <int D>
__device__ __forceinline__ void load_q_frags_q8(const DecodeArgs& a, const Piece& p, int g, int t, uint32_t (&qf)[1][D / 16][2]) {
    const int n_rep = a.geo.n_rep;
    const uint2* qrow = reinterpret_cast<const uint2*>(
        reinterpret_cast<const uint16_t*>(a.q) + ((size_t)p.tok_off * a.geo.n_q + (size_t)p.h * n_rep + (g < n_rep ? g : 0)) * D);
#pragma unroll
    for (int ks = 0; ks < D / 16; ks++) {
        // k-step ks = 2*grp + s contracts d = 32*grp + 8t + 4s + {0..3}: one 8-byte word
        const uint2 v = g < n_rep ? __ldg(qrow + (ks >> 1) * 8 + 2 * t + (ks & 1)) : make_uint2(0u, 0u);
        qf[0][ks][0] = v.x;
        qf[0][ks][1] = v.y;
    }
}

__device__ __forceinline__ void consumer_sync(int nthreads) {
    asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
}
__device__ __forceinline__ int4 lds128(uint32_t addr) {
    int4 v;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, int4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

#ifdef CBKV_MEASURE
// per-CTA timestamps, 16 slots each
#define CBKV_STAMP(slot) do { if ((a.debug & 4) && a.dbg_buf) a.dbg_buf[(size_t)blockIdx.x * 16 + (slot)] = global_ns(); } while (0)
#define CBKV_DBG(bit) (a.debug & (bit))
#else
#define CBKV_STAMP(slot) do { } while (0)
#define CBKV_DBG(bit) 0
#endif

// Merge the partial results of one segment (log-sum-exp combine) and store its output.
// Thread r of T takes every T-th (column, 4 d-values) item; the loads of up to eight
// parts are issued together, so an item costs one round trip to memory.
template <int D, bool BF16>
__device__ __forceinline__ void merge_parts(const DecodeArgs& a, int base, int nparts, uint16_t* out_row, int n_rep, int r, int T) {
    constexpr int PER_COL = D / 4;
    for (int idx = r; idx < n_rep * PER_COL; idx += T) {
        const int col = idx / PER_COL, j4 = idx - col * PER_COL;
        float M = -INFINITY, L = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int p0 = 0; p0 < nparts; p0 += 8) {
            float2 ml[8];
            float4 v[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const bool ok = p0 + q < nparts;
                const size_t rec = (size_t)(base + p0 + (ok ? q : 0)) * 8 + col;
                ml[q] = __ldcg(reinterpret_cast<const float2*>(a.part_ml) + rec);
                v[q] = __ldcg(reinterpret_cast<const float4*>(a.part_o + rec * D) + j4);
                if (!ok) ml[q] = make_float2(-INFINITY, 0.f);
            }
            float Mnew = M;
#pragma unroll
            for (int q = 0; q < 8; q++) Mnew = fmaxf(Mnew, ml[q].x);
            const float so = (M == -INFINITY) ? 0.f : exp2f(M - Mnew);
            acc.x *= so; acc.y *= so; acc.z *= so; acc.w *= so;
            L *= so;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const float f = (ml[q].x == -INFINITY) ? 0.f : exp2f(ml[q].x - Mnew);
                acc.x += f * v[q].x; acc.y += f * v[q].y; acc.z += f * v[q].z; acc.w += f * v[q].w;
                L += f * ml[q].y;
            }
            M = Mnew;
        }
        const float inv = 1.f / L;
        uint2 pk;
        pk.x = pack2<BF16>(acc.x * inv, acc.y * inv);
        pk.y = pack2<BF16>(acc.z * inv, acc.w * inv);
        *reinterpret_cast<uint2*>(out_row + col * D + j4 * 4) = pk;
    }
}

// One (column, 4 d-values) item of a piece: the C consumers' states (rows of DP floats, ccols of them each; maxima and sums)
// combined, and the output stored, or the partial of a cut segment.
template <int D, int C, bool BF16>
__device__ __forceinline__ void combine_states(const DecodeArgs& a, const float* co, const float* cml, int ccols, int col, int j4, int nparts, int slot, uint16_t* out_row) {
    constexpr int DP = D + 4;
    float M = -INFINITY;
#pragma unroll
    for (int ww = 0; ww < C; ww++) M = fmaxf(M, cml[(ww * 8 + col) * 2]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float ls = 0.f;
#pragma unroll
    for (int ww = 0; ww < C; ww++) {
        const float mw = cml[(ww * 8 + col) * 2];
        const float f = (mw == -INFINITY) ? 0.f : exp2f(mw - M);
        const float4 v = *reinterpret_cast<const float4*>(co + ((size_t)ww * ccols + col) * DP + j4 * 4);
        acc.x += f * v.x; acc.y += f * v.y; acc.z += f * v.z; acc.w += f * v.w;
        ls += f * cml[(ww * 8 + col) * 2 + 1];
    }
    if (nparts == 1) {
        const float inv = 1.f / ls;
        uint2 pk;
        pk.x = pack2<BF16>(acc.x * inv, acc.y * inv);
        pk.y = pack2<BF16>(acc.z * inv, acc.w * inv);
        *reinterpret_cast<uint2*>(out_row + col * D + j4 * 4) = pk;
    } else {
        *reinterpret_cast<float4*>(a.part_o + ((size_t)slot * 8 + col) * D + j4 * 4) = acc;
        if (j4 == 0) *reinterpret_cast<float2*>(a.part_ml + ((size_t)slot * 8 + col) * 2) = make_float2(M, ls);
    }
}

// Record index (page * n_kv + kv head) of every unit of a decode plan, once per step and
// window: the decode launches of all layers read it instead of chasing the block tables.
__global__ void resolve_units_kernel(const SegInfo* segs, int n_segs, const int32_t* tables, int n_kv, int num_pages,
                                     int32_t* unit_row, int n_units, int32_t* status,
                                     int32_t* zero_a, int n_a, int32_t* zero_b, int n_b) {
    // the step's first launch of this kernel also puts the tickets and claim counters back to zero (whatever a
    // launch that gave up left behind): one stream operation per step instead of three
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_a; i += gridDim.x * blockDim.x) zero_a[i] = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_b; i += gridDim.x * blockDim.x) zero_b[i] = 0;
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < n_units; u += gridDim.x * blockDim.x) {
        int lo = 0, hi = n_segs - 1;  // last segment whose first unit is <= u (an empty segment shares its successor's)
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (segs[mid].unit_begin <= u) lo = mid; else hi = mid - 1;
        }
        const SegInfo sg = segs[lo];
        const int phys = tables[sg.tbl_off + sg.page_lo + (u - sg.unit_begin)];
        if (phys < 0 || phys >= num_pages) {
            atomicOr(status, ST_BAD_PAGE);
            unit_row[u] = -1;  // the decode kernel reads page 0 instead and writes nothing
        } else {
            unit_row[u] = phys * n_kv + lo % n_kv;
        }
    }
}

// Warp roles: 0 = producer, 1..C = consumers, C+1 = merger.
// Q8: the layer holds int8 records; a tile is one record fetched as one box of a byte tensor map.
// ROPE: q and k_new are normed and rotated here (DecodeArgs::rope); a variant of its own, because the words it holds cost
// the other ones registers (236 bytes of spills at head_dim 128).  Its own registers are bounded by what a launch has
// resident, one CTA per SM, over int8 pages of head_dim 64 and 128 two.  Left to itself the compiler took 128 with 268 bytes
// of spills (16 bits, head_dim 128: 193 now) and 241 (int8: 168 now), which left no room for the second CTA: 32 sequences of
// 1024 to 4096 tokens, 28/4/128, 28 layers: 1058 -> 957 us, int8 1417 -> 1019 (rotated by a launch of its own 1165, 1047).
// 16-bit pages: one CTA per SM, whose ring takes its shared memory, so its registers are not held to what two would have
// (head_dim 128: 128, with 144 bytes of spills, 1949 us for 28 layers of 32 sequences, two steps; 176 and 1882 now).
template <int D, int C, bool BF16, bool Q8, bool ROPE>
__global__ void __launch_bounds__((C + 2) * 32, !Q8 ? 1 : !ROPE ? 0 : D <= 128 ? 2 : 1) decode_kernel(const __grid_constant__ CUtensorMap tmap, const DecodeArgs a) {
    constexpr uint32_t UNIT = Q8 ? (uint32_t)(2 * 16 * D + 2 * 16 * (D / 32) * 2) : 32u * D * 2u;
    constexpr int DP = D + 4;  // row pitch of the merge buffers: the four lanes of a quad land in different banks
    extern __shared__ __align__(1024) uint8_t smem[];
    const int NS = a.n_stages;            // multiple of C (checked by the host)
    const int ccols = a.comb_cols;
    const int NB = a.comb_bufs;           // 1 or 2 state buffers between consumers and merger
    float* comb_o = reinterpret_cast<float*>(smem + (size_t)NS * UNIT);      // [NB][C][ccols][DP]
    float* comb_ml = comb_o + (size_t)NB * C * ccols * DP;                    // [NB][C][8][2]
    int4* qitems = reinterpret_cast<int4*>(comb_ml + NB * C * 16);            // [QN] published items
    uint64_t* bar_full = reinterpret_cast<uint64_t*>(qitems + QN);           // [NS] tile landed
    uint64_t* bar_empty = bar_full + NS;                                      // [NS] tile consumed
    uint64_t* bar_cfull = bar_empty + NS;                                     // [2] all consumers stored their states
    uint64_t* bar_cempty = bar_cfull + 2;                                     // [2] merger is done with the buffer
    uint64_t* bar_qfull = bar_cempty + 2;                                     // [QN] item published
    uint64_t* bar_qempty = bar_qfull + QN;                                    // [QN] item read by consumers and merger
    int* flag = reinterpret_cast<int*>(bar_qempty + QN);                      // [1] a warp gave up, [2] merges left to the end, [4..4+DEFER_CAP) their segments

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cta = blockIdx.x;
    if ((smem_u32(smem) & 1023u) != 0) {
        if (tid == 0) atomicOr(a.status, ST_SMEM_ALIGN);
        return;
    }
    if (tid == 0) CBKV_STAMP(0);
    const uint32_t ring = smem_u32(smem);
    const uint32_t full0 = smem_u32(bar_full), empty0 = smem_u32(bar_empty);
    const uint32_t cfull0 = smem_u32(bar_cfull), cempty0 = smem_u32(bar_cempty);
    const uint32_t qfull0 = smem_u32(bar_qfull), qempty0 = smem_u32(bar_qempty), qitems0 = smem_u32(qitems);
    const int Hkv = a.geo.n_kv;
    const uint64_t lim = (uint64_t)a.wait_us * 1000ull;
    if (tid == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap) : "memory");
        for (int i = 0; i < NS; i++) { mbar_init(full0 + i * 8, 1); mbar_init(empty0 + i * 8, 1); }
        for (int i = 0; i < 2; i++) { mbar_init(cfull0 + i * 8, C); mbar_init(cempty0 + i * 8, 1); }
        for (int i = 0; i < QN; i++) { mbar_init(qfull0 + i * 8, 1); mbar_init(qempty0 + i * 8, C + 1); }
        flag[0] = 0; flag[1] = 0; flag[2] = 0;
        fence_mbar_init();
        fence_proxy_async();
    }
    __syncthreads();
    volatile int* vflag = flag;

    if (warp == 0) {
        // ------------------------------------------------------------ producer
        // The pages read here were written by earlier steps; only when earlier work in the
        // stream wrote this layer's pages or the unit_row array must it be waited for.
        if (a.kv_dep) pdl_wait();
        bool failed = false;
        const int rshift = NS < 8 ? 2 : 3;  // lanes per issue round (4 or 8): never more than the ring has stages
        auto fetch = [&](int id) -> int4 {
            return id < a.n_items ? __ldg(reinterpret_cast<const int4*>(a.items) + id) : make_int4(-1, -1, 0, 0);
        };
        // A claim is issued (one atomic by lane 0) when an item starts and picked up after the item's
        // first round of copies is out, so the counter's round trip never holds up a copy.
        auto claim_issue = [&]() -> int {
            int v = 0;
            if (lane == 0) v = a.n_ctas + atomicAdd(a.work_counters + a.work_slot, 1);
            return v;
        };
        auto publish = [&](int j, int4 info) {
            if (lane == 0) {
                const int s = j & (QN - 1);
                if (j >= QN && !mbar_wait_bounded(qempty0 + s * 8, ((j / QN) - 1) & 1, 4 * lim)) {
                    failed = true;
                } else {
                    sts128(qitems0 + s * 16, info);
                    mbar_arrive(qfull0 + s * 8);
                }
            }
            failed = __any_sync(0xffffffffu, failed);
        };
        int raw = claim_issue();  // this CTA's second item
        // The unit range of this CTA's first item follows from the launch's totals (the host cuts the
        // same way, build_decode_plan), so the first copies leave without waiting for its record; the
        // record itself (first segment, part index) is fetched meanwhile for the other warps.
        // (A plan whose ranges end where segments do has them in the records only.)
        int4 cur, rec0;
        if (a.aligned) {
            cur = rec0 = fetch(cta);
        } else {
            const long long rb = (long long)a.n_units * cta / a.n_ctas, re = (long long)a.n_units * (cta + 1) / a.n_ctas;
            const long long len = re - rb;
            cur = make_int4((int)rb, (int)(re - len * a.tail_pct / 100), 0, 0);
            rec0 = fetch(cta);  // the record and the first rows travel together
        }
        int row_first = lane < cur.y - cur.x ? __ldcg(a.unit_row + cur.x + lane) : 0;
        publish(0, rec0);
        int4 nxt = make_int4(-1, -1, 0, 0);
        int j = 0, T = 0;  // items started, tile slots used (copies and the fillers between items)
#pragma unroll 1
        while (!failed) {
            const int ub = cur.x, ntl = cur.y - cur.x;
            bool to_publish = true;
            int row_next = j == 0 ? row_first : (lane < ntl ? __ldcg(a.unit_row + ub + lane) : 0);
#pragma unroll 1
            for (int base = 0; base < ntl && !failed; base += 32) {
                const int row = row_next;
                if (base + 32 + lane < ntl) row_next = __ldcg(a.unit_row + ub + base + 32 + lane);
                const int nb = min(32, ntl - base);
                const int Tl = T + base + lane;
                const int st = Tl % NS, rev = Tl / NS;
                for (int r = 0; (r << rshift) < nb; r++) {
                    if ((lane >> rshift) == r && lane < nb) {
                        if (Tl >= NS && !mbar_wait_bounded(empty0 + st * 8, (rev - 1) & 1, lim)) {
                            failed = true;
                        } else if (!(cta == 0 && Tl == a.fault_tile)) {
                            const int rec = row < 0 ? 0 : row;
                            if constexpr (Q8) {
                                mbar_expect_tx(full0 + st * 8, UNIT);  // one box of UNIT/128 rows x 128 bytes = one record
                                tma_load_2d(ring + st * UNIT, &tmap, 0, rec * (int)(UNIT / 128u), full0 + st * 8);
                            } else {
                                issue_tile<D>(&tmap, ring + st * UNIT, full0 + st * 8, rec * 32);
                            }
                        }
                    }
                    __syncwarp();
                    // The item after this one is published once the first round is out: that round only
                    // needs stages of earlier items, whereas later rounds may need this item's own tiles
                    // consumed, and its consumers may already be waiting for the queue entry.
                    if (to_publish) {
                        nxt = fetch(__shfl_sync(0xffffffffu, raw, 0));
                        publish(j + 1, nxt);
                        to_publish = false;
                    }
                }
                failed = __any_sync(0xffffffffu, failed) || vflag[1] != 0;
                if (j == 0 && base == 0 && lane == 0) CBKV_STAMP(2);
            }
            if (to_publish && !failed) {  // an item without tiles (the host never makes one)
                nxt = fetch(__shfl_sync(0xffffffffu, raw, 0));
                publish(j + 1, nxt);
            }
            T += ntl;
            if (nxt.x < 0 || failed) break;  // the end marker is already in the queue
            // Fillers: every item starts on a tile slot that is a multiple of C, so that a tile's consumer
            // warp depends on its place in the item only and results do not depend on which CTA ran which
            // item.  A filler slot carries no copy: its barrier is completed by a plain arrival.
            const int pad = (C - T % C) % C;
            if (pad) {
                const int Tl = T + lane;
                if (lane < pad) {
                    const int st = Tl % NS, rev = Tl / NS;
                    if (Tl >= NS && !mbar_wait_bounded(empty0 + st * 8, (rev - 1) & 1, lim)) failed = true;
                    else mbar_arrive(full0 + st * 8);
                }
                failed = __any_sync(0xffffffffu, failed);
                T += pad;
            }
            cur = nxt;
            j++;
            raw = claim_issue();
        }
        if (lane == 0) CBKV_STAMP(7);
        // Leave last: the stages of the final tiles are released by their consumers, which means the
        // copies have landed.  After a failure nobody may be consuming, so the copies themselves are awaited.
        {
            const int from = max(0, T - NS);
            bool bad = failed || vflag[1] != 0;
            for (int n = from + lane; n < T && !bad; n += 32)
                if (!mbar_wait_bounded(empty0 + (n % NS) * 8, (n / NS) & 1, 4 * lim)) bad = true;
            bad = __any_sync(0xffffffffu, bad) || vflag[1] != 0;
            if (bad) {
                if (lane == 0) { atomicOr(a.status, ST_WAIT_TIMEOUT); atomicExch(flag + 1, 1); }
                for (int n = from + lane; n < T; n += 32)
                    if (!(cta == 0 && n == a.fault_tile)) mbar_wait_bounded(full0 + (n % NS) * 8, (n / NS) & 1, 20000000ull);
            }
        }
        return;
    }

    // consumers and merger: read entry j of the item queue (false: no more items, or a wait ran out)
    bool failed = false;
    auto get_item = [&](int j, int4& out) -> bool {
        if (failed) return false;
        const int s = j & (QN - 1);
        if (!mbar_wait_bounded(qfull0 + s * 8, (j / QN) & 1, 4 * lim)) {
            failed = true;
            if (lane == 0) { atomicOr(a.status, ST_WAIT_TIMEOUT); atomicExch(flag + 1, 1); }
            return false;
        }
        out = lds128(qitems0 + s * 16);
        __syncwarp();
        if (lane == 0) mbar_arrive(qempty0 + s * 8);
        return out.x >= 0;
    };

    // the same without waiting: 1 = entry read (out valid, possibly the end marker), 0 = not published yet
    auto peek_item = [&](int j, int4& out) -> bool {
        const int s = j & (QN - 1);
        int ok = 0;
        if (lane == 0) ok = (int)mbar_test_wait(qfull0 + s * 8, (j / QN) & 1);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) return false;
        out = lds128(qitems0 + s * 16);
        __syncwarp();
        if (lane == 0) mbar_arrive(qempty0 + s * 8);
        return true;
    };

    const int n_rep = a.geo.n_rep;
    // ALL: the CTA's last piece is combined by all its consumers and the merger, who meet first: nothing is left to overlap with,
    // and one warp's combine was much of the way from the last tile to the exit.  One sequence of 340 tokens with rotation
    // (8 segments of 22 pages, 32/8/128) 6.7 -> 5.6 us per launch, 32 sequences of 1024 to 4096 (28/4/128) 34.6 -> 33.5.  Where two
    // CTAs share an SM (int8 pages) the other one's tiles fill that time, and meeting costs 1.3 %: the merger does it there.  Every
    // warp passes the same barriers whatever happened to its waits; what a launch that gave up stores is undefined, as its output is.
    const bool ALL = !Q8 || a.combine_all != 0;
    auto combine_last = [&](int seg, const int4& x, const int4& y, int first_seg, int first_part, int buf) {
        consumer_sync((C + 1) * 32);
        if (warp == C + 1 && lane == 0) CBKV_STAMP(5);
        const int nparts = y.x, slot = nparts > 1 ? y.y + (seg == first_seg ? first_part : 0) : 0;
        uint16_t* out_row = reinterpret_cast<uint16_t*>(a.out) + ((size_t)x.w * a.geo.n_q + (size_t)(seg % Hkv) * n_rep) * D;
        for (int idx = tid - 32; idx < n_rep * (D / 4); idx += (C + 1) * 32) {
            const int col = idx / (D / 4);
            combine_states<D, C, BF16>(a, comb_o + (size_t)buf * C * ccols * DP, comb_ml + buf * C * 16, ccols, col, idx - col * (D / 4), nparts, slot, out_row);
        }
        consumer_sync((C + 1) * 32);
    };
    if (warp == C + 1) {
        // -------------------------------------------------------------- merger
        // Combines the consumers' states of each piece, writes the output (or a partial
        // plus a ticket; the last ticket holder merges the segment's partials), and hands
        // the buffer back.  The consumers never wait on global memory.
        pdl_wait();  // out and the scratch are shared with earlier launches
        if (cta == 0 && lane == 0) a.work_counters[(a.work_slot + 2) & 3] = 0;  // for the launch after the next one
        // Only now may the next launch start: at most two launches are alive at a time, which is
        // what lets four claim counters rotate.
        pdl_launch_dependents();
        int k = 0, kk = 0, n_deferred = 0;
        // The ticket of a cut piece is drawn right after its partial is stored but looked at one piece
        // later, so the counter's round trip overlaps the wait for the next piece.  A segment whose
        // last ticket this CTA drew is merged at the end of the CTA by all its warps (the consumers
        // are idle by then); only when the list is full does this warp merge alone.
        int pend_seg = -1, pend_np = 0, pend_raw = 0;
        auto settle = [&]() {
            if (pend_seg < 0) return;
            int last = 0;
            if (lane == 0 && pend_raw == pend_np - 1) {
                last = 1;
                a.seg_counter[pend_seg] = 0;  // ready for the next launch
            }
            last = __shfl_sync(0xffffffffu, last, 0);
            if (last) {
                if (n_deferred < DEFER_CAP) {
                    if (lane == 0) flag[4 + n_deferred] = pend_seg;
                    n_deferred++;
                } else {
                    const int4* sp = reinterpret_cast<const int4*>(a.segs + pend_seg);
                    const int4 x = __ldg(sp), y = __ldg(sp + 1);
                    uint16_t* orow = reinterpret_cast<uint16_t*>(a.out) + ((size_t)x.w * a.geo.n_q + (size_t)(pend_seg % Hkv) * n_rep) * D;
                    merge_parts<D, BF16>(a, y.y, y.x, orow, n_rep, lane, 32);
                }
            }
            pend_seg = -1;
        };
#ifdef CBKV_MEASURE
        int dbg_tiles = 0, dbg_cut = 0;
#endif
        auto draw = [&](int seg, int nparts) {
            if (lane == 0) {
                // release: the partial (ordered before by __syncwarp or the CTA's barrier) is visible before the ticket;
                // acquire: whoever draws the last ticket sees every other part's partial
                asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(pend_raw) : "l"(a.seg_counter + seg) : "memory");
            }
            pend_seg = seg;
            pend_np = nparts;
#ifdef CBKV_MEASURE
            dbg_cut++;
#endif
        };
        int4 it;
        bool have = get_item(0, it);
        int seg = have ? it.z : 0;
#pragma unroll 1
        while (have) {
            int pb = it.x;
            int4 nit;
            bool more = false;
#pragma unroll 1
            while (pb < it.y) {
                const int4* sp = reinterpret_cast<const int4*>(a.segs + seg);
                const int4 x = __ldg(sp), y = __ldg(sp + 1), z = __ldg(sp + 2);
                const int pe = min(it.y, z.x);
#ifdef CBKV_MEASURE
                dbg_tiles += pe - pb;
#endif
                if (pe == it.y) {
                    more = get_item(k + 1, nit);
                    if (ALL && !more) break;  // the CTA's last piece is left to all its warps
                }
                const int h = seg % Hkv;
                const int tok_off = x.w, nparts = y.x;
                const int slot = nparts > 1 ? y.y + (seg == it.z ? it.w : 0) : 0;
                const int buf = NB == 2 ? (kk & 1) : 0, use = NB == 2 ? (kk >> 1) : kk;
                if (!mbar_wait_bounded(cfull0 + buf * 8, use & 1, 4 * lim)) {
                    failed = true;
                    if (lane == 0) { atomicOr(a.status, ST_WAIT_TIMEOUT); atomicExch(flag + 1, 1); }
                    break;
                }
                if (lane == 0) CBKV_STAMP(5);
                uint16_t* out_row = reinterpret_cast<uint16_t*>(a.out) + ((size_t)tok_off * a.geo.n_q + (size_t)h * n_rep) * D;
                // lane owns 4 consecutive d-values (per pass of 128) of every query column
                constexpr int PASSES = (D + 127) / 128;
#pragma unroll
                for (int ps = 0; ps < PASSES; ps++) {
                    const int j4 = ps * 32 + lane;  // float4 index within a row of D
                    if (j4 * 4 < D) {
#pragma unroll
                        for (int col = 0; col < 8; col++)
                            if (col < n_rep) combine_states<D, C, BF16>(a, comb_o + (size_t)buf * C * ccols * DP, comb_ml + buf * C * 16, ccols, col, j4, nparts, slot, out_row);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(cempty0 + buf * 8);  // the consumers may store the next piece here
                settle();  // the previous cut piece's ticket has had a whole piece to come back
                if (nparts > 1) draw(seg, nparts);
                kk++;
                seg++;
                pb = pe;
            }
            if (failed || !more) break;
            k++;
            it = nit;
            seg = it.z;
        }
        if (ALL) {  // (a CTA whose first item never came falls through with segment 0; its output is undefined)
            const int4* sp = reinterpret_cast<const int4*>(a.segs + seg);
            const int4 x = __ldg(sp), y = __ldg(sp + 1);
            combine_last(seg, x, y, have ? it.z : 0, have ? it.w : 0, NB == 2 ? (kk & 1) : 0);
            settle();
            if (y.x > 1 && !failed) draw(seg, y.x);
            kk++;
        }
        settle();
        // hand the segments to merge to the whole CTA
        if (lane == 0) flag[2] = n_deferred;
        __syncwarp();
        consumer_sync((C + 1) * 32);
        for (int i = 0; i < n_deferred; i++) {
            const int sg = flag[4 + i];
            const int4* sp = reinterpret_cast<const int4*>(a.segs + sg);
            const int4 x = __ldg(sp), y = __ldg(sp + 1);
            uint16_t* out_row = reinterpret_cast<uint16_t*>(a.out) + ((size_t)x.w * a.geo.n_q + (size_t)(sg % Hkv) * n_rep) * D;
            merge_parts<D, BF16>(a, y.y, y.x, out_row, n_rep, C * 32 + lane, (C + 1) * 32);
        }
#ifdef CBKV_MEASURE
        if (lane == 0) {
            CBKV_STAMP(6);
            if ((a.debug & 4) && a.dbg_buf) {
                unsigned smid;
                asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
                a.dbg_buf[(size_t)blockIdx.x * 16 + 8] = (unsigned long long)kk;
                a.dbg_buf[(size_t)blockIdx.x * 16 + 9] = (unsigned long long)n_deferred;
                a.dbg_buf[(size_t)blockIdx.x * 16 + 10] = (unsigned long long)dbg_cut;
                a.dbg_buf[(size_t)blockIdx.x * 16 + 11] = (unsigned long long)smid;
                a.dbg_buf[(size_t)blockIdx.x * 16 + 12] = (unsigned long long)dbg_tiles;
                a.dbg_buf[(size_t)blockIdx.x * 16 + 13] = (unsigned long long)k;
            }
        }
#endif
        return;
    }

    // ---------------------------------------------------------------- consumers
    const int cw = warp - 1, g = lane >> 2, t = lane & 3;
    int4 it;
    bool have = get_item(0, it);  // plan and block tables were uploaded by a copy: always visible
    int seg = have ? it.z : 0, pb = have ? it.x : 0;
    Piece cur = load_piece(a, seg);
    if (have && g < a.geo.n_rep && t < (D * 2 + 127) / 128) {
        // ask for the first piece's q rows in L2 while the previous launch is still finishing (a request, not a
        // read: L2 is where that launch or a copy engine writes them, so nothing stale can be seen later)
        const char* qp = reinterpret_cast<const char*>(a.q) + ((size_t)cur.tok_off * a.geo.n_q + (size_t)cur.h * a.geo.n_rep + g) * D * 2 + t * 128;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(qp));
    }
    // the first piece's cosines and sines are no earlier launch's work: they travel under the wait
    uint32_t rcos[ROPE ? D / 32 : 1][2], rsin[ROPE ? D / 32 : 1][2];
    if constexpr (ROPE) { if (have) load_rope_words<D, Q8>(a.rope, cur.q_pos, t, rcos, rsin); }
    pdl_wait();  // q, k_new and v_new come from earlier work in the stream
    if (a.in_flag != nullptr) {
        // ... or from copies on another stream, which end by writing this launch's number behind the data:
        // one lane looks until it is there (bounded like every wait; a copy engine makes progress whatever
        // this kernel does), the warp meets, and only then are the inputs read
        if (lane == 0) {
            const uint64_t t0 = global_ns(), lim = (uint64_t)a.wait_us * 1000ull;
            uint32_t seen;
            for (;;) {
                asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.in_flag) : "memory");
                if ((int32_t)(seen - a.in_seq) >= 0) break;
                if (global_ns() - t0 > lim) { atomicOr(a.status, ST_WAIT_TIMEOUT); break; }
            }
        }
        __syncwarp();
    }
    uint32_t qf[1][D / 16][2];
    if constexpr (Q8) load_q_frags_q8<D>(a, cur, g, t, qf);
    else load_q_frags<D>(a, cur, g, t, qf);
    if (tid == 32) CBKV_STAMP(3);
    int k = 0, kk = 0, nbase = 0;  // items read, pieces handed over, tiles of the CTA before the current item
#ifdef CBKV_MEASURE
    bool first_tile = true;
#endif
#pragma unroll 1
    while (have) {
        const int pe = min(it.y, cur.se);
        const bool more = pe < it.y;
        // what comes next (the item's next segment, or the first piece of the next item): its
        // metadata and queries arrive while this piece is processed
        int4 nit = it;
        bool nhave = true, nknown = true;
        int nseg = seg + 1;
        if (!more) {
            // The next item's queue entry is looked at without waiting: the producer runs a ring ahead, so
            // it is nearly always there; if not, it is waited for after this piece's tiles (a consumer
            // never waits for the queue while tiles it has to consume are outstanding).
            nknown = !failed && peek_item(k + 1, nit);
            nhave = nknown && nit.x >= 0;
            nseg = nit.z;
        }
        Piece nxt = cur;
        uint32_t qf_next[1][D / 16][2];
        if (nknown && nhave) {
            nxt = load_piece(a, nseg);
            if constexpr (Q8) load_q_frags_q8<D>(a, nxt, g, t, qf_next);
            else load_q_frags<D>(a, nxt, g, t, qf_next);
        }
        float o[1][D / 16][4], m[1][2] = {{-INFINITY, -INFINITY}}, l[1][2] = {{0.f, 0.f}};
#pragma unroll
        for (int mt = 0; mt < D / 16; mt++) { o[0][mt][0] = o[0][mt][1] = o[0][mt][2] = o[0][mt][3] = 0.f; }
        const int qpos[1][2] = {{cur.q_pos, cur.q_pos}};
        if constexpr (ROPE) {
            if (kk > 0) load_rope_words<D, Q8>(a.rope, cur.q_pos, t, rcos, rsin);
            rope_q_frags<D, BF16, Q8>(a.rope, t, g < a.geo.n_rep, rcos, rsin, qf);
        }

        const int n0 = nbase + (pb - it.x);  // the piece's first tile, counted over the CTA's items
        const int n1 = n0 + (pe - pb);
        int T = n0 + (cw - n0 % C + C) % C;  // this warp's first tile of the piece
        // Short pieces: the step's new row and the page it goes to, for the warp that has the segment's last page, are asked for
        // here and arrive under the wait for the tiles and the products of the warp's earlier ones (us per launch, 2
        // sequences of 1000 to 3000, 4/256, 10.4 -> 9.4; 8 of 500 to 2000, 8/128, 12.2 -> 10.9; 16 of 8192 with windows of 1024,
        // 4/256, 28.1 -> 27.0).  In long pieces other warps are busy meanwhile and it costs 0.5 % (32 of 1024 to 4096); the
        // rotating variant gains nothing.
        constexpr int NROW = (2 * (D / 8) + 31) / 32;
        uint4 row_new[NROW];
        int rec_new = -1;
        bool early = false;
        if constexpr (!Q8 && !ROPE) {
            const int u_last = cur.sb + cur.page_last - cur.page_lo;
            early = a.k_new != nullptr && pe - pb <= 8 * C && u_last >= pb && u_last < pe && (n0 + u_last - pb) % C == cw;
            if (early) {
                rec_new = __ldcg(a.unit_row + u_last);
                const size_t rowi = (size_t)cur.tok_off * Hkv + cur.h;
#pragma unroll
                for (int i = 0; i < NROW; i++) {
                    const int c = lane + 32 * i, kv = c / (D / 8), j = c - kv * (D / 8);
                    if (c < 2 * (D / 8)) row_new[i] = __ldcg(reinterpret_cast<const uint4*>(kv ? a.v_new : a.k_new) + rowi * (D / 8) + j);
                }
            }
        }
        // stage and revolution parity of this warp's tiles, advanced by C per tile (NS is a multiple of C)
        int st = T % NS, par = (T / NS) & 1;
#pragma unroll 1
        for (; T < n1; T += C, st += C) {
            if (st >= NS) { st -= NS; par ^= 1; }
            const uint32_t stage = ring + st * UNIT;
            const int u = pb + (T - n0);
            if (!failed && !mbar_wait_bounded(full0 + st * 8, par, lim)) {
                failed = true;
                if (lane == 0) { atomicOr(a.status, ST_WAIT_TIMEOUT); atomicExch(flag + 1, 1); }
            }
            // After a failure nothing is released any more: a stage given back before its copy has landed
            // would be armed a second time.  The producer then finds its own wait running out and stops.
            if (failed) break;
#ifdef CBKV_MEASURE
            if (first_tile && tid == 32) { CBKV_STAMP(4); first_tile = false; }
#endif
            const int lp = cur.page_lo + (u - cur.sb);
            if (!CBKV_DBG(1)) {
                if (!Q8 && a.k_new != nullptr && lp == cur.page_last) {
                    // fused append: put the new K/V row into the tile just fetched and into its page
                    const int slot = cur.q_pos & 15;
                    const int rec = early ? rec_new : __ldcg(a.unit_row + u);
                    const size_t rowi = (size_t)cur.tok_off * Hkv + cur.h;
                    const uint16_t* krow = reinterpret_cast<const uint16_t*>(a.k_new) + rowi * D;
                    float inv_rms = 0.f;
                    if constexpr (ROPE) { if (a.rope.k_weight) inv_rms = inv_rms_of(row_sumsq<D, BF16>(krow, lane), D, a.rope.eps); }
                    auto put = [&](int kv, int j, const uint4& val) {
                        uint32_t row = page_row(kv, slot, 16, true);
                        uint32_t addr = stage + (j >> 3) * 4096u + swz(row, j & 7);
                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(val.x), "r"(val.y), "r"(val.z), "r"(val.w) : "memory");
                        if (rec >= 0) {
                            size_t drow = (size_t)rec * 32 + row;
                            reinterpret_cast<uint4*>(a.arena)[drow * (D / 8) + j] = val;
                        }
                    };
                    if constexpr (ROPE) {
                        for (int c = lane; c < 2 * (D / 8); c += 32) {
                            int kv = c / (D / 8), j = c - kv * (D / 8);
                            uint4 val;
                            if (kv == 0) {
                                uint32_t o4[4];
                                rope_k_words<D, BF16, 4>(a.rope, reinterpret_cast<const uint32_t*>(krow), 4 * j, cur.q_pos, inv_rms, o4);
                                val = make_uint4(o4[0], o4[1], o4[2], o4[3]);
                            } else {
                                val = *(reinterpret_cast<const uint4*>(a.v_new) + rowi * (D / 8) + j);
                            }
                            put(kv, j, val);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < NROW; i++) {
                            const int c = lane + 32 * i, kv = c / (D / 8), j = c - kv * (D / 8);
                            if (c >= 2 * (D / 8)) break;
                            put(kv, j, early ? row_new[i] : *(reinterpret_cast<const uint4*>(kv ? a.v_new : a.k_new) + rowi * (D / 8) + j));
                        }
                    }
                    fence_proxy_async();
                    __syncwarp();
                }
                const bool need_mask = (lp * 16 + 15 > cur.q_pos) || (a.window > 0 && lp * 16 + a.window <= cur.q_pos);
                if constexpr (Q8) {
                    if (a.k_new != nullptr && lp == cur.page_last) {
                        // fused append: quantise the new K/V row into the tile just fetched and into its record
                        const int rec = __ldcg(a.unit_row + u);
                        if (rec >= 0) {
                            const size_t rowi = ((size_t)cur.tok_off * Hkv + cur.h) * D;
                            q8_append_row<D, BF16, ROPE>(stage, reinterpret_cast<uint8_t*>(a.arena) + (size_t)rec * UNIT,
                                                   reinterpret_cast<const uint16_t*>(a.k_new) + rowi,
                                                   reinterpret_cast<const uint16_t*>(a.v_new) + rowi, cur.q_pos & 15, lane, a.rope, cur.q_pos);
                        }
                        fence_proxy_async();  // the stage is refilled by the copy engine later
                        __syncwarp();
                    }
                    Q8Tile<D> regs;
                    q8_load<D>(stage, lane, regs);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty0 + st * 8);  // the tile is in registers: the stage may be refilled
#ifdef CBKV_MEASURE
                    q8_attend<D, BF16>(regs, qf, o, m, l, lp * 16, qpos, a.window, a.scale_log2, need_mask, lane, a.debug);
#else
                    q8_attend<D, BF16>(regs, qf, o, m, l, lp * 16, qpos, a.window, a.scale_log2, need_mask, lane);
#endif
                    continue;
                }
                attend_tile<D, 1, BF16>(stage, qf, o, m, l, lp * 16, qpos, a.window, a.scale_log2, need_mask, lane);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + st * 8);  // the stage may be refilled
        }

        // ---- hand this warp's state for the piece to the merger (double-buffered), or leave the CTA's last one to all warps
        const bool late = !nknown;
        if (ALL && late) nhave = get_item(k + 1, nit);  // the entry was not there when the piece began: wait for it now
        const bool last = ALL && !more && !nhave;
        const int buf = NB == 2 ? (kk & 1) : 0, use = NB == 2 ? (kk >> 1) : kk;
        if (vflag[1] != 0) failed = true;  // another warp gave up: stop waiting
        if (use >= 1 && !failed && !mbar_wait_bounded(cempty0 + buf * 8, (use - 1) & 1, 4 * lim)) {
            failed = true;
            if (lane == 0) { atomicOr(a.status, ST_WAIT_TIMEOUT); atomicExch(flag + 1, 1); }
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            l[0][j] += __shfl_xor_sync(0xffffffffu, l[0][j], 4);
            l[0][j] += __shfl_xor_sync(0xffffffffu, l[0][j], 8);
            l[0][j] += __shfl_xor_sync(0xffffffffu, l[0][j], 16);
        }
        float* co = comb_o + ((size_t)buf * C + cw) * ccols * DP;
        float* cml = comb_ml + (buf * C + cw) * 16;
#pragma unroll
        for (int mt = 0; mt < D / 16; mt++) {
            // the d-values behind rows g and g+8 of m-tile mt (permuted for quantised tiles, see q8_attend)
            const int d0 = Q8 ? 32 * (mt >> 1) + 4 * g + 2 * (mt & 1) : mt * 16 + g;
            const int d1 = Q8 ? d0 + 1 : d0 + 8;
            if (2 * t < ccols) {
                co[(2 * t) * DP + d0] = o[0][mt][0];
                co[(2 * t) * DP + d1] = o[0][mt][2];
            }
            if (2 * t + 1 < ccols) {
                co[(2 * t + 1) * DP + d0] = o[0][mt][1];
                co[(2 * t + 1) * DP + d1] = o[0][mt][3];
            }
        }
        if (g == 0) {
            cml[(2 * t) * 2 + 0] = m[0][0]; cml[(2 * t) * 2 + 1] = l[0][0];
            cml[(2 * t + 1) * 2 + 0] = m[0][1]; cml[(2 * t + 1) * 2 + 1] = l[0][1];
        }
        if (last) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(cfull0 + buf * 8);
        kk++;
        if (late) {
            if (!ALL) nhave = get_item(k + 1, nit);
            if (nhave) {
                nseg = nit.z;
                nxt = load_piece(a, nseg);
                if constexpr (Q8) load_q_frags_q8<D>(a, nxt, g, t, qf_next);
                else load_q_frags<D>(a, nxt, g, t, qf_next);
            }
        }
        if (!nhave) break;
        if (more) {
            pb = pe;
        } else {
            // the filler slots up to the next multiple of C (see the producer): this warp owns at most one
            const int n_pad = (n1 + C - 1) / C * C;
            const int Tp = n1 + (cw - n1 % C + C) % C;
            if (Tp < n_pad) {
                const int fs = Tp % NS;
                if (!failed && !mbar_wait_bounded(full0 + fs * 8, (Tp / NS) & 1, lim)) {
                    failed = true;
                    if (lane == 0) { atomicOr(a.status, ST_WAIT_TIMEOUT); atomicExch(flag + 1, 1); }
                }
                __syncwarp();
                if (lane == 0 && !failed) mbar_arrive(empty0 + fs * 8);
            }
            nbase = n_pad;
            k++;
            it = nit;
            pb = it.x;
        }
        seg = nseg;
        cur = nxt;
#pragma unroll
        for (int ks = 0; ks < D / 16; ks++) { qf[0][ks][0] = qf_next[0][ks][0]; qf[0][ks][1] = qf_next[0][ks][1]; }
    }
    if (ALL) {
        const int4* sp = reinterpret_cast<const int4*>(a.segs + seg);
        const int4 x = __ldg(sp), y = __ldg(sp + 1);
        combine_last(seg, x, y, have ? it.z : 0, have ? it.w : 0, NB == 2 ? (kk & 1) : 0);
    }
    // idle now: help merge the segments whose last ticket this CTA drew
    consumer_sync((C + 1) * 32);
    const int n_deferred = flag[2];
    for (int i = 0; i < n_deferred; i++) {
        const int sg = flag[4 + i];
        const int4* sp = reinterpret_cast<const int4*>(a.segs + sg);
        const int4 x = __ldg(sp), y = __ldg(sp + 1);
        uint16_t* out_row = reinterpret_cast<uint16_t*>(a.out) + ((size_t)x.w * a.geo.n_q + (size_t)(sg % Hkv) * n_rep) * D;
        merge_parts<D, BF16>(a, y.y, y.x, out_row, n_rep, cw * 32 + lane, (C + 1) * 32);
    }
}

// ------------------------------------------------------------------ chunk (prefill)
// One warp per item = (sequence, kv head, block of 8*NT query columns); column c of a
// sequence is (new token c / n_rep, q head c % n_rep of the kv group).  Every warp
// streams the pages its columns can see through its own TMA ring.
template <int D, int NT, int W, int S, bool BF16>
__global__ void __launch_bounds__(W * 32) chunk_kernel(const __grid_constant__ CUtensorMap tmap, const ChunkArgs a) {
    constexpr uint32_t UNIT = 32u * D * 2u;
    constexpr int CPI = 8 * NT;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)W * S * UNIT);
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    if ((smem_u32(smem) & 1023u) != 0) {
        if (tid == 0) atomicOr(a.status, ST_SMEM_ALIGN);
        return;
    }
    const int item = blockIdx.x * W + w;
    if (item >= a.n_items) return;
    const uint32_t ring = smem_u32(smem) + (uint32_t)w * S * UNIT;
    const uint32_t bar0 = smem_u32(bars + w * S);
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < S; i++) mbar_init(bar0 + i * 8, 1);
        fence_mbar_init();
        fence_proxy_async();
    }
    __syncwarp();

    int lo = 0, hi = a.step.n_seqs - 1;  // last sequence whose first item is <= item
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (a.item_begin[mid] <= item) lo = mid; else hi = mid - 1;
    }
    const int b = lo;
    const SeqMeta sm = a.step.seq_meta[b];
    const int Hkv = a.geo.n_kv, n_rep = a.geo.n_rep;
    const int ncols = sm.snew * n_rep;
    const int ncb = (ncols + CPI - 1) / CPI;
    const int local = item - a.item_begin[b];
    const int h = local / ncb, cb = local - h * ncb;
    const int c_lo = cb * CPI, c_hi = min(c_lo + CPI, ncols) - 1;
    const int q_min = sm.pos + c_lo / n_rep, q_max = sm.pos + c_hi / n_rep;
    const int lo_key = a.window > 0 ? max(0, q_min - a.window + 1) : 0;
    const int p_lo = lo_key >> 4, p_hi = q_max >> 4;
    const size_t blk = (size_t)sm.tok_off * a.geo.n_q;  // first packed q row of this sequence

    uint32_t qf[NT][D / 16][2];
    int qpos[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        int c = c_lo + nt * 8 + g;  // the column this lane feeds into the B operand
        bool ok = c < ncols;
        int r = ok ? c / n_rep : 0, rep = ok ? c - r * n_rep : 0;
        const uint32_t* qrow = reinterpret_cast<const uint32_t*>(
            reinterpret_cast<const uint16_t*>(a.q) + (blk + (size_t)(h * n_rep + rep) * sm.snew + r) * D);
#pragma unroll
        for (int ks = 0; ks < D / 16; ks++) {
            qf[nt][ks][0] = ok ? __ldg(qrow + ks * 8 + t) : 0u;
            qf[nt][ks][1] = ok ? __ldg(qrow + ks * 8 + 4 + t) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            int cc = min(c_lo + nt * 8 + 2 * t + j, ncols - 1);  // columns past the end mimic the last one
            qpos[nt][j] = sm.pos + cc / n_rep;
        }
    }
    float o[NT][D / 16][4], m[NT][2], l[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        m[nt][0] = m[nt][1] = -INFINITY; l[nt][0] = l[nt][1] = 0.f;
#pragma unroll
        for (int mt = 0; mt < D / 16; mt++) { o[nt][mt][0] = o[nt][mt][1] = o[nt][mt][2] = o[nt][mt][3] = 0.f; }
    }

    auto issue = [&](int lp, int stage_idx) {
        if (lane == 0) {
            int phys = a.step.tables[sm.tbl_off + lp];
            if (phys < 0 || phys >= a.geo.num_pages) { atomicOr(a.status, ST_BAD_PAGE); phys = 0; }
            issue_tile<D>(&tmap, ring + stage_idx * UNIT, bar0 + stage_idx * 8, (phys * Hkv + h) * 32);
        }
    };
    int next = p_lo;
#pragma unroll 1
    for (int i = 0; i < S && next <= p_hi; i++, next++) issue(next, i);
    bool failed = false;
    int consumed = 0, issued = next - p_lo, fail_at = 0;
#pragma unroll 1
    for (int lp = p_lo; lp <= p_hi; lp++) {
        const int st = consumed % S;
        if (!failed && !mbar_wait_bounded(bar0 + st * 8, (consumed / S) & 1)) {
            failed = true;
            fail_at = consumed;
            atomicOr(a.status, ST_WAIT_TIMEOUT);
        }
        if (!failed) {
            const bool need_mask = (lp * 16 + 15 > q_min) || (a.window > 0 && lp * 16 + a.window <= q_max);
            attend_tile<D, NT, BF16>(ring + st * UNIT, qf, o, m, l, lp * 16, qpos, a.window, a.scale_log2, need_mask, lane);
        }
        __syncwarp();
        consumed++;
        if (next <= p_hi) { if (!failed) { issue(next, st); issued++; } next++; }
    }
    if (failed) {  // wait (bounded) for the copies still in flight, then leave without storing
        for (int i = fail_at; i < issued; i++) mbar_wait_bounded(bar0 + (i % S) * 8, (i / S) & 1, 20000000ull);
        return;
    }

#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            float ls = l[nt][j];
            ls += __shfl_xor_sync(0xffffffffu, ls, 4);
            ls += __shfl_xor_sync(0xffffffffu, ls, 8);
            ls += __shfl_xor_sync(0xffffffffu, ls, 16);
            int c = c_lo + nt * 8 + 2 * t + j;
            if (c < ncols) {
                int r = c / n_rep, rep = c - r * n_rep;
                uint16_t* orow = reinterpret_cast<uint16_t*>(a.out) + (blk + (size_t)(h * n_rep + rep) * sm.snew + r) * D;
                float inv = 1.f / ls;
#pragma unroll
                for (int mt = 0; mt < D / 16; mt++) {
                    orow[mt * 16 + g] = to_elem<BF16>(o[nt][mt][j] * inv);
                    orow[mt * 16 + g + 8] = to_elem<BF16>(o[nt][mt][j + 2] * inv);
                }
            }
        }
    }
}

// ------------------------------------------------------------------ generic
// Any page size and head_dim (multiple of 8, <= 512); one warp per query row.
template <bool BF16>
__global__ void generic_kernel(const GenericArgs a) {
    __shared__ float qs[4][512];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t rid = (int64_t)blockIdx.x * 4 + w;  // packed q row: sequence blocks of [n_q][snew]
    if (rid >= (int64_t)a.step.n_tokens * a.geo.n_q) return;
    const int D = a.geo.d, P = a.geo.page_size, Hkv = a.geo.n_kv;
    int lo = 0, hi = a.step.n_seqs - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if ((int64_t)a.step.seq_meta[mid].tok_off * a.geo.n_q <= rid) lo = mid; else hi = mid - 1;
    }
    const SeqMeta sm = a.step.seq_meta[lo];
    const int64_t local = rid - (int64_t)sm.tok_off * a.geo.n_q;
    const int hq = (int)(local / sm.snew), r = (int)(local % sm.snew);
    const int h = hq / a.geo.n_rep;  // repeat_kv: q head i reads kv head i / n_rep, kv.rs:177-187
    const int q_pos = sm.pos + r;
    const uint16_t* q = reinterpret_cast<const uint16_t*>(a.q) + rid * D;
    for (int j = lane; j < D; j += 32) qs[w][j] = from_elem<BF16>(q[j]);
    __syncwarp();
    const uint16_t* arena = reinterpret_cast<const uint16_t*>(a.arena);
    const int t_lo = a.window > 0 ? max(0, q_pos - a.window + 1) : 0;
    float m = -INFINITY, l = 0.f, acc[16];
#pragma unroll
    for (int i = 0; i < 16; i++) acc[i] = 0.f;
    for (int t0 = t_lo; t0 <= q_pos; t0 += 32) {
        const int tk = t0 + lane;
        const bool ok = tk <= q_pos;
        float s = -INFINITY;
        if (ok) {
            int phys = a.step.tables[sm.tbl_off + tk / P];
            if (phys < 0 || phys >= a.geo.num_pages) { atomicOr(a.status, ST_BAD_PAGE); phys = 0; }
            const uint16_t* krow = arena + ((((int64_t)phys * Hkv + h) * 2 + 0) * P + tk % P) * D;
            float d = 0.f;
            for (int j = 0; j < D; j++) d += qs[w][j] * from_elem<BF16>(krow[j]);
            s = d * a.scale;
        }
        float mx = s;
        for (int off = 16; off; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const float m_new = fmaxf(m, mx);
        const float alpha = __expf(m - m_new);
        const float p = ok ? __expf(s - m_new) : 0.f;
        float ps = p;
        for (int off = 16; off; off >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, off);
        l = l * alpha + ps;
        m = m_new;
#pragma unroll
        for (int i = 0; i < 16; i++) acc[i] *= alpha;
        const int cnt = min(32, q_pos - t0 + 1);
        for (int kk = 0; kk < cnt; kk++) {
            const float pk = __shfl_sync(0xffffffffu, p, kk);
            const int tv = t0 + kk;
            int phys = a.step.tables[sm.tbl_off + tv / P];
            if (phys < 0 || phys >= a.geo.num_pages) phys = 0;
            const uint16_t* vrow = arena + ((((int64_t)phys * Hkv + h) * 2 + 1) * P + tv % P) * D;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                int j = lane + 32 * i;
                if (j < D) acc[i] += pk * from_elem<BF16>(vrow[j]);
            }
        }
    }
    uint16_t* orow = reinterpret_cast<uint16_t*>(a.out) + rid * D;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        int j = lane + 32 * i;
        if (j < D) orow[j] = to_elem<BF16>(acc[i] / l);
    }
}

// ------------------------------------------------------------------ launchers
// default consumer warps per CTA (C8: over int8 pages) and CTAs per SM of the decode kernel
template <int D> struct DecodeCfg;
template <> struct DecodeCfg<64>  { static constexpr int C = 6, C8 = 4, CTAS = 1; };
template <> struct DecodeCfg<128> { static constexpr int C = 6, C8 = 4, CTAS = 1; };
template <> struct DecodeCfg<256> { static constexpr int C = 6, C8 = 6, CTAS = 1; };

static int decode_smem_bytes(int d, int consumers, int stages, int comb_cols, int comb_bufs, bool q8 = false) {
    const int unit = q8 ? (int)qrec_bytes(16, d) : 32 * d * 2;
    return stages * unit + comb_bufs * (consumers * comb_cols * (d + 4) * 4 + consumers * 16 * 4) + QN * 16 +
           (2 * stages + 4 + 2 * QN) * 8 + (4 + DEFER_CAP) * 4;
}

template <int D> struct ChunkCfg;
template <> struct ChunkCfg<64>  { static constexpr int W = 4, S = 4, NT = 4; };
template <> struct ChunkCfg<128> { static constexpr int W = 4, S = 3, NT = 2; };
template <> struct ChunkCfg<256> { static constexpr int W = 4, S = 2, NT = 1; };

template <int D> constexpr int chunk_smem() { return ChunkCfg<D>::W * ChunkCfg<D>::S * 32 * D * 2 + ChunkCfg<D>::W * ChunkCfg<D>::S * 8; }

template <int D, int C, bool BF16, bool Q8>
static int decode_resident() {
    static const int n = [] {  // asked once
        int r = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, decode_kernel<D, C, BF16, Q8, false>, (C + 2) * 32, 0) == cudaSuccess) return std::max(r, 1);
        cudaGetLastError();  // no device: nothing will be launched
        return 8;
    }();
    return n;
}
template <int D, bool BF16, bool Q8>
static int decode_resident(int consumers) {
    return consumers == 4 ? decode_resident<D, 4, BF16, Q8>() : consumers == 6 ? decode_resident<D, 6, BF16, Q8>() : consumers == 8 ? decode_resident<D, 8, BF16, Q8>() : decode_resident<D, 12, BF16, Q8>();
}
// CTAs of the decode kernel whose registers an SM holds at a time.  The variants over 16-bit pages are compiled for one (176
// registers at head_dim 128): two CTAs per SM that do not fit share the ring's memory and run one after the other (28 layers of 32
// sequences, two steps, 28/4/128: 3700 us; 2320 with 128 registers and both resident, 1840 with one).
static int decode_resident(int d, int consumers, bool q8) {
    auto least = [&](auto f, auto b) { return std::min(f(consumers), b(consumers)); };
    switch (d) {
        case 64: return q8 ? least(decode_resident<64, false, true>, decode_resident<64, true, true>) : least(decode_resident<64, false, false>, decode_resident<64, true, false>);
        case 128: return q8 ? least(decode_resident<128, false, true>, decode_resident<128, true, true>) : least(decode_resident<128, false, false>, decode_resident<128, true, false>);
        default: return q8 ? least(decode_resident<256, false, true>, decode_resident<256, true, true>) : least(decode_resident<256, false, false>, decode_resident<256, true, false>);
    }
}

// Stage count: the largest multiple of the consumer count that fits next to the merge
// buffers when `ctas_per_sm` CTAs share the SM's shared memory (1 KB per CTA is
// reserved by the system), at most 8 stages per consumer.  Bytes in flight matter
// more than a second merge buffer: the merge area is double-buffered only when that
// costs no stage.
DecodeConfig decode_config(int d, int n_rep, int ctas_per_sm, int stages, int consumers, bool q8) {
    int c, ctas;
    switch (d) {
        case 64: c = DecodeCfg<64>::C; ctas = DecodeCfg<64>::CTAS; break;
        case 128: c = DecodeCfg<128>::C; ctas = DecodeCfg<128>::CTAS; break;
        case 256: c = DecodeCfg<256>::C; ctas = DecodeCfg<256>::CTAS; break;
        default: return {0, 0, 0, 0, 0, 0};
    }
    // int8 tiles are bound by the consumer warps' arithmetic, not by bytes in flight: two CTAs of four consumer
    // warps per SM (each with its own ring, producer and merger) let one CTA's set-up and merge run under the
    // other's tiles; measured 0.80 ms per cfg2 step against 0.85 with one CTA of eight
    if (q8 && d <= 128) { c = DecodeCfg<128>::C8; ctas = 2; }
    if (consumers == 4 || consumers == 6 || consumers == 8 || (consumers == 12 && d <= 128)) c = consumers;  // 12 warps of head_dim 256 spill
    if (ctas_per_sm > 0) ctas = ctas_per_sm == 1 ? 1 : std::min(ctas_per_sm, decode_resident(d, c, q8));
    const int comb_cols = std::min(8, (n_rep + 1) & ~1);
    const int smem_limit = std::min(227 * 1024, (228 * 1024) / ctas - 1024);
    if (stages <= 0) {
        stages = 8 * c;
        while (stages > c && decode_smem_bytes(d, c, stages, comb_cols, 1, q8) > smem_limit) stages -= c;
    }
    stages = std::max(c, (stages / c) * c);
    const int bufs = decode_smem_bytes(d, c, stages, comb_cols, 2, q8) <= smem_limit ? 2 : 1;
    return {c, stages, decode_smem_bytes(d, c, stages, comb_cols, bufs, q8), ctas, comb_cols, bufs};
}
// The launch that is saved is worth about 4 us a layer; what it costs is the norm and rotation of q in every consumer warp of
// every piece, and of k in the one that holds the new row, so it grows with the segments that an SM works through.  Measured
// us per layer, inside / two launches, 1 to 128 sequences x 2 to 16 kv heads after 300 to 16000 tokens.  Rotation alone, 16
// bits: faster throughout (1024 segments of head_dim 128 39 / 42, one sequence 7.9 / 14).  int8 pages: head_dim 128 faster
// up to 512 segments (28 / 32), equal at 1024; 256 faster at 128 (26 / 28), slower at 512 (72 / 67).  With a norm: head_dim
// 64 faster up to 384 (22 / 23, int8 24 / 26), slower at 1024 (43 / 38); 128 faster up to 256 (21 / 23), slower at 384 (27
// / 25), int8 equal at 128 (20 / 20), slower at 192 (23 / 22); 256 faster up to 128 (22 / 23), slower at 256 (34 / 29), int8
// slower from the first (21 / 19).
bool decode_rotates(int d, int consumers, bool q8, bool norm, int64_t n_segs, int sm_count) {
    constexpr int64_t ANY = (int64_t)1 << 30;
    int default_consumers;
    int64_t per_sm;  // most segments per SM
    switch (d) {
        case 64: default_consumers = q8 ? DecodeCfg<64>::C8 : DecodeCfg<64>::C; per_sm = norm ? 3 : ANY; break;
        case 128: default_consumers = q8 ? DecodeCfg<128>::C8 : DecodeCfg<128>::C; per_sm = norm ? (q8 ? 1 : 2) : (q8 ? 5 : ANY); break;
        case 256: default_consumers = q8 ? DecodeCfg<256>::C8 : DecodeCfg<256>::C; per_sm = norm ? (q8 ? 0 : 1) : (q8 ? 1 : ANY); break;
        default: return false;
    }
    return consumers == default_consumers && n_segs <= per_sm * sm_count;
}
ChunkConfig chunk_config(int d) {
    switch (d) {
        case 64: return {ChunkCfg<64>::W, ChunkCfg<64>::S, chunk_smem<64>(), 8 * ChunkCfg<64>::NT};
        case 128: return {ChunkCfg<128>::W, ChunkCfg<128>::S, chunk_smem<128>(), 8 * ChunkCfg<128>::NT};
        case 256: return {ChunkCfg<256>::W, ChunkCfg<256>::S, chunk_smem<256>(), 8 * ChunkCfg<256>::NT};
        default: return {0, 0, 0, 0};
    }
}

template <int D, bool BF16> static cudaError_t set_attrs() {
    cudaError_t e;
    e = cudaFuncSetAttribute(decode_kernel<D, 4, BF16, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(decode_kernel<D, 6, BF16, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(decode_kernel<D, 8, BF16, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(decode_kernel<D, 4, BF16, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(decode_kernel<D, 6, BF16, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(decode_kernel<D, 8, BF16, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(decode_kernel<D, 12, BF16, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(decode_kernel<D, 12, BF16, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(decode_kernel<D, DecodeCfg<D>::C, BF16, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(decode_kernel<D, DecodeCfg<D>::C8, BF16, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(chunk_kernel<D, ChunkCfg<D>::NT, ChunkCfg<D>::W, ChunkCfg<D>::S, BF16>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, chunk_smem<D>());
}

cudaError_t kernels_init() {
    cudaError_t e;
    if ((e = set_attrs<64, false>()) != cudaSuccess) return e;
    if ((e = set_attrs<64, true>()) != cudaSuccess) return e;
    if ((e = set_attrs<128, false>()) != cudaSuccess) return e;
    if ((e = set_attrs<128, true>()) != cudaSuccess) return e;
    if ((e = set_attrs<256, false>()) != cudaSuccess) return e;
    if ((e = set_attrs<256, true>()) != cudaSuccess) return e;
    return cudaSuccess;
}

cudaError_t launch_append(const AppendArgs& a, bool bf16, bool overlap, cudaStream_t st) {
    (void)bf16;  // a bit copy: the element type does not matter
    int64_t total = (int64_t)a.step.n_tokens * a.geo.n_kv * 2 * (a.geo.d / 8);
    int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 8);
    if (blocks <= 0) return cudaSuccess;
    return launch_pdl(overlap, append_kernel<uint16_t>, blocks, 256, 0, st, a);
}

template <int D, int C, bool BF16, bool Q8, bool ROPE = false>
static cudaError_t launch_decode_t(const CUtensorMap& map, const DecodeArgs& a, int n_ctas, int smem, bool pdl, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)n_ctas);
    cfg.blockDim = dim3((C + 2) * 32);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, decode_kernel<D, C, BF16, Q8, ROPE>, map, a);
}

template <int D, bool BF16, bool Q8>
static cudaError_t launch_decode_c(const CUtensorMap& map, const DecodeArgs& a, int n_ctas, int consumers, int smem, bool pdl, cudaStream_t st) {
    constexpr int C = Q8 ? DecodeCfg<D>::C8 : DecodeCfg<D>::C;
    if (a.rope.table) return consumers == C ? launch_decode_t<D, C, BF16, Q8, true>(map, a, n_ctas, smem, pdl, st) : cudaErrorInvalidValue;
    switch (consumers) {
        case 4: return launch_decode_t<D, 4, BF16, Q8>(map, a, n_ctas, smem, pdl, st);
        case 6: return launch_decode_t<D, 6, BF16, Q8>(map, a, n_ctas, smem, pdl, st);
        case 8: return launch_decode_t<D, 8, BF16, Q8>(map, a, n_ctas, smem, pdl, st);
        case 12: return launch_decode_t<D, 12, BF16, Q8>(map, a, n_ctas, smem, pdl, st);
        default: return cudaErrorInvalidValue;
    }
}
template <int D>
static cudaError_t launch_decode_d(const CUtensorMap& map, const DecodeArgs& a, int n_ctas, int consumers, int smem, bool pdl, bool bf16, bool q8, cudaStream_t st) {
    if (q8) return bf16 ? launch_decode_c<D, true, true>(map, a, n_ctas, consumers, smem, pdl, st) : launch_decode_c<D, false, true>(map, a, n_ctas, consumers, smem, pdl, st);
    return bf16 ? launch_decode_c<D, true, false>(map, a, n_ctas, consumers, smem, pdl, st) : launch_decode_c<D, false, false>(map, a, n_ctas, consumers, smem, pdl, st);
}

cudaError_t launch_decode(const CUtensorMap& map, const DecodeArgs& a, int n_ctas, int consumers, int smem, bool pdl, bool bf16, cudaStream_t st, bool q8) {
    if (a.n_stages < consumers || a.n_stages % consumers != 0) return cudaErrorInvalidValue;
    switch (a.geo.d) {
        case 64: return launch_decode_d<64>(map, a, n_ctas, consumers, smem, pdl, bf16, q8, st);
        case 128: return launch_decode_d<128>(map, a, n_ctas, consumers, smem, pdl, bf16, q8, st);
        case 256: return launch_decode_d<256>(map, a, n_ctas, consumers, smem, pdl, bf16, q8, st);
        default: return cudaErrorInvalidValue;
    }
}

template <int D, bool BF16>
static cudaError_t launch_chunk_t(const CUtensorMap& map, const ChunkArgs& a, cudaStream_t st) {
    int blocks = (a.n_items + ChunkCfg<D>::W - 1) / ChunkCfg<D>::W;
    if (blocks <= 0) return cudaSuccess;
    chunk_kernel<D, ChunkCfg<D>::NT, ChunkCfg<D>::W, ChunkCfg<D>::S, BF16><<<blocks, ChunkCfg<D>::W * 32, chunk_smem<D>(), st>>>(map, a);
    return cudaGetLastError();
}

cudaError_t launch_chunk(const CUtensorMap& map, const ChunkArgs& a, bool bf16, cudaStream_t st) {
    switch (a.geo.d) {
        case 64: return bf16 ? launch_chunk_t<64, true>(map, a, st) : launch_chunk_t<64, false>(map, a, st);
        case 128: return bf16 ? launch_chunk_t<128, true>(map, a, st) : launch_chunk_t<128, false>(map, a, st);
        case 256: return bf16 ? launch_chunk_t<256, true>(map, a, st) : launch_chunk_t<256, false>(map, a, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_resolve_units(const SegInfo* segs, int n_segs, const int32_t* tables, int n_kv, int num_pages,
                                 int32_t* unit_row, int n_units, int32_t* status, cudaStream_t st,
                                 int32_t* zero_a, int n_a, int32_t* zero_b, int n_b) {
    if (!zero_a) n_a = 0;
    if (!zero_b) n_b = 0;
    if (n_units <= 0 && n_a <= 0 && n_b <= 0) return cudaSuccess;
    const int blocks = std::max(1, std::min((std::max(n_units, n_a) + 255) / 256, 148 * 4));
    resolve_units_kernel<<<blocks, 256, 0, st>>>(segs, n_segs, tables, n_kv, num_pages, unit_row, n_units, status, zero_a, n_a, zero_b, n_b);
    return cudaGetLastError();
}

cudaError_t launch_generic(const GenericArgs& a, bool bf16, cudaStream_t st) {
    int64_t rows = (int64_t)a.step.n_tokens * a.geo.n_q;
    int blocks = (int)((rows + 3) / 4);
    if (blocks <= 0) return cudaSuccess;
    if (bf16) generic_kernel<true><<<blocks, 128, 0, st>>>(a);
    else generic_kernel<false><<<blocks, 128, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace cbkv
