// int8 KV pages: CacheConfig::quantize_kv of the reference (kv.rs:271-358, 464-475, 740-787).
//
//   append_quant_kernel    kv_quantize (kv.rs:284-313) fused with the page scatter
//                          (kv.rs:746-768): per 32-value group scale = max(absmax/127, 1e-8)
//                          in f32, q = clamp(round(x/scale), -127, 127), one byte q + 128 per
//                          value, scale kept in the element type
//   generic_quant_kernel   attention over quantised pages for any shape: kv_dequantize
//                          (kv.rs:319-358) happens on the fly, value = elem(q * scale), f32 math
//
// One record per (page, kv head), laid out for the decode kernel (qrec_* in kernels.hpp),
// so a decode step reads d + d/16 bytes per cached token and head instead of 2d.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "kernels.hpp"
#include "pdl.cuh"
#include "q8_unpack.cuh"

namespace cbkv {

namespace {

template <bool BF16> __device__ __forceinline__ float q_up(uint16_t v) {
    if (BF16) return __bfloat162float(__ushort_as_bfloat16(v));
    return __half2float(__ushort_as_half(v));
}
template <bool BF16> __device__ __forceinline__ uint16_t q_down(float f) {
    if (BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(f));
    return __half_as_ushort(__float2half_rn(f));
}

template <bool BF16>
__global__ void __launch_bounds__(256) append_quant_kernel(const AppendArgs a) {
    const int lane = threadIdx.x & 31;
    const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int d = a.geo.d, P = a.geo.page_size, Hkv = a.geo.n_kv;
    const int words = d >> 2;                                  // 4 values per packed word
    const int64_t kv_rows = (int64_t)a.step.n_tokens * Hkv;
    uint8_t* arena = reinterpret_cast<uint8_t*>(a.arena);
    const size_t rec = qrec_bytes(P, d);
    struct Place { uint8_t* recp; int slot; };  // null: the table entry is not a page
    auto place_of = [&](int64_t R) -> Place {
        const int64_t row = R >= kv_rows ? R - kv_rows : R;
        int lo = 0, hi = a.step.n_seqs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((int64_t)a.step.seq_meta[mid].tok_off * Hkv <= row) lo = mid; else hi = mid - 1;
        }
        const SeqMeta sm = a.step.seq_meta[lo];
        const int64_t local = row - (int64_t)sm.tok_off * Hkv;
        const int h = (int)(local / sm.snew), r = (int)(local - (int64_t)h * sm.snew);
        const int gpos = sm.pos + r;                            // kv.rs:749
        const int phys = a.step.tables[sm.tbl_off + gpos / P];  // kv.rs:752
        if (phys < 0 || phys >= a.geo.num_pages) { if (lane == 0) atomicOr(a.status, ST_BAD_PAGE); return {nullptr, 0}; }
        return {arena + ((size_t)phys * Hkv + h) * rec, gpos % P};  // kv.rs:750
    };
    // the first row's look-up runs under the tail of the launch before: the records and block tables came with the step's
    // upload, which no kernel overlaps
    Place next{nullptr, 0};
    if (warp0 < 2 * kv_rows) next = place_of(warp0);
    pdl_wait();
    pdl_launch_dependents();
    for (int64_t R = warp0; R < 2 * kv_rows; R += nwarps) {
        const int is_v = R >= kv_rows;
        const int64_t row = is_v ? R - kv_rows : R;
        if (R != warp0) next = place_of(R);
        uint8_t* recp = next.recp;
        const int slot = next.slot;
        if (recp == nullptr) continue;
        const uint2* src = reinterpret_cast<const uint2*>(is_v ? a.v : a.k) + row * words;
        // every lane runs every round (the shuffles below name the full warp)
        for (int c0 = 0; c0 < words; c0 += 32) {
            const int c = c0 + lane;
            const bool live = c < words;
            float x[4] = {0.f, 0.f, 0.f, 0.f};
            if (live) {
                const uint2 raw = src[c];
                x[0] = q_up<BF16>((uint16_t)(raw.x & 0xffff)); x[1] = q_up<BF16>((uint16_t)(raw.x >> 16));
                x[2] = q_up<BF16>((uint16_t)(raw.y & 0xffff)); x[3] = q_up<BF16>((uint16_t)(raw.y >> 16));
            }
            float amax = fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fmaxf(fabsf(x[2]), fabsf(x[3])));
            // a group is 32 values = 8 consecutive lanes
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
            const float scale = fmaxf(__fdiv_rn(amax, 127.0f), 1e-8f);   // kv.rs:296-301
            if (live) {
                uint32_t word = 0;  // four bytes q + 128
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    float q = roundf(__fdiv_rn(x[i], scale));             // kv.rs:302-305
                    q = fminf(fmaxf(q, -127.f), 127.f);
                    word |= (uint32_t)((int)q + 128) << (8 * i);
                }
                if (!is_v) {
                    *reinterpret_cast<uint32_t*>(recp + qrec_value_off(0, slot, 4 * c, P, d)) = word;
                } else {  // the pair's other token sits between these bytes
#pragma unroll
                    for (int i = 0; i < 4; i++) recp[qrec_value_off(1, slot, 4 * c + i, P, d)] = (uint8_t)(word >> (8 * i));
                }
                if ((c & 7) == 0)
                    *reinterpret_cast<uint16_t*>(recp + qrec_scale_off(is_v, slot, c >> 3, P, d)) = q_down<BF16>(scale);
            }
        }
    }
}

// 16 consecutive values of a row (half a group): bytes q + 128, four to a word, and the group's scale, which the lane next
// door has the other half of.
template <bool BF16>
__device__ __forceinline__ float quantise16(const uint4& x0, const uint4& x1, uint32_t (&bytes)[4]) {
    const uint32_t w[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
    float v[16], amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        v[2 * i] = q_up<BF16>((uint16_t)(w[i] & 0xffff));
        v[2 * i + 1] = q_up<BF16>((uint16_t)(w[i] >> 16));
        amax = fmaxf(amax, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    const float scale = fmaxf(__fdiv_rn(amax, 127.0f), 1e-8f);        // kv.rs:296-301
#pragma unroll
    for (int i = 0; i < 4; i++) {
        bytes[i] = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float q = roundf(__fdiv_rn(v[4 * i + j], scale));         // kv.rs:302-305
            q = fminf(fmaxf(q, -127.f), 127.f);
            bytes[i] |= (uint32_t)((int)q + 128) << (8 * j);
        }
    }
    return scale;
}

// The same for 16-token pages and head_dim 64, 128 or 256: T = d / 16 lanes share a row, each takes 16 consecutive values,
// and V goes two tokens at a time, because the bytes of a pair of tokens alternate in a record: 32 contiguous bytes per
// lane, and one word for the pair's two scales, instead of single bytes.  A pair with only one token in this step (a
// sequence's first or last) leaves the other's bytes alone.
template <bool BF16, int T>
__global__ void __launch_bounds__(256) append_quant_vec_kernel(const AppendArgs a) {
    constexpr int D = T * 16, P = 16, RPW = 32 / T;
    constexpr int SEQ_SMEM = 1024;
    __shared__ int s_tok[SEQ_SMEM];
    const int n_seqs = a.step.n_seqs, Hkv = a.geo.n_kv;
    const bool in_smem = n_seqs <= SEQ_SMEM;
    if (in_smem) {  // the sequence records came with the step's upload, which no kernel overlaps
        for (int i = threadIdx.x; i < n_seqs; i += blockDim.x) s_tok[i] = a.step.seq_meta[i].tok_off;
        __syncthreads();
    }
    pdl_wait();
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, t = lane % T, sub = lane / T;
    const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    // K rows first, then slots for V pairs: n / 2 + 1 or one more per (sequence, kv head), so that a sequence's first
    // slot follows from the tokens before it; a slot past the sequence's last pair has nothing to do
    const int64_t k_rows = (int64_t)a.step.n_tokens * Hkv, v_slots = ((int64_t)a.step.n_tokens / 2 + n_seqs) * Hkv;
    const int64_t k_rounds = (k_rows + RPW - 1) / RPW, rounds = k_rounds + (v_slots + RPW - 1) / RPW;
    uint8_t* arena = reinterpret_cast<uint8_t*>(a.arena);
    const size_t rec = qrec_bytes(P, D);
    auto tok_off = [&](int b) { return in_smem ? s_tok[b] : a.step.seq_meta[b].tok_off; };
    for (int64_t R = warp0; R < rounds; R += nwarps) {
        const bool is_v = R >= k_rounds;  // the same for the whole warp
        const int64_t idx = (is_v ? R - k_rounds : R) * RPW + sub;
        bool live = idx < (is_v ? v_slots : k_rows);
        auto first = [&](int b) { return is_v ? ((int64_t)tok_off(b) / 2 + b) * Hkv : (int64_t)tok_off(b) * Hkv; };
        int lo = 0, hi = n_seqs - 1;  // the last sequence whose first row (slot) is <= idx
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first(mid) <= idx) lo = mid; else hi = mid - 1;
        }
        const SeqMeta sm = a.step.seq_meta[lo];
        const int local = (int)(idx - first(lo));
        const int per = is_v ? (sm.tok_off + sm.snew) / 2 - sm.tok_off / 2 + 1 : sm.snew;  // rows or slots per kv head
        const int h = per > 0 ? local / per : 0;
        int r = local - h * per;                                         // K: the token
        if (is_v) r = 2 * (sm.pos / 2 + r) - sm.pos;                     // V: the pair's first token, -1 when that one is cached already
        const bool has0 = r >= 0 && r < sm.snew, has1 = is_v && r + 1 < sm.snew;
        live = live && h < Hkv && (has0 || has1);
        const int gpos = sm.pos + r;                                     // kv.rs:749
        int phys = live ? a.step.tables[sm.tbl_off + gpos / P] : 0;      // kv.rs:752
        if (live && (phys < 0 || phys >= a.geo.num_pages)) { if (t == 0) atomicOr(a.status, ST_BAD_PAGE); live = false; }
        const int slot = gpos & (P - 1);                                 // kv.rs:750
        const size_t row = (size_t)sm.tok_off * Hkv + (size_t)h * sm.snew;
        const uint4* src = reinterpret_cast<const uint4*>(is_v ? a.v : a.k) + (int64_t)(row * (2 * T)) + (int64_t)r * (2 * T) + 2 * t;
        const uint4 zero = make_uint4(0, 0, 0, 0);
        uint4 x0 = zero, x1 = zero, y0 = zero, y1 = zero;
        if (live && has0) { x0 = src[0]; x1 = src[1]; }
        if (live && has1) { y0 = src[2 * T]; y1 = src[2 * T + 1]; }
        uint32_t bx[4], by[4];
        const float sx = quantise16<BF16>(x0, x1, bx);
        uint8_t* recp = arena + ((size_t)(live ? phys : 0) * Hkv + (live ? h : 0)) * rec;
        const int j0 = 16 * t, grp = j0 >> 5;
        if (!is_v) {
            if (live) {
                *reinterpret_cast<uint4*>(recp + qrec_value_off(0, slot, j0, P, D)) = make_uint4(bx[0], bx[1], bx[2], bx[3]);
                if ((t & 1) == 0) *reinterpret_cast<uint16_t*>(recp + qrec_scale_off(0, slot, grp, P, D)) = q_down<BF16>(sx);
            }
            continue;
        }
        const float sy = quantise16<BF16>(y0, y1, by);
        if (!live) continue;
        if (has0 && has1) {
            uint32_t o[8];  // byte 2 i of the first token's value, 2 i + 1 of the second's
#pragma unroll
            for (int i = 0; i < 4; i++) {
                o[2 * i] = __byte_perm(bx[i], by[i], 0x5140);
                o[2 * i + 1] = __byte_perm(bx[i], by[i], 0x7362);
            }
            uint4* dst = reinterpret_cast<uint4*>(recp + qrec_value_off(1, slot, j0, P, D));
            dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
            dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
            if ((t & 1) == 0)
                *reinterpret_cast<uint32_t*>(recp + qrec_scale_off(1, slot, grp, P, D)) = (uint32_t)q_down<BF16>(sx) | ((uint32_t)q_down<BF16>(sy) << 16);
        } else {
            const int s1 = has0 ? slot : slot + 1;  // r = -1: the pair's second token, in the same page
#pragma unroll
            for (int i = 0; i < 16; i++)
                recp[qrec_value_off(1, s1, j0 + i, P, D)] = (uint8_t)((has0 ? bx[i >> 2] : by[i >> 2]) >> (8 * (i & 3)));
            if ((t & 1) == 0) *reinterpret_cast<uint16_t*>(recp + qrec_scale_off(1, s1, grp, P, D)) = q_down<BF16>(has0 ? sx : sy);
        }
    }
}

// A fresh quantised arena reads as the reference's zero-filled one (kv.rs:699-705): packed words 0
// mean q = -128 in lanes 0-2 and q = 0 in lane 3, i.e. record bytes 0, 0, 0, 0x80; scales 0.
__global__ void init_quant_kernel(uint8_t* arena, size_t n_records, int P, int d) {
    const size_t rec = qrec_bytes(P, d), values = (size_t)2 * P * d;
    const size_t words = n_records * (rec / 4);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / (rec / 4), w = i - r * (rec / 4), off = w * 4;
        uint32_t v = 0;
        if (off < (size_t)P * d) v = 0x80000000u;                  // K: lane 3 is the top byte of each word
        else if (off < values) v = (w & 1) ? 0x80800000u : 0u;      // V: lane 3 of both tokens = bytes 6, 7 of each 8
        reinterpret_cast<uint32_t*>(arena)[i] = v;
    }
}

// kv_dequantize (kv.rs:319-358) of every page the step's sequences hold, into a float layer in the tiled
// row order, so that the tensor-core chunk kernels can run over an int8 layer.  One warp per
// (block-table entry, kv head): value = elem(q * scale), exactly what the reference's gather produces.
template <bool BF16>
__global__ void __launch_bounds__(256) dequant_pages_kernel(const int32_t* tables, int n_entries, GeomDev geo, const uint8_t* arena,
                                                            uint16_t* scratch, int32_t* status) {
    const int lane = threadIdx.x & 31;
    const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    pdl_wait();
    pdl_launch_dependents();
    const int D = geo.d, P = geo.page_size, Hkv = geo.n_kv, G = D / 32;
    const size_t rec = qrec_bytes(P, D);
    const int k_chunks = P * D / 16, sw = qrec_swizzled(D) ? 1 : 0;
    const bool tiled = geo.tiled != 0;
    for (int64_t it = warp0; it < (int64_t)n_entries * Hkv; it += nwarps) {
        const int e = (int)(it / Hkv), h = (int)(it - (int64_t)e * Hkv);
        const int phys = tables[e];
        if (phys < 0 || phys >= geo.num_pages) { if (lane == 0) atomicOr(status, ST_BAD_PAGE); continue; }
        const uint8_t* recp = arena + ((size_t)phys * Hkv + h) * rec;
        const uint16_t* ksc = reinterpret_cast<const uint16_t*>(recp + (size_t)2 * P * D);
        const uint32_t* vsc = reinterpret_cast<const uint32_t*>(ksc + P * G);  // group-major: one word = two neighbouring tokens
        uint16_t* dst = scratch + ((size_t)phys * Hkv + h) * 2 * P * D;
        // a lane takes 16-byte pieces of the record as they lie (coalesced) and works out which values they hold
        for (int c = lane; c < 2 * k_chunks; c += 32) {
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(recp) + c);
            if (c < k_chunks) {  // K: 16 consecutive d of one token, inside one 32-value group (qrec_value_off)
                const int off = c * 16, slot = off / D, pos = off - slot * D;
                const int grp = (pos >> 5) ^ qrec_swz(slot, D), j0 = grp * 32 + (pos & 31);
                const uint32_t s1 = ksc[slot * G + grp];
                uint4 lo, hi;
                q8_unpack_k16<BF16>(raw, s1 | (s1 << 16), lo, hi);
                uint4* out = reinterpret_cast<uint4*>(dst + (size_t)page_row(0, slot, P, tiled) * D + j0);
                out[0] = lo; out[1] = hi;
            } else {             // V: 8 consecutive d of a token pair, interleaved per d
                const int off = (c - k_chunks) * 16, pair = off / (2 * D), rem = off - pair * 2 * D;
                const int grp = (rem >> 6) ^ (sw * (pair & 1));
                const int chunk = ((rem & 63) >> 3) ^ (sw * 4 * ((pair >> 1) & 1));
                const int j0 = grp * 32 + chunk * 4;
                uint4 even, odd;
                q8_unpack_v8x2<BF16>(raw, vsc[(grp * P + 2 * pair) >> 1], even, odd);
                *reinterpret_cast<uint4*>(dst + (size_t)page_row(1, 2 * pair, P, tiled) * D + j0) = even;
                *reinterpret_cast<uint4*>(dst + (size_t)page_row(1, 2 * pair + 1, P, tiled) * D + j0) = odd;
            }
        }
    }
}

// One warp per query row, any page size and head_dim (multiple of 32, <= 512).
template <bool BF16>
__global__ void generic_quant_kernel(const GenericArgs a) {
    __shared__ float qs[4][512];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t rid = (int64_t)blockIdx.x * 4 + w;
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
    const int h = hq / a.geo.n_rep;
    const int q_pos = sm.pos + r;
    const uint16_t* q = reinterpret_cast<const uint16_t*>(a.q) + rid * D;
    for (int j = lane; j < D; j += 32) qs[w][j] = q_up<BF16>(q[j]);
    __syncwarp();
    const uint8_t* arena = reinterpret_cast<const uint8_t*>(a.arena);
    const size_t rec = qrec_bytes(P, D);
    // kv_dequantize (kv.rs:319-358): value = elem(q * scale); every byte of a record is q + 128
    auto value = [&](const uint8_t* recp, int is_v, int slot, int j) -> float {
        const uint8_t b = recp[qrec_value_off(is_v, slot, j, P, D)];
        const int qi = (int)b - 128;
        const float sc = q_up<BF16>(*reinterpret_cast<const uint16_t*>(recp + qrec_scale_off(is_v, slot, j >> 5, P, D)));
        return q_up<BF16>(q_down<BF16>(__fmul_rn((float)qi, sc)));
    };
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
            const uint8_t* recp = arena + ((size_t)phys * Hkv + h) * rec;
            float dot = 0.f;
            for (int j = 0; j < D; j++) dot += qs[w][j] * value(recp, 0, tk % P, j);
            s = dot * a.scale;
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
            const uint8_t* recp = arena + ((size_t)phys * Hkv + h) * rec;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int j = lane + 32 * i;
                if (j < D) acc[i] += pk * value(recp, 1, tv % P, j);
            }
        }
    }
    uint16_t* out = reinterpret_cast<uint16_t*>(a.out) + rid * D;
    const float inv = 1.f / l;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const int j = lane + 32 * i;
        if (j < D) out[j] = q_down<BF16>(acc[i] * inv);
    }
}

}  // namespace

cudaError_t launch_init_quant(void* arena, size_t n_records, int page_size, int d, cudaStream_t st) {
    init_quant_kernel<<<148 * 8, 256, 0, st>>>(reinterpret_cast<uint8_t*>(arena), n_records, page_size, d);
    return cudaGetLastError();
}

cudaError_t launch_append_quant(const AppendArgs& a, bool bf16, bool overlap, cudaStream_t st) {
    const int64_t rows = 2 * (int64_t)a.step.n_tokens * a.geo.n_kv;
    if (rows <= 0) return cudaSuccess;
    // Token pairs where there is work for them: a lane has 32 divisions to make one after the other, 7 to 9 us however few
    // rows there are, while a row per warp takes 3 us as long as every row finds a warp (9472 of them) and 1 us per 1700
    // rows beyond.  us, pairs / rows, at 272, 8192, 16384 and 65536 rows of 128: 6.6 / 2.9, 8.7 / 5.9, 10.1 / 10.0, 19.4 /
    // 38.2; 1998, 12288 and 24576 of 64: 8.1 / 3.4, 8.6 / 9.1, 9.0 / 16.0; 8192, 16384 of 256: 9.8 / 8.4, 13.7 / 16.0.
    // And only where k and v allow 16 bytes a load; the other kernel takes them at any multiple of 8.
    const bool aligned16 = ((reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v)) & 15) == 0;
    if (rows >= 12288 && aligned16 && a.geo.page_size == 16 && (a.geo.d == 64 || a.geo.d == 128 || a.geo.d == 256)) {
        const int rpw = 512 / a.geo.d;  // rows or pairs of a warp
        const int64_t warps = (rows / 2 + rpw - 1) / rpw + ((a.step.n_tokens / 2 + a.step.n_seqs) * (int64_t)a.geo.n_kv + rpw - 1) / rpw;
        const int blocks = (int)std::min<int64_t>((warps + 7) / 8, 148 * 8);
        switch (a.geo.d) {
            case 64: return launch_pdl(overlap, bf16 ? append_quant_vec_kernel<true, 4> : append_quant_vec_kernel<false, 4>, blocks, 256, 0, st, a);
            case 128: return launch_pdl(overlap, bf16 ? append_quant_vec_kernel<true, 8> : append_quant_vec_kernel<false, 8>, blocks, 256, 0, st, a);
            default: return launch_pdl(overlap, bf16 ? append_quant_vec_kernel<true, 16> : append_quant_vec_kernel<false, 16>, blocks, 256, 0, st, a);
        }
    }
    const int blocks = (int)std::min<int64_t>((rows + 7) / 8, 148 * 8);
    return launch_pdl(overlap, bf16 ? append_quant_kernel<true> : append_quant_kernel<false>, blocks, 256, 0, st, a);
}

cudaError_t launch_dequant_pages(const int32_t* tables, int n_entries, const GeomDev& geo, const void* arena, void* scratch,
                                 int32_t* status, bool bf16, bool overlap, cudaStream_t st) {
    const int64_t items = (int64_t)n_entries * geo.n_kv;
    if (items <= 0) return cudaSuccess;
    const int blocks = (int)std::min<int64_t>((items + 7) / 8, 148 * 8);
    return launch_pdl(overlap, bf16 ? dequant_pages_kernel<true> : dequant_pages_kernel<false>, blocks, 256, 0, st, tables, n_entries, geo,
                      reinterpret_cast<const uint8_t*>(arena), reinterpret_cast<uint16_t*>(scratch), status);
}

cudaError_t launch_generic_quant(const GenericArgs& a, bool bf16, cudaStream_t st) {
    const int64_t rows = (int64_t)a.step.n_tokens * a.geo.n_q;
    if (rows <= 0) return cudaSuccess;
    const int blocks = (int)((rows + 3) / 4);
    if (bf16) generic_quant_kernel<true><<<blocks, 128, 0, st>>>(a);
    else generic_quant_kernel<false><<<blocks, 128, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace cbkv
