// Host-side cache manager (see manager.hpp).  Reference: combs-models/src/kv.rs.
#include "manager.hpp"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>

namespace cbkv {

static thread_local std::string g_err;
void set_error(const std::string& msg) { g_err = msg; }
void set_error_nothrow(const char* msg) noexcept {
    try { g_err = msg; } catch (...) { g_err.clear(); }  // clear() cannot throw
}
const char* last_error() { return g_err.c_str(); }

void Allocator::init(int64_t n) {
    // Reversed so page 0 is allocated first (kv.rs:424-429).
    initial_.resize((size_t)n);
    for (int64_t i = 0; i < n; i++) initial_[(size_t)i] = n - 1 - i;
    free_ = initial_;
}

bool Allocator::set_initial(const int64_t* ids, int64_t n) {
    if (n != (int64_t)initial_.size() || free_.size() != initial_.size()) return false;
    std::vector<char> seen((size_t)n, 0);
    for (int64_t i = 0; i < n; i++) {
        if (ids[i] < 0 || ids[i] >= n || seen[(size_t)ids[i]]) return false;
        seen[(size_t)ids[i]] = 1;
    }
    for (int64_t i = 0; i < n; i++) initial_[(size_t)(n - 1 - i)] = ids[i];
    free_ = initial_;
    return true;
}

int32_t arena_create(const cbkv_config* c, Arena** out) {
    if (!c || !out) { set_error("null argument"); return CBKV_ERR_ARG; }
    if (c->num_layers <= 0 || c->n_q_heads <= 0 || c->n_kv_heads <= 0 || c->head_dim <= 0 ||
        c->page_size <= 0 || c->max_seq_len <= 0 || c->num_pages < 0) {
        set_error("invalid cache geometry"); return CBKV_ERR_ARG;
    }
    if (c->n_q_heads % c->n_kv_heads != 0) { set_error("n_q_heads must be a multiple of n_kv_heads"); return CBKV_ERR_ARG; }
    if (c->head_dim % 8 != 0) { set_error("head_dim must be a multiple of 8 (16-byte rows)"); return CBKV_ERR_ARG; }
    if (c->dtype != CBKV_F16 && c->dtype != CBKV_BF16) { set_error("dtype must be CBKV_F16 or CBKV_BF16"); return CBKV_ERR_ARG; }
    if (c->max_seq_len > (int64_t)1 << 30) { set_error("max_seq_len too large"); return CBKV_ERR_ARG; }
    Arena* a = new Arena();
    a->cfg = *c;
    a->windows.assign((size_t)c->num_layers, 0);
    if (c->layer_windows) {
        for (int i = 0; i < c->num_layers; i++) {
            int64_t w = c->layer_windows[i];
            if (w != 0 && w < 2) {  // kv.rs:514-516
                set_error("sliding window must be >= 2, got " + std::to_string(w));
                delete a; return CBKV_ERR_ARG;
            }
            a->windows[(size_t)i] = w;
        }
    }
    a->cfg.layer_windows = nullptr;  // owned copy lives in `windows`
    a->num_pages = c->num_pages > 0 ? c->num_pages : (c->max_seq_len + c->page_size - 1) / c->page_size;  // kv.rs:82-84
    if (a->num_pages > (int64_t)1 << 30) { set_error("num_pages too large"); delete a; return CBKV_ERR_ARG; }
    a->alloc.init(a->num_pages);
    a->refcnt.assign((size_t)a->num_pages, 0);
    *out = a;
    return CBKV_OK;
}

int32_t seq_create(Arena* a, Seq** out) {
    if (!a || !out) { set_error("null argument"); return CBKV_ERR_ARG; }
    Seq* s = new Seq();
    s->arena = a;
    a->seqs.push_back(s);
    *out = s;
    return CBKV_OK;
}

// Drop the last table entry; the page returns to the free stack when its last
// holder lets go (one holder: exactly kv.rs:830-833).
static void table_pop_release(Seq* s) {
    int64_t page = s->table.back();
    s->table.pop_back();
    if (--s->arena->refcnt[(size_t)page] == 0) s->arena->alloc.free_page(page);
}

int32_t seq_destroy(Seq* s) {
    if (!s) return CBKV_OK;
    Arena* a = s->arena;
    if (a->step_open && std::find(a->step_seqs.begin(), a->step_seqs.end(), s) != a->step_seqs.end()) {
        a->step_open = false;  // the step's tables no longer describe live sequences
    }
    while (!s->table.empty()) table_pop_release(s);
    a->seqs.erase(std::remove(a->seqs.begin(), a->seqs.end(), s), a->seqs.end());
    delete s;
    return CBKV_OK;
}

int32_t seq_fork_prefix(Seq* parent, int64_t n_tokens, Seq** out) {
    if (!parent || !out) { set_error("null argument"); return CBKV_ERR_ARG; }
    Arena* a = parent->arena;
    if (n_tokens < 0 || n_tokens > parent->seq_len || n_tokens % a->cfg.page_size != 0) {
        set_error("fork_prefix: prefix must be whole pages within the parent"); return CBKV_ERR_ARG;
    }
    Seq* c = nullptr;
    seq_create(a, &c);
    int64_t pages = n_tokens / a->cfg.page_size;
    c->table.assign(parent->table.begin(), parent->table.begin() + pages);
    for (int64_t p : c->table) a->refcnt[(size_t)p]++;
    c->seq_len = n_tokens;
    *out = c;
    return CBKV_OK;
}

int32_t begin_step(Arena* a, Seq* const* seqs, const int64_t* new_tokens, const int64_t* pos, int32_t n) {
    if (!a || (n > 0 && (!seqs || !new_tokens)) || n < 0) { set_error("null argument"); return CBKV_ERR_ARG; }
    const int64_t P = a->cfg.page_size;
    int64_t pages_wanted = 0, tokens = 0;
    const uint64_t mark = ++a->mark_gen;  // a sequence seen in this call carries the call's mark
    // validate everything first: state is only mutated when the whole step fits
    for (int32_t b = 0; b < n; b++) {
        Seq* s = seqs[b];
        if (!s || s->arena != a) { set_error("sequence does not belong to this arena"); return CBKV_ERR_ARG; }
        if (s->mark == mark) { set_error("sequence listed twice in one step"); return CBKV_ERR_ARG; }
        s->mark = mark;
        if (new_tokens[b] < 1) { set_error("new_tokens must be >= 1"); return CBKV_ERR_ARG; }
        if (pos && pos[b] != s->seq_len) {  // kv.rs:671-674
            set_error("paged cache expects dense contiguous appends (pos == seq_len)"); return CBKV_ERR_POS;
        }
        int64_t total = s->seq_len + new_tokens[b];
        if (total > a->cfg.max_seq_len) {  // kv.rs:679-683
            set_error("paged cache capacity exceeded: " + std::to_string(total) + " > " + std::to_string(a->cfg.max_seq_len));
            return CBKV_ERR_CAPACITY;
        }
        if (s->seq_len % P != 0 && a->refcnt[(size_t)s->table[(size_t)(s->seq_len / P)]] > 1) {
            set_error("append would write into a page shared with another sequence"); return CBKV_ERR_STATE;
        }
        int64_t need = (total + P - 1) / P;
        pages_wanted += std::max<int64_t>(0, need - (int64_t)s->table.size());
        tokens += new_tokens[b];
    }
    if (pages_wanted > a->alloc.num_free()) {  // kv.rs:552-555
        set_error("page allocator exhausted (max_seq_len exceeded)"); return CBKV_ERR_EXHAUSTED;
    }
    if (tokens > (int64_t)1 << 30) { set_error("step too large"); return CBKV_ERR_ARG; }

    a->step_seqs.assign(seqs, seqs + n);
    a->step_meta.resize((size_t)n);
    a->step_tables.clear();
    a->step_is_decode = n > 0;
    int64_t tok_off = 0;
    for (int32_t b = 0; b < n; b++) {
        Seq* s = seqs[b];
        int64_t total = s->seq_len + new_tokens[b];
        int64_t need = (total + P - 1) / P;
        while ((int64_t)s->table.size() < need) {  // ensure_pages, kv.rs:549-559
            int64_t p = a->alloc.alloc();
            a->refcnt[(size_t)p] = 1;
            s->table.push_back(p);
        }
        SeqMeta& m = a->step_meta[(size_t)b];
        m.pos = (int32_t)s->seq_len;
        m.snew = (int32_t)new_tokens[b];
        m.tok_off = (int32_t)tok_off;
        m.tbl_off = (int32_t)a->step_tables.size();
        for (int64_t p : s->table) a->step_tables.push_back((int32_t)p);
        s->seq_len = total;  // kv.rs:675
        tok_off += new_tokens[b];
        if (new_tokens[b] != 1) a->step_is_decode = false;
    }
    a->step_tokens = tok_off;
    a->step_open = true;
    a->step_id++;
    return CBKV_OK;
}

int32_t popn(Seq* s, int64_t n, int64_t* popped) {
    if (!s || !popped) { set_error("null argument"); return CBKV_ERR_ARG; }
    Arena* a = s->arena;
    *popped = 0;
    n = std::min(n, s->seq_len);  // kv.rs:808
    if (n <= 0) return CBKV_OK;
    if (a->cfg.sliding_popn_refuses) {
        for (int64_t w : a->windows)
            if (w > 0 && s->seq_len > w - 1) return CBKV_OK;  // kv.rs:812-816: eviction would have happened
    }
    const int64_t P = a->cfg.page_size;
    int64_t new_len = s->seq_len - n;
    int64_t keep = (new_len + P - 1) / P;
    // A rollback may not end inside a page other sequences also hold: the next
    // append would overwrite their rows.  Refused, state untouched.
    if (new_len % P != 0 && a->refcnt[(size_t)s->table[(size_t)(keep - 1)]] > 1) return CBKV_OK;
    s->seq_len = new_len;                                  // kv.rs:828
    while ((int64_t)s->table.size() > keep) table_pop_release(s);  // kv.rs:829-833
    if (a->step_open && std::find(a->step_seqs.begin(), a->step_seqs.end(), s) != a->step_seqs.end())
        a->step_open = false;
    *popped = n;
    return CBKV_OK;
}

int32_t reset(Seq* s) {
    if (!s) { set_error("null argument"); return CBKV_ERR_ARG; }
    Arena* a = s->arena;
    if (a->seqs.size() == 1) {  // kv.rs:837-846: table cleared, allocator rebuilt
        for (int64_t p : s->table) a->refcnt[(size_t)p] = 0;
        s->table.clear();
        a->alloc.reset();
    } else {
        while (!s->table.empty()) table_pop_release(s);
    }
    s->seq_len = 0;
    a->step_open = false;
    return CBKV_OK;
}

void page_stats(const Seq* s, int64_t layers_materialized, cbkv_page_stats_t* out) {  // kv.rs:535-546
    const Arena* a = s->arena;
    out->pages_used = (int64_t)s->table.size();
    out->pages_free = a->alloc.num_free();
    out->num_pages = a->num_pages;
    out->page_size = a->cfg.page_size;
    out->seq_len = s->seq_len;
    out->layers_materialized = layers_materialized;
    out->layers_total = a->cfg.num_layers;
    out->layers_sliding = 0;  // windows are masks over pages here; no rolling stores exist
}

namespace {

// The parts of every segment, the first segment and part of every item: sweeps the items in unit order (range by range,
// level by level).
void number_parts(DecodePlan* pl) {
    const int n_ctas = pl->n_ctas, levels = pl->levels;
    for (SegInfo& sg : pl->segs) { sg.nparts = 0; sg.part_base = -1; }
    std::vector<int32_t> order;
    order.reserve((size_t)pl->n_items);
    for (int c = 0; c < n_ctas; c++)
        for (int j = 0; j < levels; j++)
            if (pl->items[(size_t)j * n_ctas + c].u_end > pl->items[(size_t)j * n_ctas + c].u_begin) order.push_back(j * n_ctas + c);
    size_t io = 0;
    int parts = 0;
    for (int s = 0; s < pl->n_segs; s++) {
        SegInfo& sg = pl->segs[(size_t)s];
        const int32_t sb = sg.unit_begin, se = pl->segs[(size_t)s + 1].unit_begin;
        if (se == sb) continue;
        while (io < order.size() && pl->items[(size_t)order[io]].u_end <= sb) io++;
        int cnt = 0;
        for (size_t k = io; k < order.size() && pl->items[(size_t)order[k]].u_begin < se; k++) {
            ItemInfo& it = pl->items[(size_t)order[k]];
            if (it.u_begin >= sb) { it.first_seg = s; it.first_part = cnt; }
            cnt++;
        }
        sg.nparts = cnt;
        if (cnt > 1) { sg.part_base = parts; parts += cnt; }
    }
    pl->n_parts = parts;
    for (ItemInfo& it : pl->items)  // empty items (possible only when units < items) are never claimed usefully
        if (it.u_end <= it.u_begin) { it.first_seg = 0; it.first_part = 0; }
}

}  // namespace

void build_decode_plan(const Arena& a, int64_t window, int32_t n_ctas, const DecodeSplit& split, DecodePlan* pl) {
    const int64_t P = a.cfg.page_size;
    const int Hkv = a.cfg.n_kv_heads;
    const int n = (int)a.step_meta.size();
    pl->window = window;
    pl->n_segs = n * Hkv;
    pl->segs.assign((size_t)pl->n_segs + 1, SegInfo{});
    int64_t units = 0;
    for (int b = 0; b < n; b++) {
        const SeqMeta& m = a.step_meta[(size_t)b];
        int64_t L = (int64_t)m.pos + m.snew;
        int64_t q_pos = L - 1;                                   // the single decode query
        int64_t lo_key = window > 0 ? std::max<int64_t>(0, q_pos - window + 1) : 0;  // keys in (p - w, p], kv.rs:112-115
        int64_t p_lo = lo_key / P, p_hi = q_pos / P;
        for (int h = 0; h < Hkv; h++) {
            SegInfo& sg = pl->segs[(size_t)b * Hkv + h];
            sg.unit_begin = (int32_t)units;
            sg.page_lo = (int32_t)p_lo;
            sg.q_pos = (int32_t)q_pos;
            sg.tok_off = m.tok_off;
            sg.nparts = 0;
            sg.part_base = -1;
            sg.tbl_off = m.tbl_off;
            units += p_hi - p_lo + 1;
        }
    }
    pl->segs[(size_t)pl->n_segs].unit_begin = (int32_t)units;
    pl->n_units = (int32_t)units;
    n_ctas = (int32_t)std::max<int64_t>(1, std::min<int64_t>(n_ctas, units));
    pl->n_ctas = n_ctas;

    // Levels of the tail, decided on the shortest range so that every range has the same number of items.
    const int64_t lmin = units / n_ctas;
    int levels = 1;
    {
        const int64_t tail = lmin * split.tail_pct / 100;
        if (split.min_item > 0 && tail >= split.min_item) {
            int pieces = 1;
            while (pieces + 1 < split.max_levels && (tail >> pieces) >= split.min_item) pieces++;
            levels = 1 + pieces;
        }
    }
    pl->levels = levels;
    pl->n_items = n_ctas * levels;
    pl->items.assign((size_t)pl->n_items, ItemInfo{});
    // item (level j, range c) sits at claim index j * n_ctas + c; inside a range the levels follow each other
    for (int c = 0; c < n_ctas; c++) {
        const int64_t rb = units * c / n_ctas, re = units * (c + 1) / n_ctas;
        const int64_t len = re - rb;
        int64_t rest = levels > 1 ? len * split.tail_pct / 100 : 0;
        int64_t at = rb;
        for (int j = 0; j < levels; j++) {
            int64_t take;
            if (j == 0) take = len - rest;
            else if (j == levels - 1) take = rest;
            else take = (rest + 1) / 2;
            if (j > 0) rest -= take;
            ItemInfo& it = pl->items[(size_t)j * n_ctas + c];
            it.u_begin = (int32_t)at;
            it.u_end = (int32_t)(at + take);
            at += take;
        }
    }
    pl->aligned = false;
    number_parts(pl);
}

bool align_decode_plan(int32_t n_kv_heads, int32_t min_pages, int32_t slack, int32_t max_ctas, DecodePlan* pl) {
    if (pl->levels != 1 || pl->n_units <= 0 || pl->n_segs > max_ctas) return false;
    auto pages_of = [&](int s) { return pl->segs[(size_t)s + 1].unit_begin - pl->segs[(size_t)s].unit_begin; };
    int32_t longest = 0;
    for (int s = 0; s < pl->n_segs; s += n_kv_heads) longest = std::max(longest, pages_of(s));
    auto fits = [&](int32_t most) {  // the heads of a sequence have the same pages
        int64_t n = 0;
        for (int s = 0; s < pl->n_segs; s += n_kv_heads) n += (pages_of(s) + most - 1) / most;
        return n * n_kv_heads <= max_ctas;
    };
    const int32_t even = (pl->n_units + pl->n_ctas - 1) / pl->n_ctas;
    int32_t lo = std::max(min_pages, 1), hi = std::max(lo, std::min(longest, std::max(even, lo) + slack));
    if (!fits(hi)) return false;
    while (lo < hi) {  // the shortest ranges that do
        const int32_t mid = lo + (hi - lo) / 2;
        if (fits(mid)) hi = mid; else lo = mid + 1;
    }
    pl->items.clear();
    for (int s = 0; s < pl->n_segs; s++) {
        const int32_t p = pages_of(s), n = (p + lo - 1) / lo, begin = pl->segs[(size_t)s].unit_begin;
        for (int i = 0; i < n; i++) {
            ItemInfo it{};
            it.u_begin = begin + (int32_t)((int64_t)p * i / n);
            it.u_end = begin + (int32_t)((int64_t)p * (i + 1) / n);
            pl->items.push_back(it);
        }
    }
    pl->n_items = pl->n_ctas = (int32_t)pl->items.size();
    pl->aligned = false;  // one sequence, or several of one length: the even cut of as many CTAs, which the kernel computes
    for (int64_t c = 0; c < pl->n_ctas && !pl->aligned; c++)
        pl->aligned = pl->items[(size_t)c].u_begin != (int64_t)pl->n_units * c / pl->n_ctas;
    number_parts(pl);
    return true;
}

// A CTA whose range straddles two segments works through two chains one after the other (the second's queries and tiles, its
// combine, its partial and ticket wait for the first's), and the launch ends with the slowest: 3 to 4 us of the 10 to 15 that
// decode launches of a few sequences take.  So the ranges end where segments do, unless that makes the longest of them longer
// than the even cut's by more than it saves: 64 pages at head_dim 64, 48 at 128, 16 at 256; int8 pages, whose tiles are bound by
// arithmetic, 20, 16 and 8.  Measured even / aligned, us per launch (16 bits; B sequences of lo to hi tokens, kv heads/head_dim):
//   1 x 1500 3/64 10.7 / 6.6, 4/128 13.2 / 7.4, 4/256 13.8 / 8.0;  4 x 300-2000 3/64 12.1 / 7.9, 4/128 13.3 / 8.8, 4/256 14.3 / 10.5
//   16 x 4000 4/128 29 / 28, 8/128 47 / 44;  32 x 1024-4096 4/128 33.9 / 33.9 (35.4 with 96 more pages);  16 x 8192 with windows of
//   1024 4/256 29.7 / 28.1;  8 x 8000 4/256 49 / 52 with 24 more pages
//   int8: 4 x 300-2000 4/128 24 / 14.6;  32 x 300-1000 8/128 23 / 21;  16 x 4000 8/128 36 / 37, 4/256 48 / 50 with 32 more pages
// The lines are where batches of nearly as many segments as CTAs break even, all of one length but one sequence, which a range
// then holds whole (pages of the others + of that one; with half of the batch longer the ranges that end with segments win by more):
//   3/64 5 + 69 10.2 / 9.5, 5 + 120 11.1 / 12.9, 80 + 144 15.7 / 15.5, 200 + 264 26.2 / 26.3;  8/128 5 + 53 11.4 / 9.7, 40 + 88
//   14.6 / 14.9, 120 + 168 28.3 / 29.4;  4/256 5 + 21 11.5 / 10.0, 40 + 56 22.9 / 24.2, 200 + 216 78 / 79
//   int8: 3/64 5 + 25 12.3 / 10.9, 5 + 36 12.3 / 12.7, 40 + 60 18.7 / 18.0, 40 + 80 18.9 / 21.1;  4/128 5 + 36 14.5 / 14.8, 40 + 56
//   24.7 / 21.6, 40 + 80 25.3 / 26.4;  8/128 (the long one in two) 5 + 36 12.8 / 13.3, 5 + 69 14.0 / 17.0, 40 + 140 25.0 / 27.2;
//   4/256 5 + 13 14.7 / 12.8, 40 + 48 27.0 / 22.2, 40 + 80 27.8 / 31.7
//
// Segments of a few pages are not cut at all: a CTA per segment streams its pages in the time that a cut spends on partials,
// tickets and the merge.  One sequence, cut into a page per consumer warp / uncut, us per launch:
//   head_dim  64: 12 pages 5.3 / 4.1, 23 pages 5.6 / 5.4, 27 pages 5.6 / 5.8, 32 pages 5.6 / 6.7
//   head_dim 128: 12 pages 6.6 / 4.9, 23 pages 6.9 / 6.5, 27 pages 6.9 / 6.7, 32 pages 6.8 / 7.6
//   head_dim 256: 12 pages 6.5 / 5.6, 16 pages 6.6 / 6.2, 19 pages 6.8 / 7.0, 23 pages 6.9 / 8.1
//   int8: 64 12 pages 5.8 / 5.1, 26 6.0 / 6.6; 128 19 pages 6.4 / 6.2, 26 6.8 / 7.2; 256 12 pages 7.8 / 7.5, 16 7.6 / 8.2
// An arena of one layer launches once a step, behind that step's upload and unit table: no launch runs under another's tail, and
// an upload of more than 1 KB, which a cut makes of many a short one, takes 5 us longer.  So segments of up to 40 pages stay whole
// there, up to 16 of them; with more, both uploads are that long.  16 bits, us per step, cut / uncut at 33 and 40 pages:
//   1 sequence:  3/64 12.7 / 12.7, 12.8 / 12.6;  1/128 12.5 / 12.6, 12.3 / 13.4;  4/128 12.7 / 12.8, 13.1 / 13.7;  8/128 18.7 / 13.4, 17.4 / 14.5
//   2 sequences: 3/64 19.2 / 12.8, 18.6 / 13.0;  1/128 12.5 / 12.5, 12.7 / 13.5;  4/128 18.9 / 13.5, 18.6 / 14.5;  8/128 18.5 / 19.7, 17.4 / 21.1
//   4 sequences: 3/64 17.6 / 17.2, 17.6 / 19.7;  1/128 17.6 / 13.1, 17.5 / 13.9;  4/128 17.4 / 17.0, 17.7 / 18.5;  8/128 19.2 / 19.7, 18.5 / 20.4
// With two layers one sequence is equal at 33 pages and better cut at 40 (3/64 17.6 / 17.6, 17.6 / 19.3; 4/128 18.4 / 18.6, 19.0 / 19.7).
void choose_decode_plan(const Arena& a, int64_t window, bool quant, int32_t consumers, int32_t max_ctas, const DecodeSplit& split, DecodePlan* pl) {
    build_decode_plan(a, window, max_ctas, split, pl);
    // at least one page per consumer warp, at most one resident wave of CTAs
    const int32_t want = std::max(1, (pl->n_units + consumers - 1) / consumers);
    if (want < pl->n_ctas) build_decode_plan(a, window, want, split, pl);
    const int32_t d = a.cfg.head_dim, at = d <= 64 ? 0 : d <= 128 ? 1 : 2;
    static constexpr int32_t kSlack[2][3] = {{64, 48, 16}, {20, 16, 8}}, kUncut[2][3] = {{24, 28, 17}, {19, 20, 12}};
    int32_t longest = 0;
    for (int s = 0; s < pl->n_segs; s += a.cfg.n_kv_heads) longest = std::max(longest, pl->segs[(size_t)s + 1].unit_begin - pl->segs[(size_t)s].unit_begin);
    const int32_t uncut = a.cfg.num_layers == 1 && pl->n_segs <= 16 && !quant && d <= 128 ? 40 : kUncut[quant ? 1 : 0][at];
    align_decode_plan(a.cfg.n_kv_heads, longest <= uncut ? longest : consumers, kSlack[quant ? 1 : 0][at], max_ctas, pl);
}

void build_chunk_plan(const Arena& a, int32_t cols_per_item, ChunkPlan* pl) {
    const int n = (int)a.step_meta.size();
    pl->cols_per_item = cols_per_item;
    pl->item_begin.assign((size_t)n + 1, 0);
    int64_t items = 0;
    for (int b = 0; b < n; b++) {
        pl->item_begin[(size_t)b] = (int32_t)items;
        int64_t cols = (int64_t)a.step_meta[(size_t)b].snew * a.n_rep();
        items += (int64_t)a.cfg.n_kv_heads * ((cols + cols_per_item - 1) / cols_per_item);
    }
    pl->item_begin[(size_t)n] = (int32_t)items;
    pl->n_items = (int32_t)items;
}

namespace {

// Launch model of the tcgen05 chunk kernels, in units of one K/V tile of a full item: a CTA costs kCtaCost
// besides its tiles (tensor-memory allocation, first loads, epilogue), a K/V tile of an item that fills one of
// its two query tiles kHalfTile, a slice kSliceCost more (its partial rows), and the merge at the end
// kMergeCost for each slice of the full 256 rows.
constexpr float kCtaCost = 3.f, kHalfTile = 0.7f, kSliceCost = 0.7f, kMergeCost = 0.7f;
constexpr float kPairCtaCost = 5.f, kPairSliceCost = 1.f, kPairMergeCost = 1.f;  // the same for pairs of CTAs, whose K/V tiles are shorter

// Measured per head_dim over batches of 1 to 64 sequences with 33 to 2000 cached tokens (GQA groups of 2 to 7, f16):
// a tcgen05 launch takes fixed_us, then per wave of one CTA per SM cta_us + tile_us for each K/V tile (head_dim 128:
// [0] with one query tile, [1] with both); the mma.sync kernel, one warp per item over all its pages, mma_us + page_us
// for each page of the longest item, `warps` of them per SM at a time; with more items than that, kMmaRounds times as
// much per round.  Pairs of CTAs: pair_cta_us and pair_tile_us per wave of one pair per two SMs.
//
// The merge of cut items counts as well (head_dim 128 and 256): merge_us[pairs] for each round of loads that the last
// slice's threads make (four slices and 8 columns of a row per thread and round), which is as long as the tiles where few
// K/V tiles are cut often.  Fitted over 384 steps at head_dim 128 and 170 at 256 (2 to 1024 new tokens and mixes of many with
// one, 1 to 48 sequences, 0 to 8192 cached tokens, with and without a window, GQA groups of 1 to 8): estimates off by 7 to
// 9 % rms (38 % for the two-tile kernel without the merge), the kernel they choose within 5 % of the fastest of the three
// but for 24 and 3 steps, the worst 1.36 times (2 prompts of 100 tokens beside 1 to 3 decoding sequences, 25 us).  us, one
// tile / pairs at head_dim 256: 48 sequences x 2 tokens after 2048 74 / 117, 16 x 5 after 8192 94 / 123, 1 x 9 after 8192 45
// / 30, a prompt of 512 after 512 49 / 24; two tiles / pairs at 128: 2 prompts of 333 after 1024 (4 kv heads) 35 / 43.
//
// The tcgen05 kernels are 5 to 15 % faster than when this was fitted, all by about as much; the mma.sync kernel is not, so near
// its line it is taken a little too often.  Over 92 steps (1 to 64 sequences, 1 to 512 new tokens and mixes, four geometries) the
// kernel taken was within 7 % of the fastest, but for one (a prompt of 100 tokens at head_dim 256, 12.6 us against 11.1).
//
// pair_margin: pairs are taken where their estimate is below this share of the others'.  At head_dim 128, where the kernels
// are closer, a tenth, the estimates' own error: 8 sequences x 5 tokens after 512 to 6144 (28 q heads) come out equal and
// take 29.3 us a layer with two tiles per CTA, 31.6 on pairs.
struct ChunkTimes { float cta_us[2], tile_us[2], mma_us, page_us; int32_t warps; float pair_cta_us, pair_tile_us, merge_us[2], pair_margin; };
constexpr float kChunkFixedUs = 1.7f, kMmaRounds = 1.5f;
ChunkTimes chunk_times(int32_t d) {
    switch (d) {
        case 64: return {{5.f, 5.f}, {1.f, 1.f}, 11.f, 1.04f, 12, 0.f, 0.f, {0.f, 0.f}, 1.f};
        case 128: return {{5.8f, 10.f}, {2.1f, 2.45f}, 8.f, 0.84f, 8, 8.f, 1.25f, {0.9f, 1.f}, 0.9f};
        default: return {{6.f, 6.f}, {1.4f, 1.4f}, 7.5f, 0.88f, 4, 8.5f, 1.85f, {1.2f, 1.f}, 1.f};  // 256
    }
}

// SMs that take CTAs in launch order, each the next one that is free: a heap of the times at which they are, padded so that
// every inner node has two children and the way down has no branch but its end.
class Sms {
public:
    void start(int n) {
        n_ = (size_t)n;
        taken_ = 0;
        end_ = 0.f;
        free_at_.clear();
    }
    void run(float us) {
        if (taken_ < n_) {  // an idle SM
            free_at_.push_back(us);
            end_ = std::max(end_, us);
            if (++taken_ == n_) {
                std::make_heap(free_at_.begin(), free_at_.end(), [](float x, float y) { return x > y; });
                free_at_.resize(2 * n_ + 1, INFINITY);
            }
            return;
        }
        float* f = free_at_.data();
        const float t = f[0] + us;
        end_ = std::max(end_, t);
        size_t i = 0;
        while (i < n_) {
            const size_t c = 2 * i + 1 + (f[2 * i + 2] < f[2 * i + 1] ? 1 : 0);
            if (!(f[c] < t)) break;
            f[i] = f[c];
            i = c;
        }
        f[i] = t;
    }
    float end() const { return end_; }

private:
    std::vector<float> free_at_;
    size_t n_ = 0, taken_ = 0;
    float end_ = 0.f;
};

// CTAs are launched longest (sequence, kv head) first; the items of one (sequence, kv head) stay together, slice
// by slice, because they read the same K/V.  Whether and how finely items are cut is decided by running the
// launch model over a few candidates: no cut, the remainder of the last wave cut in equal parts (a launch of
// several waves whose last is mostly empty), and every item longer than a limit cut into slices of at most that
// (a launch that has too few items for the chip: a few tokens of a few sequences over long contexts).
//
// This runs on the host in front of a step's first chunk launch, once per window, so what it costs is seen by steps of
// few layers: the kv heads of a sequence share everything but their place in the order, and a candidate whose work
// divided evenly would already end later than the best so far is not run through the model.
class TilePlanner {
public:
    TilePlanner(const Arena& a, int32_t tokens_per_tile, const TileCut& cut)
        : a_(a), cut_(cut), tokens_(tokens_per_tile), tile_tokens_(cut.tile_tokens > 0 ? cut.tile_tokens : tokens_per_tile) {
        const int n = (int)a.step_meta.size();
        item_begin_.assign((size_t)n + 1, 0);
        for (int b = 0; b < n; b++) {
            const SeqMeta& m = a.step_meta[(size_t)b];
            const int n_qt = (m.snew + tokens_ - 1) / tokens_;
            item_begin_[(size_t)b] = (int32_t)items_;
            items_ += (int64_t)a.cfg.n_kv_heads * n_qt;
            if (n_qt == 0) continue;
            Group g{b, (int32_t)work_.size(), n_qt, 0.f};
            for (int qt = 0; qt < n_qt; qt++) {
                const int r0 = qt * tokens_, toks = std::min(tokens_, m.snew - r0);
                const int64_t q_first = m.pos + r0, q_last = q_first + toks - 1;
                const int64_t lo_key = cut.window > 0 ? std::max<int64_t>(0, q_first - cut.window + 1) : 0;
                const int32_t pages = (int32_t)((q_last >> 4) - (lo_key >> 4) + 1), ppt = cut.kv_tile / 16;
                const bool both = toks > tile_tokens_;
                // one query tile per CTA: the same for every item
                Work w{(pages + ppt - 1) / ppt, both || tile_tokens_ == tokens_ ? 1.f : kHalfTile, (float)toks / (float)tokens_, both ? 1 : 0,
                       std::min(toks, cut.pair ? tokens_ / 2 : tile_tokens_) * a.n_rep()};
                g.cost = std::max(g.cost, w.per_tile * w.n_tiles);
                work_.push_back(w);
            }
            groups_.push_back(g);
        }
        item_begin_[(size_t)n] = (int32_t)items_;
        std::stable_sort(groups_.begin(), groups_.end(), [](const Group& x, const Group& y) { return x.cost > y.cost; });
    }

    // How the items are cut: the candidate that ends first.
    void choose() {
        how_ = How{};
        if (!(cut_.sm_count > 0 && cut_.max_parts > 1 && items_ > 0 && items_ <= 8192)) return;
        float best = end_of(How{}, INFINITY);
        auto consider = [&](const How& how) {
            const float e = end_of(how, best);
            if (e < best) { best = e; how_ = how; }
        };
        const int64_t r = items_ % cut_.sm_count;
        if (items_ > cut_.sm_count && r > 0)
            for (int p = 2; p <= std::min<int64_t>(4, cut_.sm_count / r); p++) consider(How{0.f, r, p});
        if (items_ > 4 * cut_.sm_count) return;
        double total = 0.;
        float longest = 0.f;
        for (const Work& w : work_) { total += (double)w.per_tile * w.n_tiles; longest = std::max(longest, w.per_tile * (float)w.n_tiles); }
        const float even = (float)(total * a_.cfg.n_kv_heads / cut_.sm_count);  // tiles per SM
        for (float f : {1.3f, 1.f, 0.75f, 0.5f, 0.35f}) {
            const float lim = std::max(1.f, even * f);
            if (lim < longest) consider(How{lim, 0, 1});
        }
    }

    // Expected time of the launch in microseconds, and what it cannot be below however its items are cut.
    float launch_us() {
        const ChunkTimes t = chunk_times(a_.cfg.head_dim);
        const int threads = cut_.pair ? 512 : 256, row_items = a_.cfg.head_dim / 8;
        int rounds = 0;  // of the longest merge
        sms_.start(cut_.sm_count);
        each_cta(how_, [&](const Work& w, int, int, int, int tiles, int part, int parts) {
            if (part == 0 && parts > 1) rounds = std::max(rounds, (parts + 3) / 4 * ((w.tile_rows * row_items + threads - 1) / threads));
            sms_.run(cta_us(t, w, tiles));
            modelled_++;
        });
        return kChunkFixedUs + sms_.end() + t.merge_us[cut_.pair ? 1 : 0] * (float)rounds;
    }
    float least_us() const {
        const ChunkTimes t = chunk_times(a_.cfg.head_dim);
        double total = 0.;
        float shortest = INFINITY;
        for (const Work& w : work_) { total += cta_us(t, w, w.n_tiles); shortest = std::min(shortest, cta_us(t, w, 1)); }
        return work_.empty() ? 0.f : 0.999f * (kChunkFixedUs + std::max(shortest, (float)(total * a_.cfg.n_kv_heads / cut_.sm_count)));
    }

    void emit(ChunkPlan* pl) {
        pl->cols_per_item = tokens_;
        pl->item_begin = item_begin_;
        pl->n_items = (int32_t)items_;
        pl->tiles.clear();
        pl->n_slots = pl->n_cut = 0;
        std::vector<int32_t> base, id;  // of the current (sequence, kv head), by block of query tokens
        each_cta(how_, [&](const Work& w, int seq, int h, int qt, int tiles, int part, int parts) {
            if (part == 0) {
                base.resize(std::max(base.size(), (size_t)qt + 1)); id.resize(base.size());
                base[(size_t)qt] = parts > 1 ? pl->n_slots : -1; id[(size_t)qt] = parts > 1 ? pl->n_cut : -1;
                if (parts > 1) { pl->n_slots += parts; pl->n_cut++; }
            }
            const int t0 = part * ((w.n_tiles + parts - 1) / parts);
            pl->tiles.push_back({seq, h, qt, t0, t0 + tiles, part | (parts << 16), base[(size_t)qt], id[(size_t)qt]});
        });
    }

    int64_t modelled() const { return modelled_; }

private:
    struct Work { int32_t n_tiles; float per_tile, rows; int32_t both, tile_rows; };  // an uncut item, the same for every kv head
    struct Group { int32_t seq, first, n_qt; float cost; };
    // parts of an item: ceil(cost / limit), and for the last `rem` items of the launch order at least rem_parts
    struct How { float limit = 0.f; int64_t rem = 0; int rem_parts = 1; };

    float cta_us(const ChunkTimes& t, const Work& w, int tiles) const {
        return cut_.pair ? t.pair_cta_us + t.pair_tile_us * (float)tiles : t.cta_us[w.both] + t.tile_us[w.both] * (float)tiles;
    }

    int parts_of(const Work& w, const How& how, bool tail) const {
        int p = how.limit > 0.f ? (int)std::min(1e6f, w.per_tile * (float)w.n_tiles / how.limit + 0.999f) : 1;
        if (tail) p = std::max(p, how.rem_parts);
        p = std::max(1, std::min(std::min(p, cut_.max_parts), w.n_tiles));
        const int per = (w.n_tiles + p - 1) / p;
        return (w.n_tiles + per - 1) / per;  // no empty slices
    }

    // f(item, sequence, kv head, block of query tokens, its K/V tiles, part, parts) of every CTA in launch order
    template <typename F>
    void each_cta(const How& how, F&& f) {
        int64_t at = 0;
        for (const Group& g : groups_) {
            int most = 1;
            for (int h = 0; h < a_.cfg.n_kv_heads; h++, at += g.n_qt) {
                if (h == 0 || (how.rem > 0 && at + g.n_qt > items_ - how.rem)) {  // the heads share their cut up to the tail
                    parts_.resize((size_t)g.n_qt);
                    most = 1;
                    for (int qt = 0; qt < g.n_qt; qt++)
                        most = std::max(most, parts_[(size_t)qt] = parts_of(work_[(size_t)(g.first + qt)], how, at + qt >= items_ - how.rem));
                }
                for (int p = 0; p < most; p++)
                    for (int qt = 0; qt < g.n_qt; qt++) {
                        const int np = parts_[(size_t)qt];
                        if (p >= np) continue;
                        const Work& w = work_[(size_t)(g.first + qt)];
                        const int per = (w.n_tiles + np - 1) / np;
                        f(w, g.seq, h, qt, std::min(w.n_tiles, (p + 1) * per) - p * per, p, np);
                    }
            }
        }
    }

    // When the launch ends, in the model's units, or infinity when that is not before `best` or takes too many slots.
    float end_of(const How& how, float best) {
        const float cta_cost = cut_.pair ? kPairCtaCost : kCtaCost, slice_cost = cut_.pair ? kPairSliceCost : kSliceCost,
                    merge_cost = cut_.pair ? kPairMergeCost : kMergeCost;
        float merge = 0.f, longest = 0.f;
        int64_t slots = 0;
        if (how.rem == 0) {  // what one kv head says about all of them
            double total = 0.;
            for (const Work& w : work_) {
                const int np = parts_of(w, how, false), per = (w.n_tiles + np - 1) / np;
                if (np > 1) { slots += np; merge = std::max(merge, merge_cost * (0.5f + (float)np * w.rows)); }
                total += w.per_tile * (double)w.n_tiles + np * (double)(cta_cost + (np > 1 ? slice_cost : 0.f));
                longest = std::max(longest, cta_cost + w.per_tile * (float)per + (np > 1 ? slice_cost : 0.f));
            }
            if (slots * a_.cfg.n_kv_heads > (int64_t)kSplitSlotsPerSm * cut_.sm_count) return INFINITY;
            if (std::max(longest, 0.999f * (float)(total * a_.cfg.n_kv_heads / cut_.sm_count)) + merge >= best) return INFINITY;
        }
        sms_.start(cut_.sm_count);
        slots = 0;
        each_cta(how, [&](const Work& w, int, int, int, int tiles, int part, int parts) {
            if (part == 0 && parts > 1) { slots += parts; merge = std::max(merge, merge_cost * (0.5f + (float)parts * w.rows)); }
            sms_.run(cta_cost + w.per_tile * (float)tiles + (parts > 1 ? slice_cost : 0.f));
            modelled_++;
        });
        return slots > (int64_t)kSplitSlotsPerSm * cut_.sm_count ? INFINITY : sms_.end() + merge;
    }

    const Arena& a_;
    const TileCut cut_;
    const int32_t tokens_, tile_tokens_;
    int64_t items_ = 0, modelled_ = 0;
    std::vector<int32_t> item_begin_, parts_;
    std::vector<Work> work_;  // per sequence and block of query tokens
    std::vector<Group> groups_;
    How how_;
    Sms sms_;
};

}  // namespace

void build_chunk_tile_plan(const Arena& a, int32_t tokens_per_tile, ChunkPlan* pl, const TileCut& cut) {
    TilePlanner p(a, tokens_per_tile, cut);
    p.choose();
    p.emit(pl);
}

// Pairs of SMs take a query tile per CTA, with half of K and V each: a launch that leaves SMs idle ends sooner (a prompt
// of 512 after 512, 8 kv heads, head_dim 128: 19.5 against 31.0 us), one that fills them does not at head_dim 128 (four of
// them after 1024: 92 against 73); at head_dim 256, where one CTA has room for K/V tiles of half the size only, prompts do
// (8 of 512 after 7680: 236 against 338), steps of a few tokens of many sequences, whose second tile is empty, do not.
//
// One tcgen05 CTA per SM at a time costs more to start than a few pages take the mma.sync kernel, of which eight warps
// (items) share an SM: steps with more (sequence, kv head) pairs than SMs over short contexts, and prompts of some tens of
// tokens.  64 sequences x 2 tokens after 33 (8 kv heads, head_dim 128): 12.7 against 28.7 us, after 600: 45 against 65;
// 32 x 2 after 600: 43 against 34; a 40-token prompt (4 kv heads) 10.3 against 13.0.
ChunkLaunch plan_chunk_launch(const Arena& a, const ChunkChoice& c) {
    ChunkLaunch out;
    const float mma_us = c.mma_cols > 0 ? chunk_mma_launch_us(a, c.one.window, c.mma_cols, c.one.sm_count) : INFINITY;
    std::unique_ptr<TilePlanner> one, two;
    float least = INFINITY;
    if (c.one_tokens > 0) { one.reset(new TilePlanner(a, c.one_tokens, c.one)); if (c.chooses()) least = one->least_us(); }
    if (c.pairs) { two.reset(new TilePlanner(a, c.pair_tokens, c.pair)); if (c.chooses()) least = std::min(least, two->least_us()); }
    if (mma_us < least) { out.mma = true; return out; }  // whatever a plan would say
    float us = INFINITY;
    if (one) { one->choose(); if (c.chooses()) us = one->launch_us(); }
    const float margin = chunk_times(a.cfg.head_dim).pair_margin;
    if (two && two->least_us() < margin * us) {
        two->choose();
        const float pair_us = c.chooses() ? two->launch_us() : 0.f;
        if (pair_us < margin * us) { out.pair = true; us = pair_us; }
    }
    out.modelled = (one ? one->modelled() : 0) + (two ? two->modelled() : 0);
    out.mma = mma_us < us;
    if (!out.mma) (out.pair ? two : one)->emit(&out.plan);
    return out;
}

float chunk_mma_launch_us(const Arena& a, int64_t window, int32_t cols_per_item, int32_t sm_count) {
    const ChunkTimes t = chunk_times(a.cfg.head_dim);
    int64_t items = 0, longest = 0;
    for (const SeqMeta& m : a.step_meta) {
        if (m.snew == 0) continue;
        const int64_t lo_key = window > 0 ? std::max<int64_t>(0, (int64_t)m.pos - window + 1) : 0;
        items += (int64_t)a.cfg.n_kv_heads * (((int64_t)m.snew * a.n_rep() + cols_per_item - 1) / cols_per_item);
        longest = std::max<int64_t>(longest, (((int64_t)m.pos + m.snew - 1) >> 4) - (lo_key >> 4) + 1);
    }
    const int64_t at_once = (int64_t)sm_count * t.warps, rounds = (items + at_once - 1) / at_once;
    return t.mma_us + t.page_us * (float)longest * (rounds > 1 ? kMmaRounds * (float)rounds : 1.f);
}

}  // namespace cbkv
