// C interface of the host runtime (loaded from Python with ctypes): cache manager, scheduler and
// the assembly of a step's metadata into one packed int32 buffer that a single copy sends to the
// device.
#include <algorithm>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "cache_manager.h"
#include "scheduler.h"

#define XB_API extern "C" __attribute__((visibility("default")))

using namespace xb;

// ---- cache manager -------------------------------------------------------------------------
XB_API void* xb_cm_create(int n_groups, const int* page_sizes, const int* num_pages, const int* windows,
                          const int* keep_first, int max_requests) {
    if (n_groups <= 0 || max_requests <= 0) return nullptr;
    std::vector<GroupSpec> groups(n_groups);
    for (int g = 0; g < n_groups; ++g) {
        if (page_sizes[g] <= 0 || num_pages[g] <= 0) return nullptr;
        groups[g].page_size = page_sizes[g];
        groups[g].num_pages = num_pages[g];
        groups[g].window = windows[g];
        groups[g].keep_first = keep_first ? keep_first[g] : 0;
    }
    return new CacheManager(groups, max_requests);
}
XB_API void xb_cm_destroy(void* h) { delete static_cast<CacheManager*>(h); }
XB_API int xb_cm_open(void* h) { return static_cast<CacheManager*>(h)->open_request(); }
XB_API int xb_cm_close(void* h, int slot) { return static_cast<CacheManager*>(h)->close_request(slot) ? 1 : 0; }
XB_API int xb_cm_is_live(void* h, int slot) { return static_cast<CacheManager*>(h)->is_live(slot) ? 1 : 0; }
XB_API int xb_cm_length(void* h, int slot) { return static_cast<CacheManager*>(h)->length(slot); }
XB_API int xb_cm_can_extend(void* h, int slot, int new_len) { return static_cast<CacheManager*>(h)->can_extend(slot, new_len) ? 1 : 0; }
XB_API int xb_cm_extend(void* h, int slot, int new_len) { return static_cast<CacheManager*>(h)->extend(slot, new_len) ? 1 : 0; }
XB_API int xb_cm_advance(void* h, int slot, int new_len) { return static_cast<CacheManager*>(h)->advance(slot, new_len) ? 1 : 0; }
XB_API int xb_cm_free_pages(void* h, int g) { return static_cast<CacheManager*>(h)->free_pages(g); }
XB_API int xb_cm_table_size(void* h, int slot, int g) { return static_cast<CacheManager*>(h)->table_size(slot, g); }
XB_API int xb_cm_copy_table(void* h, int slot, int g, int32_t* out, int cap) { return static_cast<CacheManager*>(h)->copy_table(slot, g, out, cap); }
XB_API int xb_cm_live_requests(void* h) { return static_cast<CacheManager*>(h)->live_requests(); }
XB_API void xb_cm_log_freed(void* h, int on) { static_cast<CacheManager*>(h)->log_freed(on != 0); }
XB_API int xb_cm_drain_freed(void* h, int32_t* groups, int32_t* pages, int cap) {
    return static_cast<CacheManager*>(h)->drain_freed(groups, pages, cap);
}
XB_API int xb_cm_consistent(void* h, char* why, int cap) {
    std::string s;
    const bool ok = static_cast<CacheManager*>(h)->consistent(&s);
    if (why && cap > 0) {
        std::strncpy(why, s.c_str(), cap - 1);
        why[cap - 1] = 0;
    }
    return ok ? 1 : 0;
}

// ---- step metadata ---------------------------------------------------------------------------
// Packs, for B entries (slot, count, tokens) whose start is the slot's cached length:
//   token_ids[Tp] positions[Tp] req_of_token[Tp] q_start[Bp+1] start_pos[Bp] slots[Bp]
//   logit_rows[Rp] and, per group, block_table[Bp, stride_g]
// Tp/Bp/Rp are T, B and R padded up to pad_tokens / pad_entries / pad_rows (padding rows read
// row 0; padding tokens belong to request -1
// and are skipped by the kernels); every array starts on a 16-byte boundary.  `strides` holds a
// wanted row length per group (0: as long as the longest table here, rounded up to 8).
// offsets_out[0..6] = array offsets in int32 units, [7 + g] = table offset of group g,
// [7 + G + g] = stride of group g, and the return value is the number of int32 used
// (negative on error: -1 capacity, -2 slot not live, -3 pages missing, -4 bad want).
XB_API long long xb_assemble(void* h, int B, const int* slots, const int* counts, const int* tokens,
                             int R, const int* want_entry, const int* want_offset, int pad_tokens,
                             int pad_entries, int pad_rows, const int* strides, int32_t* out, long long capacity,
                             long long* offsets_out) {
    CacheManager* cm = static_cast<CacheManager*>(h);
    const int G = cm->num_groups();
    int T = 0;
    for (int b = 0; b < B; ++b) {
        if (!cm->is_live(slots[b]) || counts[b] <= 0) return -2;
        T += counts[b];
    }
    const int Tp = std::max(T, pad_tokens), Bp = std::max(B, pad_entries), Rp = std::max(std::max(R, pad_rows), 1);
    auto up4 = [](long long x) { return (x + 3) / 4 * 4; };
    std::vector<int> stride(G);
    for (int g = 0; g < G; ++g) {
        int longest = 1;
        const int ps = cm->group(g).page_size;
        for (int b = 0; b < B; ++b) {
            const int new_len = cm->length(slots[b]) + counts[b];
            if (cm->table_size(slots[b], g) * ps < new_len) return -3;
            longest = std::max(longest, (new_len + ps - 1) / ps);
        }
        stride[g] = (longest + 7) / 8 * 8;
        if (strides && strides[g] > 0) {
            if (strides[g] < longest) return -1;
            stride[g] = strides[g];
        }
    }
    long long off = 0;
    long long o_tok = off; off = up4(off + Tp);
    long long o_pos = off; off = up4(off + Tp);
    long long o_req = off; off = up4(off + Tp);
    long long o_qs = off; off = up4(off + Bp + 1);
    long long o_sp = off; off = up4(off + Bp);
    long long o_sl = off; off = up4(off + Bp);
    long long o_rows = off; off = up4(off + Rp);
    std::vector<long long> o_tab(G);
    for (int g = 0; g < G; ++g) {
        o_tab[g] = off;
        off = up4(off + (long long)Bp * stride[g]);
    }
    if (off > capacity) return -1;
    int t = 0;
    for (int b = 0; b < B; ++b) {
        const int start = cm->length(slots[b]);
        out[o_qs + b] = t;
        out[o_sp + b] = start;
        out[o_sl + b] = slots[b];
        for (int i = 0; i < counts[b]; ++i, ++t) {
            out[o_tok + t] = tokens[t];
            out[o_pos + t] = start + i;
            out[o_req + t] = b;
        }
    }
    for (int b = B; b <= Bp; ++b) out[o_qs + b] = T;
    for (int b = B; b < Bp; ++b) {
        out[o_sp + b] = 0;
        out[o_sl + b] = -1;
    }
    for (; t < Tp; ++t) {
        out[o_tok + t] = 0;
        out[o_pos + t] = 0;
        out[o_req + t] = -1;
    }
    for (int r = 0; r < R; ++r) {
        const int e = want_entry[r];
        if (e < 0 || e >= B || want_offset[r] < 0 || want_offset[r] >= counts[e]) return -4;
        out[o_rows + r] = out[o_qs + e] + want_offset[r];
    }
    for (int r = R; r < Rp; ++r) out[o_rows + r] = 0;
    for (int g = 0; g < G; ++g) {
        for (int b = 0; b < Bp; ++b) {
            int32_t* row = out + o_tab[g] + (long long)b * stride[g];
            int n = 0;
            if (b < B) n = cm->copy_table(slots[b], g, row, stride[g]);
            for (int i = std::max(n, 0); i < stride[g]; ++i) row[i] = -1;
        }
    }
    offsets_out[0] = o_tok; offsets_out[1] = o_pos; offsets_out[2] = o_req; offsets_out[3] = o_qs;
    offsets_out[4] = o_sp; offsets_out[5] = o_sl; offsets_out[6] = o_rows;
    for (int g = 0; g < G; ++g) {
        offsets_out[7 + g] = o_tab[g];
        offsets_out[7 + G + g] = stride[g];
    }
    return off;
}

// ---- work lists of the prefill attention kernel ---------------------------------------------------
// The step's portions of more than dec_max tokens are cut into items of 128 queries (a query tile) of
// two query heads that share a key/value head (one head where a group has an odd head left); an item's
// cost is its number of 64-key tiles times the cost of a tile (of two heads, or of one) plus a fixed
// start-up.  The items go, longest first, each onto the CTA with the least work so far, so that all CTAs
// end together whatever the portions' lengths are; items of equal cost - the heads of one query tile,
// which read the same keys - land on different CTAs and run at the same time.  The same is tried with
// one head per item (twice the items, each two thirds as long), and the cut that ends earlier is taken:
// one head where two-head items would leave CTAs idle (short portions, few heads), two otherwise.
// out: [ctas + 1] offsets (in items) then 4 int32 per item: portion, query tile, first query head, heads.
// Returns the number of int32 written (-1: capacity too small) and the number of CTAs in *ctas_out.
// keep_first > 0 (beside a sliding window): the key tiles of the sequence's first keep_first positions count too.
XB_API long long xb_attn_prefill_work(int B, const int* counts, const int* starts, int dec_max, int window,
                                      int keep_first, int heads, int kv_heads, int max_ctas, int32_t* out, long long capacity,
                                      int* ctas_out) {
    // costs in sixths of a key tile of two heads: a tile of one head takes about two thirds of the time of a tile
    // of two (measured at long contexts: 0.76 us against 1.15 us), an item's start about three tiles
    constexpr int QT = 128, KT = 64, TILE_OF_TWO = 6, TILE_OF_ONE = 4, START_UP = 18, INTS = 4;
    struct Tile { int tiles, b, tile; };
    std::vector<Tile> tiles;
    for (int b = 0; b < B; ++b) {
        const int n = counts[b];
        if (n <= dec_max) continue;
        for (int ti = 0; ti * QT < n; ++ti) {
            const int p0 = starts[b] + ti * QT, rows = std::min(QT, n - ti * QT);
            // window > 0: a sliding window; window < 0: chunks of -window positions counted from position 0
            const int last_key = p0 + rows - 1;
            const int first_key = window > 0 ? std::max(0, p0 - window + 1) : (window < 0 ? p0 / (-window) * (-window) : 0);
            const int kept = window > 0 && keep_first > 0 ? std::min((keep_first + KT - 1) / KT, first_key / KT) : 0;
            tiles.push_back({kept + last_key / KT - first_key / KT + 1, b, ti});
        }
    }
    *ctas_out = 0;
    if (tiles.empty() || heads <= 0 || kv_heads <= 0 || heads % kv_heads) return 0;
    std::stable_sort(tiles.begin(), tiles.end(), [](const Tile& x, const Tile& y) { return x.tiles > y.tiles; });
    const int G = heads / kv_heads, per_group = (G + 1) / 2;
    struct Head { int h0, nhd; };
    struct Shared { std::vector<std::vector<int32_t>> lists; long long longest = 0, n_items = 0; };
    // items of two heads (`singles` false) or of one, shared out: least loaded CTA first, ties to the lower index
    auto share_out = [&](bool singles, Shared& made) {
        std::vector<Head> head_items;
        for (int g = 0; g < kv_heads; ++g) {
            if (singles) {
                for (int h = 0; h < G; ++h) head_items.push_back({g * G + h, 1});
            } else {
                for (int pr = 0; pr < per_group; ++pr) head_items.push_back({g * G + 2 * pr, 2 * pr + 1 < G ? 2 : 1});
            }
        }
        made.n_items = (long long)tiles.size() * (long long)head_items.size();
        const int ctas = (int)std::min<long long>(max_ctas, made.n_items);
        std::vector<std::pair<long long, int>> heap;
        for (int c = 0; c < ctas; ++c) heap.emplace_back(0, c);
        auto later = [](const std::pair<long long, int>& x, const std::pair<long long, int>& y) { return x > y; };
        std::make_heap(heap.begin(), heap.end(), later);
        made.lists.assign(ctas, {});
        for (const Tile& t : tiles) {
            for (const Head& h : head_items) {
                std::pop_heap(heap.begin(), heap.end(), later);
                auto& top = heap.back();
                made.lists[top.second].insert(made.lists[top.second].end(), {t.b, t.tile, h.h0, h.nhd});
                top.first += (long long)t.tiles * (h.nhd == 2 ? TILE_OF_TWO : TILE_OF_ONE) + START_UP;
                made.longest = std::max(made.longest, top.first);
                std::push_heap(heap.begin(), heap.end(), later);
            }
        }
    };
    // two heads per item load a key/value tile once for both; one head per item gives twice as many items to
    // fill the CTAs with.  Whichever ends earlier by these costs is taken (a few thousand items at most).
    Shared made;
    share_out(false, made);
    if (G >= 2) {
        Shared ones;
        share_out(true, ones);
        if (ones.longest < made.longest) made = std::move(ones);
    }
    const std::vector<std::vector<int32_t>>& lists = made.lists;
    const long long n_items = made.n_items;
    const int ctas = (int)lists.size();
    *ctas_out = ctas;
    if ((long long)ctas + 1 + INTS * n_items > capacity) return -1;
    int32_t* items = out + ctas + 1;
    int at = 0;
    for (int c = 0; c < ctas; ++c) {
        out[c] = at;
        std::copy(lists[c].begin(), lists[c].end(), items + INTS * (long long)at);
        at += (int)lists[c].size() / INTS;
    }
    out[ctas] = at;
    return (long long)ctas + 1 + INTS * n_items;
}

// What a step's portions bring and see, of those of more than `most` tokens and of the others:
// out[0..4]: portions, tokens, keys seen, pairs of query and key, longest walk of a query over keys; out[5..9]: of the others.
XB_API void xb_portion_sums(int B, const int* q_start, const int* starts, int most, int window, double* out) {
    for (int i = 0; i < 10; ++i) out[i] = 0;
    for (int b = 0; b < B; ++b) {
        const double n = q_start[b + 1] - q_start[b], before = window > 0 ? std::min(starts[b], window) : starts[b];
        double* o = out + (n > most ? 0 : 5), pairs = n * before + n * (n + 1) / 2;
        if (window > 0) pairs = std::min(pairs, n * window);
        o[0] += 1;
        o[1] += n;
        o[2] += before + n;
        o[3] += pairs;
        o[4] = std::max(o[4], before + n);
    }
}

// ---- work lists of the attention over keys and values formed for the step --------------------------
// The step's portions of more than dec_max tokens: their visible rows lie one portion after the other, from the 64-key
// tile of the first query's first key on, in runs of 64 rows.  Items are 256 (or 128) queries of one head; they go,
// longest first, onto the CTA with the least work so far, and the cut into items that ends earlier is taken.
// out: [ctas + 1] offsets (in items), 4 int32 per item (portion, first query of it, head | tiles of 128 queries << 16,
// row of the position 0), then (portion, first position) of every run of 64 rows.  Returns the number of int32 written
// (-1: capacity too small), the number of CTAs and of rows.
XB_API long long xb_latent_prefill_work(int B, const int* counts, const int* starts, int dec_max, int window, int heads,
                                        int max_ctas, int32_t* out, long long capacity, int* ctas_out, int* rows_out) {
    // costs in sixths of a key tile of two query tiles, as for the kernel over pages
    constexpr int QT = 128, KT = 64, TILE_OF_TWO = 6, TILE_OF_ONE = 4, START_UP = 18, INTS = 4;
    struct Piece { int cost, b, first, nt, row0; };
    std::vector<int32_t> runs;
    std::vector<Piece> cuts[2];       // [0]: two query tiles per item where a portion has them, [1]: one
    for (int b = 0; b < B; ++b) {
        const int n = counts[b];
        if (n <= dec_max) continue;
        const int base = (window > 0 ? std::max(0, starts[b] - window + 1) : 0) / KT * KT, end = starts[b] + n;
        const int row0 = (int)runs.size() / 2 * KT - base;
        for (int j = base; j < end; j += KT) {
            runs.push_back(b);
            runs.push_back(j);
        }
        for (int c = 0; c < 2; ++c) {
            for (int first = 0, nt; first < n; first += nt * QT) {
                nt = c == 0 && n - first > QT ? 2 : 1;
                const int p0 = starts[b] + first, last = p0 + std::min(nt * QT, n - first) - 1;
                const int lo = (window > 0 ? std::max(0, p0 - window + 1) : 0) / KT;
                cuts[c].push_back({(last / KT - lo + 1) * (nt == 2 ? TILE_OF_TWO : TILE_OF_ONE) + START_UP, b, first, nt, row0});
            }
        }
    }
    *ctas_out = 0;
    *rows_out = (int)runs.size() / 2 * KT;
    if (runs.empty() || heads <= 0 || heads > 65535) return 0;
    std::vector<std::vector<int32_t>> lists[2];
    long long longest[2] = {0, 0};
    for (int c = 0; c < 2; ++c) {
        std::stable_sort(cuts[c].begin(), cuts[c].end(), [](const Piece& x, const Piece& y) { return x.cost > y.cost; });
        const int ctas = (int)std::min<long long>(max_ctas, (long long)cuts[c].size() * heads);
        std::vector<std::pair<long long, int>> heap;
        for (int i = 0; i < ctas; ++i) heap.emplace_back(0, i);
        auto later = [](const std::pair<long long, int>& x, const std::pair<long long, int>& y) { return x > y; };
        std::make_heap(heap.begin(), heap.end(), later);
        lists[c].assign(ctas, {});
        for (const Piece& p : cuts[c]) {
            for (int h = 0; h < heads; ++h) {
                std::pop_heap(heap.begin(), heap.end(), later);
                auto& top = heap.back();
                lists[c][top.second].insert(lists[c][top.second].end(), {p.b, p.first, h | p.nt << 16, p.row0});
                top.first += p.cost;
                longest[c] = std::max(longest[c], top.first);
                std::push_heap(heap.begin(), heap.end(), later);
            }
        }
    }
    const int take = longest[1] < longest[0] ? 1 : 0;
    const long long n_items = (long long)cuts[take].size() * heads;
    const int ctas = (int)lists[take].size();
    *ctas_out = ctas;
    const long long used = ctas + 1 + INTS * n_items + (long long)runs.size();
    if (used > capacity) return -1;
    int32_t* items = out + ctas + 1;
    int at = 0;
    for (int c = 0; c < ctas; ++c) {
        out[c] = at;
        std::copy(lists[take][c].begin(), lists[take][c].end(), items + INTS * (long long)at);
        at += (int)lists[take][c].size() / INTS;
    }
    out[ctas] = at;
    std::copy(runs.begin(), runs.end(), items + INTS * n_items);
    return used;
}

// ---- work lists of the attention with talking heads over many tokens -------------------------------
// All portions of the step, cut into blocks of 128 queries whose score tiles (128 queries x 32 keys of one head, from the
// first query's first key on, aligned to 128 keys) lie one after the other: [head][32-key tile].  Blocks are taken in order
// into chunks of at most cap_tiles tiles; a chunk is one pair of launches.  Per chunk: its blocks, the items of the first
// launch (512 / heads queries of a block x a run of 128-key tiles) and of the second (a block x two heads of a key/value
// head), each shared out longest first onto the CTA with the least work so far.
// out: per chunk 6 int32 per block (portion, first query of it, first 32-key tile, 32-key tiles, first score tile, 0), then
// [ctas + 1] offsets and 4 int32 per item (block, query tile, first 128-key tile, how many), then the same for the second
// launch (block, first head, heads, 0).  chunks: 5 int32 per chunk: where its blocks, first and second list begin, CTAs of
// both.  Returns the number of chunks, -1 where out or chunks are too small, -2 where one block has more than cap_tiles.
namespace {
struct WorkItem { long long cost; int32_t v[4]; };
int share_items(std::vector<WorkItem>& items, int max_ctas, std::vector<int32_t>& out, long long* longest = nullptr) {
    std::stable_sort(items.begin(), items.end(), [](const WorkItem& x, const WorkItem& y) { return x.cost > y.cost; });
    const int ctas = (int)std::min<size_t>(max_ctas, items.size());
    std::vector<std::vector<int32_t>> lists(ctas);
    std::vector<std::pair<long long, int>> heap;
    for (int i = 0; i < ctas; ++i) heap.emplace_back(0, i);
    auto later = [](const std::pair<long long, int>& x, const std::pair<long long, int>& y) { return x > y; };
    std::make_heap(heap.begin(), heap.end(), later);
    if (longest) *longest = 0;
    for (const WorkItem& it : items) {
        std::pop_heap(heap.begin(), heap.end(), later);
        auto& top = heap.back();
        lists[top.second].insert(lists[top.second].end(), it.v, it.v + 4);
        top.first += it.cost;
        if (longest) *longest = std::max(*longest, top.first);
        std::push_heap(heap.begin(), heap.end(), later);
    }
    int at = 0;
    for (int c = 0; c < ctas; ++c) {
        out.push_back(at);
        at += (int)lists[c].size() / 4;
    }
    out.push_back(at);
    for (const auto& l : lists) out.insert(out.end(), l.begin(), l.end());
    return ctas;
}
}  // namespace

XB_API int xb_talk_work(int B, const int* counts, const int* starts, int window, int heads, int kv_heads, int max_ctas,
                        long long cap_tiles, int32_t* out, long long capacity, int32_t* chunks, int max_chunks,
                        long long* used_out, long long* tiles_out) {
    constexpr int ROWS = 128, KEYS = 128;
    struct Block { int b, first, kb0, nkb, rows, p0; };
    std::vector<Block> blocks;
    auto first_key = [&](int p) { return window > 0 ? std::max(0, p - window + 1) : 0; };
    for (int b = 0; b < B; ++b)
        for (int first = 0; first < counts[b]; first += ROWS) {
            const int p0 = starts[b] + first, rows = std::min(ROWS, counts[b] - first);
            const int lo = first_key(p0) / KEYS, hi = (p0 + rows - 1) / KEYS;
            blocks.push_back({b, first, lo * 4, (hi - lo + 1) * 4, rows, p0});
        }
    *used_out = *tiles_out = 0;
    const int qn = 512 / heads, per = 128 / heads, rep = heads / kv_heads;
    std::vector<int32_t> all;
    int n_chunks = 0;
    for (size_t at = 0; at < blocks.size();) {
        size_t end = at;
        long long tiles = 0;
        while (end < blocks.size() && tiles + (long long)blocks[end].nkb * heads <= cap_tiles) tiles += (long long)blocks[end++].nkb * heads;
        if (end == at) return -2;
        if (n_chunks == max_chunks) return -1;
        int32_t* ch = chunks + 5 * n_chunks++;
        *tiles_out = std::max(*tiles_out, tiles);
        ch[0] = (int32_t)all.size();
        long long tile0 = 0, key_tiles = 0;
        for (size_t i = at; i < end; ++i) {
            const Block& k = blocks[i];
            const int32_t rec[6] = {k.b, k.first, k.kb0, k.nkb, (int32_t)tile0, 0};
            all.insert(all.end(), rec, rec + 6);
            tile0 += (long long)k.nkb * heads;
            key_tiles += (long long)(k.nkb / 4) * ((k.rows + qn - 1) / qn);
        }
        // runs of key tiles short enough to share them out evenly, long enough that the queries are not loaded often
        const int run = (int)std::max<long long>(4, key_tiles / (4LL * max_ctas));
        std::vector<WorkItem> one, two, singles;
        for (size_t i = at; i < end; ++i) {
            const Block& k = blocks[i];
            for (int qt = 0; qt * qn < k.rows; ++qt) {
                const int rows = std::min(qn, k.rows - qt * qn), p0 = k.p0 + qt * qn;
                const int lo = first_key(p0) / KEYS, hi = (p0 + rows - 1) / KEYS;
                const int batches = (std::min(rows, qn / 2) + per - 1) / per;      // of the warps that have most queries
                for (int kt = lo; kt <= hi; kt += run) {
                    const int n = std::min(run, hi - kt + 1);
                    one.push_back({(long long)n * (1 + 4 * batches) + 3, {(int32_t)(i - at), qt, kt, n}});
                }
            }
            const int n = (k.p0 + k.rows - 1) / 64 - first_key(k.p0) / 64 + 1;
            for (int g = 0; g < kv_heads; ++g)
                for (int h = 0; h < rep; h += 2) {
                    const int nh = std::min(2, rep - h);
                    two.push_back({(long long)n * (nh == 2 ? 6 : 4) + 18, {(int32_t)(i - at), g * rep + h, nh, 0}});
                }
            for (int h = 0; h < heads; ++h) singles.push_back({(long long)n * 4 + 18, {(int32_t)(i - at), h, 1, 0}});
        }
        ch[1] = (int32_t)all.size();
        ch[3] = share_items(one, max_ctas, all);
        ch[2] = (int32_t)all.size();
        // items of two heads load a value tile once for both; where those are too few to fill the CTAs, one head each
        long long longest[2];
        std::vector<int32_t> lists[2];
        const int n2 = share_items(two, max_ctas, lists[0], &longest[0]), n1 = share_items(singles, max_ctas, lists[1], &longest[1]);
        const int take = longest[1] < longest[0] ? 1 : 0;
        ch[4] = take ? n1 : n2;
        all.insert(all.end(), lists[take].begin(), lists[take].end());
        at = end;
    }
    *used_out = (long long)all.size();
    if (*used_out > capacity) return -1;
    std::copy(all.begin(), all.end(), out);
    return n_chunks;
}

// ---- scheduler ---------------------------------------------------------------------------------
struct SchedHandle {
    Scheduler sched;
    std::vector<StepEntry> last;    // scheduled, not yet committed
    std::vector<StepEntry> ahead;   // the step after `last`, decided while `last` runs
    SchedHandle(CacheManager* c, const SchedulerConfig& cfg) : sched(c, cfg) {}
};

XB_API void* xb_sched_create(void* cm, int max_num_seqs, int max_batched_tokens, int prefill_chunk,
                             int max_model_len, const int* eos_ids, int n_eos) {
    if (!cm || max_num_seqs <= 0 || max_batched_tokens <= 0 || prefill_chunk <= 0 || max_model_len <= 1) return nullptr;
    SchedulerConfig cfg;
    cfg.max_num_seqs = max_num_seqs;
    cfg.max_num_batched_tokens = max_batched_tokens;
    cfg.prefill_chunk_size = prefill_chunk;
    cfg.max_model_len = max_model_len;
    if (n_eos > 0) cfg.eos_token_ids.assign(eos_ids, eos_ids + n_eos);
    return new SchedHandle(static_cast<CacheManager*>(cm), cfg);
}
XB_API void xb_sched_destroy(void* h) { delete static_cast<SchedHandle*>(h); }
XB_API int xb_sched_add(void* h, long long req_id, const int* prompt, int n, int max_tokens, int ignore_eos,
                        const int* stop_ids, const int* stop_lens, int n_stop) {
    return (int)static_cast<SchedHandle*>(h)->sched.add(req_id, prompt, n, max_tokens, ignore_eos != 0, stop_ids, stop_lens, n_stop);
}
XB_API int xb_sched_abort(void* h, long long req_id) { return static_cast<SchedHandle*>(h)->sched.abort(req_id) ? 1 : 0; }

// Returns the number of entries (or -1 if the arrays are too small) and keeps them for commit.
XB_API int xb_sched_schedule(void* h, int cap_entries, long long* req_ids, int* slots, int* starts,
                             int* counts, int* wants, int cap_tokens, int* tokens, int* n_tokens) {
    SchedHandle* s = static_cast<SchedHandle*>(h);
    std::vector<int32_t> toks;
    s->last = s->sched.schedule(&toks);
    if ((int)s->last.size() > cap_entries || (int)toks.size() > cap_tokens) return -1;
    for (size_t i = 0; i < s->last.size(); ++i) {
        req_ids[i] = s->last[i].req_id;
        slots[i] = s->last[i].slot;
        starts[i] = s->last[i].start;
        counts[i] = s->last[i].count;
        wants[i] = s->last[i].want ? 1 : 0;
    }
    std::copy(toks.begin(), toks.end(), tokens);
    *n_tokens = (int)toks.size();
    return (int)s->last.size();
}
// Commits the oldest uncommitted step; a step decided ahead becomes the one awaiting commit.
XB_API void xb_sched_commit(void* h, const int* sampled, int n_sampled) {
    SchedHandle* s = static_cast<SchedHandle*>(h);
    std::vector<int32_t> v(sampled, sampled + (n_sampled > 0 ? n_sampled : 0));
    s->sched.commit(s->last, v);
    s->last.swap(s->ahead);
    s->ahead.clear();
}
// The step after the uncommitted one (see Scheduler::schedule_ahead).  Returns the number of
// entries, 0 when it cannot be decided ahead, -1 if the arrays are too small.
XB_API int xb_sched_schedule_ahead(void* h, int cap_entries, long long* req_ids, int* slots, int* starts, int* src) {
    SchedHandle* s = static_cast<SchedHandle*>(h);
    if (!s->ahead.empty()) return 0;
    std::vector<int> from;
    std::vector<StepEntry> e = s->sched.schedule_ahead(s->last, &from);
    if ((int)e.size() > cap_entries) return -1;
    for (size_t i = 0; i < e.size(); ++i) {
        req_ids[i] = e[i].req_id;
        slots[i] = e[i].slot;
        starts[i] = e[i].start;
        src[i] = from[i];
    }
    s->ahead = e;
    return (int)e.size();
}
// A scheduled step failed on the device or on the way there: every request of the steps that are
// scheduled and not committed (the running one and the one decided ahead) ends as aborted, its pages
// go back, and nothing stays scheduled.  Returns how many requests that ended.
XB_API int xb_sched_fail_steps(void* h) {
    SchedHandle* s = static_cast<SchedHandle*>(h);
    int n = 0;
    for (std::vector<StepEntry>* v : {&s->last, &s->ahead}) {
        for (const StepEntry& e : *v)
            if (s->sched.abort(e.req_id)) ++n;
        v->clear();
    }
    return n;
}
XB_API int xb_sched_drain_finished(void* h, long long* out, int cap) {
    auto v = static_cast<SchedHandle*>(h)->sched.drain_finished();
    const int n = std::min((int)v.size(), cap);
    for (int i = 0; i < n; ++i) out[i] = v[i];
    return n;
}
XB_API int xb_sched_num_waiting(void* h) { return static_cast<SchedHandle*>(h)->sched.num_waiting(); }
XB_API int xb_sched_num_running(void* h) { return static_cast<SchedHandle*>(h)->sched.num_running(); }
XB_API int xb_sched_preemptions(void* h) { return static_cast<SchedHandle*>(h)->sched.preemptions(); }
XB_API int xb_sched_finish_reason(void* h, long long id) { return static_cast<SchedHandle*>(h)->sched.finish_reason(id); }
XB_API int xb_sched_output_length(void* h, long long id) { return static_cast<SchedHandle*>(h)->sched.output_length(id); }
XB_API int xb_sched_copy_output(void* h, long long id, int* out, int cap) { return static_cast<SchedHandle*>(h)->sched.copy_output(id, out, cap); }
XB_API int xb_sched_prompt_length(void* h, long long id) { return static_cast<SchedHandle*>(h)->sched.prompt_length(id); }
XB_API int xb_sched_num_drawn(void* h, long long id) { return static_cast<SchedHandle*>(h)->sched.num_drawn(id); }
XB_API int xb_sched_copy_tail(void* h, long long id, int* out, int n) { return static_cast<SchedHandle*>(h)->sched.copy_tail(id, out, n); }
XB_API int xb_sched_release(void* h, long long id) { return static_cast<SchedHandle*>(h)->sched.release(id) ? 1 : 0; }
