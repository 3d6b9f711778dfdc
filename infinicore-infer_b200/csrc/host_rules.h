// Rules of the engine that run on the host and that more than one part of it follows, each written ONCE.
//
// Plain C++ without CUDA: the Python engine calls them through libjk_host.so (host.cpp gives them C names), the native
// step (runner.cu) and the C interface (capi.cu) include this header.  What lives here:
//   - the page pool behind a cache group (which pages are free, last freed first, never page 0);
//   - the layout of a step's metadata buffer and the packing of a batch into it;
//   - the attention mixer's work lists (rows of requests that bring few rows, tiles of the others);
//   - how many ways the decode attention cuts a row's keys;
//   - which kernel takes a product of a given shape;
//   - the rotary tables;
//   - the uniform number for the token at a position of a request.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

namespace jk {

// ---- the page pool ---------------------------------------------------------------------------------------------
// Pages are handed out last-freed-first, so a page that a finished request gave back is the next one to be used
// again.  The first `reserved` pages are never handed out; page 0 is the null page that padding rows read and write.
class PagePool {
  public:
    PagePool(int num_pages, int reserved) : num_pages_(num_pages), reserved_(reserved), held_((size_t)num_pages, 0) {
        free_.reserve((size_t)num_pages);
        for (int p = num_pages - 1; p >= reserved; --p) free_.push_back(p);      // the lowest page goes out first
    }
    int capacity() const { return num_pages_ - reserved_; }
    int available() const { return (int)free_.size(); }
    int in_use() const { return capacity() - available(); }
    int high_water() const { return high_water_; }
    int num_pages() const { return num_pages_; }
    int reserved() const { return reserved_; }
    // n pages into out; false (and nothing taken) if fewer are free
    bool alloc(int n, int *out) {
        if (n < 0 || n > (int)free_.size()) return false;
        for (int i = 0; i < n; ++i) {
            out[i] = free_.back();
            free_.pop_back();
            held_[(size_t)out[i]] = 1;
        }
        high_water_ = std::max(high_water_, in_use());
        return true;
    }
    // 0 ok; 1 a page that is not this pool's; 2 a page that is not out (freed twice); 3 a page twice in one call.
    // Nothing is freed unless all of them can be.
    int free(const int *pages, int n) {
        for (int i = 0; i < n; ++i) {
            if (pages[i] < reserved_ || pages[i] >= num_pages_) return 1;
            if (!held_[(size_t)pages[i]]) return 2;
        }
        for (int i = 0; i < n; ++i) {
            if (held_[(size_t)pages[i]] == 2) {
                for (int j = 0; j < i; ++j) held_[(size_t)pages[j]] = 1;
                return 3;
            }
            held_[(size_t)pages[i]] = 2;
        }
        for (int i = 0; i < n; ++i) {
            held_[(size_t)pages[i]] = 0;
            free_.push_back(pages[i]);
        }
        return 0;
    }
    bool is_held(int page) const { return page >= 0 && page < num_pages_ && held_[(size_t)page] != 0; }

  private:
    int num_pages_, reserved_, high_water_ = 0;
    std::vector<int> free_;
    std::vector<unsigned char> held_;
};

// ---- a step's metadata -----------------------------------------------------------------------------------------
constexpr int MAX_CACHE_GROUPS = 8;
constexpr int MAX_STEP_LISTS = 8;

inline int align4(int n) { return (n + 3) & ~3; }

// Offsets (in 32-bit words) of a step's arrays inside the one buffer that is copied to the device per step: what
// every model needs (tokens, positions, the request of each row, the wanted rows, each request's first row, first
// position and state slot, a block table per cache group), then `extra_words` for the work lists that the model's
// mixers ask for (see attention_work_lists below for this architecture's).
struct StepLayout {
    int tokens, positions, row_req, want_rows, req_start, req_pos, slot_ids;
    int tables[MAX_CACHE_GROUPS];
    int extra, total;
    StepLayout(int T, int B, int n_groups, int max_blocks, int extra_words) {
        int o = 0;
        tokens = o; o += align4(T);
        positions = o; o += align4(T);
        row_req = o; o += align4(T);
        want_rows = o; o += align4(T);
        req_start = o; o += align4(B + 1);
        req_pos = o; o += align4(B);
        slot_ids = o; o += align4(B);
        for (int g = 0; g < MAX_CACHE_GROUPS; ++g) {
            tables[g] = o;
            if (g < n_groups) o += align4(B * max_blocks);
        }
        extra = o; o += align4(extra_words);
        total = o;
    }
};

// Packs a batch of B requests (request i brings lens[i] tokens that start at position starts[i]; padded to pad_B
// requests by requests of one row that use slot 0 and the null page at position 0) into `host`, which holds
// `lay.total` zeroed words.  `tables[g]` is [B, max_blocks] page ids, or null (then the caller fills that table);
// `want` lists the wanted places as row indices of the whole step.  Returns the number of rows.
inline int pack_step(int *host, const StepLayout &lay, int B, int pad_B, const int *tokens, const int *lens, const int *starts,
                     const int *slots, const int *want, int n_want, int n_groups, int max_blocks, const int *const *tables) {
    int row = 0;
    for (int i = 0; i < B; ++i) {
        const int n = lens[i], s = starts[i];
        host[lay.req_start + i] = row;
        host[lay.req_pos + i] = s;
        host[lay.slot_ids + i] = slots ? slots[i] : 0;
        for (int t = 0; t < n; ++t) {
            host[lay.tokens + row + t] = tokens[row + t];
            host[lay.positions + row + t] = s + t;
            host[lay.row_req + row + t] = i;
        }
        row += n;
    }
    for (int i = B; i < pad_B; ++i) {       // padding rows of a captured step
        host[lay.req_start + i] = row;
        host[lay.row_req + row] = i;
        ++row;
    }
    host[lay.req_start + pad_B] = row;
    for (int i = 0; i < n_want; ++i) host[lay.want_rows + i] = want[i];
    for (int g = 0; g < n_groups; ++g)
        if (tables && tables[g]) memcpy(host + lay.tables[g], tables[g], sizeof(int) * (size_t)B * max_blocks);
    return row;
}

// ---- the attention mixer's work lists ------------------------------------------------------------------------------
// The softmax attention of this architecture treats requests that bring few rows to a step and requests that bring
// many differently: a request with at most SHORT_ROWS rows goes to the split-key decode kernels row by row; the rows of
// the others are cut into tiles of TILE_ROWS query rows for the prefill kernels.  Its two lists: the short rows, and
// (request, first row) of every tile, the tiles that see the most keys first (the kernels start tiles in list order).
constexpr int SHORT_ROWS = 8;
constexpr int TILE_ROWS = 128;
inline int attention_short_rows_capacity(int T) { return align4(T); }
inline int attention_tiles_capacity(int T, int B) { return align4(2 * (T / TILE_ROWS + B)); }
struct AttentionLists {
    int n_short, n_tiles;
};
inline AttentionLists attention_work_lists(int B, int pad_B, const int *lens, const int *starts, int *short_rows, int *tiles) {
    struct Tile { int keys, req, row; };
    std::vector<Tile> found;
    AttentionLists c{0, 0};
    int row = 0;
    for (int i = 0; i < B; ++i) {
        const int n = lens[i];
        if (n <= SHORT_ROWS)
            for (int t = 0; t < n; ++t) short_rows[c.n_short++] = row + t;
        else
            for (int t0 = 0; t0 < n; t0 += TILE_ROWS) found.push_back({starts[i] + t0, i, row + t0});
        row += n;
    }
    for (int i = B; i < pad_B; ++i) short_rows[c.n_short++] = row++;
    std::stable_sort(found.begin(), found.end(), [](const Tile &a, const Tile &b) { return a.keys > b.keys; });
    for (size_t t = 0; t < found.size(); ++t) {
        tiles[2 * t] = found[t].req;
        tiles[2 * t + 1] = found[t].row;
    }
    c.n_tiles = (int)found.size();
    return c;
}

// The first key that a query at `pos` sees (jk_mask_lo of csrc/common.cuh).
inline int mask_lo(int pos, int window) { return window > 0 ? std::max(pos - window + 1, 0) : window < 0 ? pos / -window * -window : 0; }
// The keys that a step's query tiles walk, counted in the longest one's: req_start [nreq + 1], req_pos [nreq].
inline double attention_tile_load(int nreq, const int *req_start, const int *req_pos, int window) {
    long long sum = 0, most = 0;
    for (int r = 0; r < nreq; ++r) {
        const int n = req_start[r + 1] - req_start[r];
        for (int t0 = 0; t0 < n && n > SHORT_ROWS; t0 += TILE_ROWS) {
            const long long keys = req_pos[r] + std::min(t0 + TILE_ROWS, n) - mask_lo(req_pos[r] + t0, window);
            sum += keys;
            most = std::max(most, keys);
        }
    }
    return most > 0 ? (double)sum / (double)most : 0.0;
}
// Keys a tile of the tcgen05 prefill attention, heads of 128.  Tiles of 64 let two blocks share an SM: more keys an SM and microsecond, but
// a block alone walks its own at 0.82 of the rate of tiles of 128.  So they pay where the blocks' work makes more than one wave of the
// longest block (B200, tiles of 128 -> 64; work in longest blocks over 148 SMs): 16 heads, 2,048 rows 45 -> 52 us (0.9); after 1,000 positions
// 76 -> 75 (1.2), after 4,000 164 -> 138 (1.4); 1,024 rows after 4,000 87 -> 106 (0.8); 32 heads, 1,536 rows 55 -> 48 (1.4), 1,024 rows 32 -> 34
// (1.0), 128 rows after 4,000 72 -> 88 (0.2); 1,000 rows beside 64 after 3,000 56 -> 72 (0.5), beside 200 39 -> 34 (1.1).
inline int attention_tile_keys(int heads, double load, int sms) { return heads * load > sms ? 64 : 128; }

// ---- the pieces of a linear-attention recurrence -------------------------------------------------------------------
// A request that brings more than SCAN_PIECE rows to a step has its recurrence cut into pieces of that many rows, which
// run side by side and are then joined (csrc/mixers.cu); the others run from their state slot in one go.  A step of
// `rows` rows has at most scan_max_pieces(rows) pieces.
constexpr int SCAN_PIECE = 64;
inline long long scan_max_pieces(long long rows) { return 2 * rows / SCAN_PIECE + 1; }
// Whether the pieces of a recurrence run as tiled products within the piece (csrc/mixers.cu: piece_state, piece_rows): rows that read the
// state after their own write, sizes of whole vectors of four floats, and a constant decay per head; or a projected one (`rank` > 0) for
// heads of at most 128 key channels (a warp's four channels a lane), while its weights and a piece's columns fit shared memory.
inline bool scan_runs_tiled(int dk, int dv, int ld, int q_off, int k_off, int v_off, int rank, bool bonus) {
    const bool decay = rank == 0 ? dk <= 256 : dk <= 128 && (long long)rank * (SCAN_PIECE + dk + 1) <= 24 * 1024;
    return decay && !bonus && ((dk | dv | ld | q_off | k_off | v_off) & 3) == 0;
}
inline long long scan_scratch_floats(long long rows, int heads, int dk, int dv, bool projected) {
    return scan_max_pieces(rows) * heads * dk * dv + (projected ? (rows + scan_max_pieces(rows)) * heads * dk : 0);
}

// ---- how many ways the decode attention cuts each row's key range ------------------------------------------------
// It depends on the batch's size and on `keys`, the context length the step is planned for (a captured step keeps
// its grid, so the caller passes a bucket of the live lengths, not the lengths themselves).
// Head sizes 64 and 128 (the tensor-core kernel: a block per row, key/value head and up to 16 query heads, two blocks
// an SM), from measurements on the 1B, 2B and 8B shapes: as many cuts as make the blocks fill the SMs once (rounded),
// as long as a block keeps 256 keys; then further, up to two rounds of blocks, as long as a block keeps 1024 keys (a
// block's fixed part costs about as much as a few hundred keys, and blocks that all start and end together read
// slower than blocks that overlap).  Other head sizes (the kernel of the CUDA cores, three blocks an SM): the choice
// weighs full waves of blocks against a block's fixed cost of about 128 keys' worth of time.
inline int decode_splits(int nrows, int nkvh, int group, int keys, int sms, int dh) {
    keys = std::max(1, keys);
    if (dh == 64 || dh == 128) {
        const long long blocks = std::max(1, nrows * nkvh * ((group + 15) / 16));
        const long long slots = 2LL * sms;
        long long s = std::max(1LL, std::min({(2 * slots + blocks) / (2 * blocks), (long long)keys / 256, 32LL}));
        while (blocks * (s + 1) <= 2 * slots && keys / (s + 1) >= 1024 && s < 32) ++s;
        // heads of 128: a launch of at most one block an SM runs blocks of eight warps, which pass keys twice as fast;
        // half the cuts is then better than two rounds of the narrow blocks (16 rows x 4,096 keys, 2 key/value heads:
        // 18.3 against 21.5 us)
        if (dh == 128 && blocks * s > sms && blocks * (s / 2) <= sms && s >= 2) s /= 2;
        return (int)s;
    }
    const long long blocks = std::max(1, nrows * nkvh * (group > 4 ? (group + 3) / 4 : 1));
    const long long slots = (long long)sms * 3;
    int best = 1;
    double best_cost = -1;
    for (int s = 1; s <= 32; ++s) {
        if (s > 1 && (double)keys / s < 64) break;
        const long long waves = (blocks * s + slots - 1) / slots;
        const double cost = waves * (128 + (double)keys / s);
        if (best_cost < 0 || cost < best_cost * 0.97) best = s, best_cost = cost;      // fewer cuts unless clearly better
    }
    return best;
}
// `keys` for a row that sees at most `window` keys (0: all) of a context planned for `context` positions: half of what a
// row can see stands for the lengths (the thresholds above were measured with that convention).
inline int decode_keys_hint(int context, int window) {
    const int reach = window > 0 ? std::min(window, context) : context;
    return std::max(1, reach / 2);
}
// floats of scratch that `splits` cuts of `nrows` rows need (partial outputs, maxima and sums); none for one cut
// (`dv`: the size of a value head)
inline long long decode_scratch_floats(int nrows, int nh, int dv, int splits) {
    return splits <= 1 ? 0 : (long long)nrows * nh * splits * (dv + 2);
}
// the head size by which decode_splits plans a launch: keys and values of unlike sizes run as heads of 64 or 128
inline int decode_head(int dh, int dv) { return dv > 0 && dv != dh ? ((dh > dv ? dh : dv) <= 64 ? 64 : 128) : dh; }
// The context length a step is planned for: the longest live request rounded up to a power of two, at least 4,096, at
// most the model's maximum.  Captured decode steps are kept per (batch bucket, this bucket), so a model with a context of
// 32k that serves short requests cuts their keys as a model of 4k would.  (Below 4,096 the measured optimum does not move:
// at 512 keys, batch 1 and 8, the cuts chosen for 4,096 are 3 % faster than those chosen for 1,024.)
inline int context_bucket(int longest, int max_positions) {
    int b = 4096;
    while (b < longest && b < max_positions) b *= 2;
    return std::min(b, std::max(1, max_positions));
}

// Head and page sizes for which the tcgen05 prefill attention is built (the page must divide a tile of 128 keys and
// fill whole groups of 8 swizzled rows): heads of 64 and 128, and keys and values of unlike sizes that are multiples of 8 up to 128
// (`dv` 0: as dh), which run padded to 64 or 128.
inline bool attention_unlike_heads(int dh, int dv) { return dv > 0 && dv != dh && dh % 8 == 0 && dv % 8 == 0 && dh <= 128 && dv <= 128; }
inline bool attention_tcgen05_takes(int dh, int page_size, int dv = 0) {
    const bool size = dv > 0 && dv != dh ? attention_unlike_heads(dh, dv) : (dh == 64 || dh == 128);
    return size && (page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64 || page_size == 128);
}

// ---- the float32 row attention's two kernels (csrc/attention.cu) -------------------------------------------------------------------
constexpr int ROW_PAIRS = 32;       // (row, head) pairs of a block at most
// Rows and heads of a block: as many heads of one key/value head as there are, then rows until the pairs are full, but fewer rows until there
// are three blocks for every SM (a block alone there waits for its chunks and its barriers).  `parts`: blocks a key/value head.
struct RowCut { int heads, rows; long long parts; };
inline RowCut attention_rows_cut(int T, int nh, int nkvh) {
    RowCut c;
    c.heads = std::min(nh / nkvh, ROW_PAIRS);
    c.rows = ROW_PAIRS / c.heads;
    c.parts = (nh / nkvh + c.heads - 1) / c.heads;
    while (c.rows > 1 && (T + c.rows - 1) / c.rows * c.parts * nkvh < 3 * 148) c.rows = (c.rows + 1) / 2;
    return c;
}
// Whether a warp a pair walks its keys in memory instead (attention_walk_kernel): where a block would have few pairs for its eight warps and
// there are more blocks than run at once, or where there are too few keys to make up for staging them.  `context`: the longest
// history that is known of (a bound); `size`: the larger of a key's and a value's; T rows of `nreq` requests.  Results are the same bits.
// B200, warps -> blocks (us), single rows after n keys where nothing else is said:
//   bfloat16, heads of 16 to 32, whose rows a lane reads with few lines: 512 requests, 4 heads of 16, n = 100 18 -> 70; one of them 13 -> 14, n = 1,000
//     96 -> 70; 512, 7 of 30, n = 100 38 -> 194, a prompt of 300 40 -> 66, of 2,048 744 -> 567; 1,024, 4 heads of 32 over one, n = 400 216 -> 116.
//   bfloat16, 512 requests, n = 100: 36 heads of 64 666 -> 701, 8 of 96 284 -> 310, 16 of 256 1,034 -> 2,129; 64, 16 of 256, n = 300 585 -> 676.
//   float32, 512 requests, n = 100: 4 heads of 16 37 -> 61, 7 of 30 151 -> 225, 16 of 256 1,134 -> 1,603, but 36 of 64 713 -> 556.
//   short histories, float32: a prompt of 17 rows, 16 heads of 256 18 -> 26, 36 of 64 9 -> 12, but 24 of 64 over 8 8 -> 7; 4 rows, 64 requests, 36 heads of
//     128 27 -> 78; 16 rows, 256 requests, 16 of 80 172 -> 266.
// Decode steps know their histories to the next power of two from 256 on only: below 40 keys some of them would be faster the other way.
inline bool attention_rows_walk(int T, int nreq, int context, int nh, int nkvh, int size, int elem) {
    if (nreq <= 0 || context <= 0) return false;
    const RowCut c = attention_rows_cut(T, nh, nkvh);
    const long long n = (T + nreq - 1) / nreq, pairs = c.heads * std::min<long long>(c.rows, n), blocks = nreq * ((n + c.rows - 1) / c.rows) * c.parts * nkvh;
    const bool single = pairs == 1 && blocks >= 3 * 148;
    if (context <= 8) return true;
    if (context <= 24 && (size < 32 || (size > 128 && size <= 256) || single || (elem == 2 && size == 32))) return true;
    if (context <= 24 && blocks >= 1500 && size > 64 && size < 128) return true;
    if (context <= 16 && pairs <= 4 && blocks >= 3 * 148 && size <= 96) return true;
    if (elem == 4) {
        if (size < 32) return (pairs == 1 && (blocks >= 5000 || (blocks >= 1500 && context <= 512))) || (pairs <= 4 && blocks >= 3 * 148 && context <= 64);
        return size > 128 && size <= 256 && single && context <= 256;
    }
    if (size % 8 != 0 && size < 32) return context <= 512 || pairs <= 8;            // nor can a block copy 16 bytes at a time
    if (size <= 32) return single || (pairs <= 4 && context <= 256) || (size < 32 && context <= 64);
    if (size <= 128) return pairs == 1 && blocks >= 4096 && context <= 256;
    return single && n <= 8 && context <= 512;
}

// Whether a float32 attention without options runs in tiles of query rows (csrc/attention_f32.cu, the same bits): every request brings more rows than
// go one by one, and there are enough of them.  B200, by rows -> in tiles (us): 24 heads of 64 over 8, 9 rows 6.0 -> 7.4, 24 rows 7.2 -> 7.4, 40 rows 10 -> 8, 10
// requests of 20 rows after 100 46 -> 17; 4 heads over 1, 40 rows 8.2 -> 6.7, 32 rows after 1,000 76 -> 75; pages that are no power of two it
// does not take (with a division a key: 3 heads, 200 rows 20 -> 22, 32 rows after 1,000 76 -> 85).
inline bool attention_f32_takes(int rows, int n_short, int n_tiles, int page_size) {
    return n_short == 0 && n_tiles > 0 && rows >= 32 && page_size > 0 && (page_size & (page_size - 1)) == 0;
}

// Whether its tiles have 64 rows, four a lane, instead of 32: where `blocks` tiles of 64 are enough.  Fewer reads a multiply-add, half the blocks.
// B200, two -> four rows a lane (us): 24 heads of 64 over 600 rows 87 -> 93, over 1,200 255 -> 227; 36 over 600 113 -> 106; 8 heads of 128 over
// 600 72 -> 102, over 1,200 220 -> 191; 32 over 200 47 -> 43.
inline bool attention_f32_tall(long long blocks, int dh) { return blocks >= (dh == 64 ? 350 : 120); }

// ---- routed experts and heads' products of few rows (csrc/blocks.cu) ---------------------------------------------------------------
// Bytes of shared memory of a block of a per-head product of few rows, and whether that form takes `rows` rows with K columns.
constexpr int HEAD_ROWS = 16, HEAD_FEATURES = 32;
inline long long head_rows_bytes(int K) { return (long long)(HEAD_ROWS + HEAD_FEATURES) * (2LL * K + 16) + 64; }
inline bool head_takes_rows(int rows, int K) { return rows <= 64 && K % 16 == 0 && head_rows_bytes(K) <= 100 * 1024; }
// Groups of 16 rows of its matrix that a block of an expert's product of few rows takes, for K columns of `elem` bytes and `blocks` blocks of one
// group: a short row's copy costs a block more than its bytes, so where blocks make several waves (four an SM) a block takes more of
// them.  B200, 48 entries of 64 experts of 64 features over 2,048: 53.4 us with one group, 45.2 with four; but 2 entries of 512 18.5 and 20.6: one there.
inline int expert_row_groups(int K, int elem, long long blocks) {
    int groups = 1;
    while (2 * groups * K * elem <= 2048 && groups < 4 && blocks / (2 * groups) >= 4 * 148) groups *= 2;
    return groups;
}

// Whether a causal convolution over `rows` rows of `nreq` requests walks eight rows a thread (csrc/blocks.cu) instead of making an element
// a thread: a walk is a chain that takes a large launch to hide, the more so where every row is a request of its own and reads and
// moves its own tail.  B200, element a thread -> rows (us): 64 channels, 128 to 2,048 rows 9 -> 13; 512 channels, 512 rows 11 to 13 -> 13,
// 2,048 17 to 20 -> 15; 4,096 channels, 128 rows 13 to 15 -> 13 to 15, 256 17 to 20 -> 15, 2,048 75 to 95 -> 36 to 42; requests of one row: 4,096
// channels, 128 of them 12 to 15 -> 16 to 19, 256 18 to 21 -> 19 to 23, 8,192 channels, 256 of them 27 to 36 -> 21 to 26.
inline bool conv_walks_rows(long long rows, long long nreq, long long channels) {
    return rows >= 128 && rows * channels >= (rows < 2 * nreq ? 1LL << 21 : 1LL << 20);
}

// Whether a selective scan over `rows` rows of `nreq` requests runs over pieces of SELECTIVE_PIECE rows side by side (csrc/blocks.cu) rather
// than from end to end.  The pieces make every row twice, so they pay where the walks leave the chip idle: long requests, and with more than
// 16 states, whose pieces keep too much to hide anything, few channels of them all.  The rule knows the mean length only: a long prompt beside
// many decoding rows walks.  B200, step sizes included, walk -> pieces (us): 16 states, 4,096 channels, one request: 512 rows 148 -> 148,
// 2,048 589 -> 360; 64 channels, 8 requests of 768 104 -> 113, 4 of 1,024 132 -> 113; 512 channels, 2 of 768 127 -> 133, one of 1,000 149 -> 111.  32
// states, 512 channels: one of 768 135 -> 178, 4 of 1,024 279 -> 302, one of 2,048 548 -> 276, 4 of 2,048 647 -> 374; 4,096 channels: 2 of 2,048
// 989 -> 768, 4 of 2,048 1,161 -> 1,357.
constexpr int SELECTIVE_PIECE = 128;
inline bool selective_scan_cuts(long long rows, long long nreq, long long channels, long long states) {
    if (states > 16) return states <= 32 && rows >= 1280 * nreq && nreq * channels <= 8192;
    return rows >= (channels < 1024 ? 896 : 768) * nreq;
}

// Whether the routed experts' products run in tiles of 128 entries on tcgen05 (csrc/experts_tcgen05.cuh) rather than of 64 on mma.sync:
// from two entries an expert on, and for products large enough to pay for the gather and the tensor memory's setup, about 5 us a layer:
// by themselves, by all experts' weights or by the multiply-adds of many entries.  B200, whole layers, tiles of 64 -> of 128 (us):
// 64 x 64 to 512 x 128, up to 32 experts, 64 to 512 rows 26 to 48 -> 31 to 49; 512 x 512, 4 experts, 512 rows 48 -> 49 to 52, 16 experts, 64 rows 48 -> 43,
// 8 experts, 2,048 rows 87 -> 61; 1,024 x 256, 1 to 8 experts 44 to 53 -> 43 to 51; 512 x 128, 64 experts, 64 rows 54 -> 46; 2,048 x 1,408, 8 experts: 48
// rows 102 -> 72, 128 119 -> 77, 512 172 -> 88, 2,048 408 -> 141, 64 experts, 128 rows 367 -> 223.  Below two entries an expert nothing is measured.
inline bool experts_take_tiles(long long entries, long long experts, long long width, long long ff) {
    const long long one = width * ff;
    return entries >= 2 * experts && ((width >= 1024 && one >= 1LL << 18) || experts * one >= 1LL << 22 || (entries >= 2048 && entries * one >= 1LL << 28));
}

// Whether a latent attention over `rows` query rows of `nreq` requests makes the heads' keys and values from the latent rows
// (one product per cached position) instead of running over the latent rows: heads of 64 or 128 for keys and values alike, a
// rotated part of 64 or none, whole vectors; `keys`: positions of all requests, or 0 when one of them brings few rows (a step goes one way
// as a whole).  With `reach` the positions that a row sees of a request's on average, two lines:
//   rows x reach >= 16 keys (without a window: 16 rows a request on average), so that enough rows share the product per position;
//   a latent of 256 or reach x (latent + rotated part) >= 12,288: the way over heads costs 24 us at the least, over short contexts of
//   small latents the other one less.
// B200, over the latent rows -> over heads (us): 16 heads of 128 + 64, latent 512: 4 requests of 17 rows after 500 101 -> 42, one of 48 rows
// after 2,000 288 -> 60, 256 rows after 0 73 -> 30, 2,048 after 0 887 -> 75; 2 of 16 rows after 0 36 -> 28; 2 heads of 64, latent 64: 32 rows after 0
// 17 -> 24, 16 requests of 20 after 100 26 -> 30, 256 rows after 0 34 -> 24, 32 after 500 52 -> 28; 4 heads of 64 + 64, latent 160: 32 rows after 0 22 -> 24,
// 16 requests of 20 after 100 34 -> 30; 16 heads of 64, latent 256: 32 rows after 0 24 -> 24.  8 requests of one row over latents of 512 take 17.
inline bool latent_heads_fit(int dn, int dr, int dv, int R) { return dn == dv && (dn == 64 || dn == 128) && (dr == 0 || dr == 64) && R % 8 == 0 && R >= 64; }
constexpr int LATENT_HEADS_ROWS = 32;       // the fewest rows of a step that goes this way; an engine of smaller steps has neither the room nor the modules
inline bool latent_takes_heads(int rows, int nreq, long long keys, int window, int dn, int dr, int dv, int R) {
    if (keys <= 0 || rows < LATENT_HEADS_ROWS || nreq <= 0 || !latent_heads_fit(dn, dr, dv, R)) return false;
    const long long reach = window > 0 ? std::min<long long>(window, keys / nreq) : keys / nreq;
    return rows * reach >= 16LL * keys && (R >= 256 || reach * (R + dr) >= 12288);
}
// The positions that room is kept for in an engine of steps of up to `rows` rows: four times as many as a step may have rows (prompts, and
// portions of longer ones up to there; steps that see more run over the latent rows), but no more than its requests can have: the
// rule above takes at most rows / 16 of them, of at most `max_positions` each, and without a window all their positions lie in the
// cache's `cached`.
inline long long latent_heads_positions(long long rows, long long max_positions, long long cached, int window) {
    const long long most = std::min(4 * rows, std::max(1LL, rows / 16) * max_positions);
    return window > 0 ? most : std::min(most, cached);
}

// ---- which kernel takes a bfloat16 product ------------------------------------------------------------------------
struct Routing {
    int sms = 148;
    int tcgen05_min_rows = 129, tcgen05_min_tiles = 200, tcgen05_min_fill_pct = 80;     // measured: see takes_tcgen05
    int skinny_min_blocks = 0;        // fewest blocks for the few-rows tcgen05 kernel (0: one per SM)
    int library_only = 0;             // 1: every bfloat16 product goes to the library
};
enum ProductKind { PRODUCT_F32 = 0, PRODUCT_RESIDUAL = 1, PRODUCT_SWIGLU = 2 };
enum Route { ROUTE_LIBRARY = 0, ROUTE_SMALL = 1, ROUTE_SKINNY = 2, ROUTE_TCGEN05 = 3 };

// Whether the tiled tcgen05 product takes `rows` x `n` over `k`.  Measured on the 1B, 2B and 8B shapes, whole steps of
// 160 to 2,048 rows against the library's product with separate elementwise kernels: from `min_rows` rows on, a product
// with at least `min_tiles` output tiles of 128 x 128 whose rows fill their tiles of 128 to `min_fill_pct` per cent is
// as fast or faster on the tcgen05 kernel (fused epilogues, dependent launch, cuts of K for the products that add into
// the residual stream); products of fewer tiles go to the library, whose smaller tiles fill the SMs better.  Very wide
// outputs (the logits) are taken from 17 rows.
inline bool takes_tcgen05(const Routing &r, int rows, int n, int k) {
    if (r.library_only || rows <= 16 || k < 8 || k % 8) return false;
    const long long row_tiles = (rows + 127) / 128;
    if (row_tiles * ((n + 255) / 256) >= 3LL * r.sms) return true;
    if (rows < r.tcgen05_min_rows || rows * 100LL < (long long)r.tcgen05_min_fill_pct * row_tiles * 128) return false;
    return row_tiles * ((n + 127) / 128) >= r.tcgen05_min_tiles;
}
// Blocks that the few-rows tcgen05 kernel starts for a product with `n` output features over `k`: tiles of 128 features
// (64 for SwiGLU, whose tile holds as many up rows again); a product that is added into the residual stream splits K
// until the blocks fill the SMs twice, as long as a block keeps 8 steps of 64.
inline long long skinny_blocks(int sms, int n, int k, int kind) {
    const int nk = (k + 63) / 64;
    if (kind == PRODUCT_SWIGLU) return (n + 63) / 64;
    const int tiles = (n + 127) / 128;
    int splits = 1;
    if (kind == PRODUCT_RESIDUAL) splits = std::max(1, std::min(2 * sms / tiles, nk / 8));
    const int ksteps = (nk + splits - 1) / splits;
    return (long long)tiles * ((nk + ksteps - 1) / ksteps);
}
// Which kernel takes a product of `rows` rows: up to 128 rows the few-rows tcgen05 kernel once it has a block for every
// SM (it then reads W at 5 to 6 TB/s), always once it has four blocks for every SM; up to 16 rows the small-row kernel
// (if it takes the shape: `small_ok`) where it
// has a second block on the SM to overlap its load phase with (a slice of 16 rows x K fits twice), or so few tiles that
// they make one wave, or nothing better; above that the tiled tcgen05 kernel by the rule above; else the library.
// `tcgen05_ok`: the tcgen05 module is there.
inline Route product_route(const Routing &r, int rows, int n, int k, int kind, bool small_ok, bool tcgen05_ok) {
    if (r.library_only) return ROUTE_LIBRARY;
    if (rows <= 128) {
        const long long need = r.skinny_min_blocks > 0 ? r.skinny_min_blocks : r.sms;
        const bool skinny = tcgen05_ok && k >= 8 && k % 8 == 0 && skinny_blocks(r.sms, n, k, kind) >= need;
        // a very wide output (the logits): with four rounds of blocks and more the few-rows tcgen05 kernel reads W at 0.95 of
        // the copy bandwidth for any row count (2B, 1B and 8B output matrices at 1, 8 and 16 rows: 91, 38 and 92 us against
        // 132, 50 and 211 us of the small-row kernel at 8 rows)
        if (skinny && skinny_blocks(r.sms, n, k, kind) >= 4LL * r.sms) return ROUTE_SKINNY;
        if (rows <= 16 && small_ok) {
            const long long out_rows = kind == PRODUCT_SWIGLU ? 2LL * n : n;
            if (!skinny || 2 * (32LL * k + 8192) <= 227 * 1024 || (out_rows + 15) / 16 <= r.sms) return ROUTE_SMALL;
        }
        if (skinny) return ROUTE_SKINNY;
    }
    if (tcgen05_ok && takes_tcgen05(r, rows, n, k)) return ROUTE_TCGEN05;
    return ROUTE_LIBRARY;
}

// ---- which kernel takes a float32 product ---------------------------------------------------------------------------
// On the CUDA cores (csrc/gemm_f32.cu), the tile by what a launch of it takes, from measurements at K 1,536 (us): `first` for a
// block on every SM, `each` for every further one, where blocks of one SM run side by side.  Outputs of few tiles take small ones
// until they fill the SMs (24 x 2,560: 27 us with 16 x 32 against 37 with 32 x 64; 60 x 7,680: 45 with 64 x 64 against 51 with 16 x 32).
struct F32Tile { int rows, cols; double first, each; };
constexpr F32Tile F32_TILES[] = {{8, 64, 14., 14.}, {16, 32, 21., 7.}, {32, 64, 33., 22.}, {64, 64, 42., 42.}};
// the tile's place in that list, or -1 where no launch holds them; `us`: what it takes at K 1,536
inline int f32_tile(long long M, long long N, int sms, double *us) {
    int best = -1;
    for (int i = 0; i < 4; ++i) {
        const F32Tile &t = F32_TILES[i];
        const long long down = (M + t.rows - 1) / t.rows, blocks = down * ((N + t.cols - 1) / t.cols);
        const double cost = std::max(t.first, t.each * (double)((blocks + sms - 1) / sms));
        if (down <= 65535 && (best < 0 || cost < *us)) { best = i; *us = cost; }
    }
    return best;
}
// On the tensor cores (csrc/gemm_f32_tcgen05.cu) with the operands split: tokens a tile and cuts of K, or a tile of 0 where the
// product stays on the CUDA cores.  A wave takes 0.8 us, 2.8 more with cuts, 0.036 a token of the tile, and a chunk of 64 columns of K its
// tile's time; fitted to 1,700 launches of 18 shapes with 16 to 2,048 rows, nine of ten within 8 %, and what the fit chooses is within
// 12 % of the fastest form everywhere.  A block fills an SM, and clusters of four or eight leave some SMs of a chip of 148 without a block:
// 33 and 14 of them run at once (three tiles of 96 x 12 of 128, four cuts, 36 clusters: 29 us where 24 clusters take 20).
// From K 512: below, a launch costs what it saves.  CUDA cores -> tensor cores (us): 301 rows, 7,680 x 1,536 199 -> 45, 2,560 x 1,536 73 -> 27,
// 1,536 x 1,536 46 -> 20, 1,536 x 3,840 108 -> 33; 48 rows, 2,560 x 1,536 23 -> 14; 2,048 rows, 4,608 x 4,096 1,768 -> 402.
//
// The cuts set the order of the sums (the tile does not).  Below F32_ONE_ORDER_ROWS rows, where the norms of a step add in one order too,
// way and cuts follow from N and K alone, so that a row's result depends neither on what else is in the step nor on how its prompt
// was cut.  One choice for all of them: the cuts that are cheapest for three steps of 32 rows (decoding, short prompts) and one of 255.
// What it costs and gives, whole steps of the 1B shape against cuts by the rows and CUDA cores below 24 rows (us): prompts of 24 rows 4,454 -> 4,508, 64
// 4,863 -> 4,955, 160 6,820 -> 6,868, 200 8,453 -> 10,494, 255 8,617 -> 10,736; one decoding row 8,724 -> 4,524, 24 4,932 -> 4,962.  (With eight cuts of
// 1,536 x 1,536; with four 64 rows took 5,245 and 200 10,063.)  Wide products of few rows lose: 8 rows, 11,520 x 2,304 37 -> 48, 73,440 x 1,536 89 -> 137.
struct F32Plan { int tile, cuts; };
constexpr int F32_ONE_ORDER_ROWS = 256, F32_TENSOR_K = 512;
// microseconds of the best tile for the given cuts, and that tile; `waves`: how often it fills the chip
inline double f32_tensor_cost(long long M, long long N, long long K, int sms, int cuts, int *tile, long long *waves) {
    constexpr int TILES[5] = {32, 64, 96, 128, 160};
    constexpr double CHUNK[5] = {1.25, 1.30, 1.30, 1.42, 1.57};
    const int at_once = std::max(1, cuts == 8 ? sms * 14 / 148 : cuts == 4 ? sms * 33 / 148 : sms / cuts);
    double least = -1.;
    for (int i = 0; i < 5; ++i) {
        const long long tiles = (M + TILES[i] - 1) / TILES[i] * ((N + 127) / 128), w = (tiles + at_once - 1) / at_once;
        if (tiles * cuts > (1LL << 30)) continue;
        const double cost = (double)w * (0.8 + (cuts > 1 ? 2.8 : 0.) + 0.036 * TILES[i] + CHUNK[i] * (double)(((K + 63) / 64 + cuts - 1) / cuts));
        if (least < 0. || cost < least) { least = cost; *tile = TILES[i]; *waves = w; }
    }
    return least;
}
inline F32Plan f32_plan(long long M, long long N, long long K, int sms) {
    F32Plan best = {0, 1};
    if (M < 1 || K < F32_TENSOR_K || sms <= 0) return best;
    const long long chunks = (K + 63) / 64;
    const bool one_order = M < F32_ONE_ORDER_ROWS;
    double least = -1.;
    if (!one_order && f32_tile(M, N, sms, &least) >= 0) least = least * (double)K / 1536. + 2.;
    for (int cuts = 1; cuts <= 8; cuts *= 2) {
        if (cuts > 1 && chunks < 2 * cuts) continue;
        int tile = 0;
        long long waves = 0;
        double cost;
        if (one_order) {
            const double few = f32_tensor_cost(32, N, K, sms, cuts, &tile, &waves), many = f32_tensor_cost(F32_ONE_ORDER_ROWS - 1, N, K, sms, cuts, &tile, &waves);
            if (few < 0. || many < 0.) continue;
            cost = 3. * few + many;
        } else {
            cost = f32_tensor_cost(M, N, K, sms, cuts, &tile, &waves);
            if (cost < 0. || (cuts > 1 && waves > 1)) continue;
        }
        if (least < 0. || cost < least) { least = cost; best = {tile, cuts}; }
    }
    long long waves = 0;
    if (one_order && best.tile > 0) f32_tensor_cost(M, N, K, sms, best.cuts, &best.tile, &waves);
    return best;
}

// ---- rotary tables --------------------------------------------------------------------------------------------
// Angle of pair j at position p: p / theta^(j / half), computed in double and rounded once to float32.
inline void rotary_tables(double theta, int half, int positions, double angle_scale, float *cos_out, float *sin_out) {
    std::vector<double> inv((size_t)half);
    for (int j = 0; j < half; ++j) inv[(size_t)j] = angle_scale * std::pow(theta, -((double)j / half));
    for (int p = 0; p < positions; ++p)
        for (int j = 0; j < half; ++j) {
            const double a = (double)p * inv[(size_t)j];
            cos_out[(size_t)p * half + j] = (float)std::cos(a);
            sin_out[(size_t)p * half + j] = (float)std::sin(a);
        }
}

// ---- the uniform number of a drawn token ---------------------------------------------------------------------------
// A float in [0, 1) from (seed, absolute position of the new token): the splitmix64 finaliser, top 24 bits.  It does
// not depend on what else is in the batch or on how the prompt was cut.
inline float uniform_for(uint64_t seed, uint64_t index) {
    uint64_t z = seed * 0x9E3779B97F4A7C15ull + (index + 1) * 0xBF58476D1CE4E5B9ull;
    z ^= z >> 30;
    z *= 0xBF58476D1CE4E5B9ull;
    z ^= z >> 27;
    z *= 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (float)(z >> 40) / (float)(1 << 24);
}

}  // namespace jk
