// A mine (or the tail of one) whose levels are small, in one launch: every level's candidates counted on the full
// columns, the survivors compacted into the next level, level after level, by one cooperative kernel.
//
// What bounds such a mine is not its counting but the launches, copies and waits between its steps: a level of the
// general path takes some twenty launches and six host reads, about 0.9 ms, whatever its size. Here a level is three
// phases with a grid barrier after each (about 2 us):
//
//   count    tiles of 8 x 8 members of a prefix group by a warp each, every column read once (etm_tile.cuh); where the
//            tiles are too few for the SMs their words are cut into slabs that add their counts. Counts are laid out
//            by candidate: row r's pairs with the later rows of its group, row after row, which is the
//            lexicographic order of the next level.
//   select   each CTA marks and counts the survivors of its run of candidates.
//   compact  new rows are written in candidate order with their parent row, which is their prefix group: the next
//            level's groups need no search and no scan of the rows.
//
// Up to SMEM_ROWS rows every CTA computes the candidate and tile offsets of a level itself (ordered scans over the rows,
// in shared memory), which costs less than a further barrier; past it each CTA scans its part. The kernel stops, and says
// so, before a level past its limits (rows, candidates, candidate words) and the caller goes on from the last complete
// level.
//
// Past K=2 the columns are cut to the rows of the first item (project_columns), where the levels ahead read them often
// enough: the reads of full columns bound those levels (7 TB/s from L2), and a column cut so is as long as the first
// item is frequent, 3% of the rows on average when the generators are in ascending support. It is done only from a given
// level 2, which the caller has in that order; over columns in the caller's order the share was 8 to 32%, and cutting
// cost more than it gave (1M rows, 164,130 itemsets: 4.4 ms on the device against 1.6).
//
// Measured per mine, general path against this kernel: 10,000 rows (108 frequent items, 5 levels) 3.1 -> 0.28 ms, of
// which 0.08 ms on the device; 33,333 rows under the free-set prune 7.6 -> 0.7 ms; 1M rows (267 frequent items, 6
// levels, 7.8e8 candidate words) 4.7 -> 0.95 ms, 0.59 on the device. With the projection, and levels of a million rows, against 16,384 rows
// at most on full columns: 1M rows, 164,130 itemsets of up to 11 items 17 -> 7.8 ms; 400K rows, 1.1M itemsets 11 -> 6.8;
// 20M rows, 1,600 prefixes 8.4 -> 6.8 ms. The caller's limit of 2^30 candidate words a level (about 0.6 ms) lies where
// the general path's launches and its tensor-core Gram take as long.
//
// The grid barriers hold only while every CTA is resident, hence the cooperative launch; their waits are bounded in
// time (%globaltimer), after which every CTA leaves and the header keeps the value the caller set it to.
#include "etm_tile.cuh"

namespace {

using namespace etm;

constexpr int DT = 512;                   // threads per CTA: 128 registers each, for the tiles
constexpr int DWARPS = DT / 32;
constexpr int SMEM_ROWS = 16384;  // rows whose offsets a CTA holds in shared memory
constexpr int FEW_CANDS = 8192;    // candidates whose counts every CTA reads to place its survivors
constexpr int ROW_CANDS = 65535;  // candidates a row counts as at most: a group past that is past every limit
constexpr int SLAB_MIN = 256;     // words of a slab at least
constexpr int SLAB_MAX = 2048;    // and at most
constexpr int MAXW = ETM_DIRECT_LEVELS;
constexpr int MAX_GRID = 256;
constexpr uint64_t BARRIER_NS = 2000000000ull;

// Projection by first item.
constexpr int PROJ_ITEMS = 2048;            // items of level 1 at most
constexpr int PROJ_MEMBERS = 16;            // members a warp projects for one row list
constexpr int PROJ_LIST = 1088;             // rows of a warp's list
constexpr int PROJ_SEG = 256;               // words of a segment
constexpr int PROJ_WORDS = 24;              // 32-bit words of a member gathered at a time
constexpr int PROJ_BUFS = 3;                // segments a warp copies there in turn
constexpr int64_t PROJ_UNITS = 1ll << 30;   // (run of members, segment) units at most
constexpr int64_t PROJ_WORK = 1ll << 26;    // candidate words of the level from which it pays
constexpr int PROJ_NOT = 0, PROJ_DONE = 1, PROJ_LOST = 2;  // outcomes: would not fit or pay; done; a wait gave up
constexpr int PROJ_SHARE = 8;               // projected words at most a PROJ_SHARE-th of the full columns'

constexpr int SMEM_OFFSETS = 2 * (SMEM_ROWS + 1) * 4;
constexpr int SMEM_BUFS = DWARPS * PROJ_BUFS * PROJ_SEG * 8;
constexpr int SMEM_PROJ = SMEM_BUFS + PROJ_ITEMS * 8 + (PROJ_ITEMS + 4) * 4 + DWARPS * PROJ_LIST * 2;
constexpr int SMEM_WORK = (SMEM_OFFSETS > SMEM_PROJ ? SMEM_OFFSETS : SMEM_PROJ) + 15 & ~15;
constexpr int SMEM_COLS = DWARPS * (2 * GB + MAXW) * 8;                // then each warp's column offsets,
constexpr int STATE_BYTES = 384;
constexpr int MAP_ITEMS = 1024;           // items whose columns are looked up in shared memory
constexpr int SMEM_BYTES = SMEM_WORK + SMEM_COLS + 2 * STATE_BYTES + MAP_ITEMS * 4;  // the state, the arguments, the map

// Scratch layout, in 32-bit words.
struct Scratch {
    int64_t bar, partial, par, pstart, mask, cnt, coff, toff, words;
};
// The projection's part, apart: a launch may go on from what one before it left there.
struct ProjScratch {
    int64_t gfirst, gsize, cw, table, seg, proj, words;
};

struct Take {
    int64_t at = 0;
    int64_t operator()(int64_t n) {
        const int64_t here = at;
        at += (n + 63) / 64 * 64;
        return here;
    }
};

Scratch scratch_layout(int64_t cap_rows, int64_t cap_cands) {
    Scratch s;
    Take take;
    s.bar = take(64);                    // barrier counter, abort flag, claimed units
    s.partial = take(7 * MAX_GRID);      // sums of each CTA: survivors or groups; three of 64 bits
    s.par = take(cap_rows);              // parent row of each row of the level being written / read
    s.pstart = take(cap_rows + 1);       // first new row of each parent
    s.mask = take(cap_cands / 32 + 1);   // survivor bits, by candidate
    s.cnt = take(cap_cands);             // counts, by candidate
    s.coff = take(cap_rows + 1);         // offsets of a level past SMEM_ROWS
    s.toff = take(cap_rows + 1);
    s.words = take.at;
    return s;
}

ProjScratch proj_layout(int64_t n_cols, int64_t n_words, int64_t proj_words) {
    ProjScratch s;
    Take take;
    const int64_t items = proj_words > 0 ? min64(PROJ_ITEMS, n_cols) : 0;
    s.gfirst = take(items);  // by item: the first row of its K=3 group, the group's rows (0: none),
    s.gsize = take(items);
    s.cw = take(items);      // and the words of a projected column
    s.table = take(items * items);  // [first item][item]: the projected column, in 2 words
    s.seg = take(items * ((n_words + PROJ_SEG - 1) / PROJ_SEG));
    s.proj = take(2 * proj_words);
    s.words = take.at;
    return s;
}

struct DirectArgs {
    const uint64_t* bv;  // columns [.][ld]
    int64_t ld;
    int64_t n_words, n_cols;
    const int64_t* col_counts;  // K=1 start: counts of the n_cols columns (nullptr: start from `rows`)
    int64_t n_rows;
    int min_count, prune, max_k;
    int64_t work_limit, deep_limit;  // candidate words of a level at most; of one past K=2 whose columns are not projected
    const int32_t* rows;        // start level [n][width] over the columns of bv
    const int32_t* counts;
    int n, width;
    int64_t* header;
    int32_t* out_counts;
    int64_t counts_cap;
    int32_t* out_rows;
    int64_t rows_cap;
    int32_t* scratch;
    Scratch at;
    int32_t* pscratch;
    ProjScratch pat;
    int cap_rows, cap_cands;
    int64_t proj_words;         // 0: no projection
    int projected;              // the columns are there, from an earlier launch of the mine
};

extern __shared__ __align__(16) int32_t offsets[];

// This warp's tile: word offsets of block a's members, block b's, and the prefix columns.
__device__ __forceinline__ int64_t* tile_cols() {
    return reinterpret_cast<int64_t*>(offsets + SMEM_WORK / 4) + (threadIdx.x >> 5) * (2 * GB + MAXW);
}

// The state of a CTA between the phases. It lies in shared memory and every phase is a function of its own, so that
// little is spilled: an acquire at a grid barrier empties L1, and the first reload of each spilled register after it
// goes to L2. With the state in registers and one function a mine of 10,000 rows took 93 us on the device, so 79.
struct State {
    const int32_t* rows;    // nullptr: row r of level 1 is item r
    const int32_t* counts;
    const int32_t* map;     // column of an item (nullptr: the item)
    int64_t rows_used, counts_used;
    int64_t T, tiles;       // the next level's candidates and tiles,
    unsigned long long work;  // the words of its candidates' projected columns,
    int groups;             // and its prefix groups
    int n, w;               // rows and items of a row
    int n_items;            // of level 1
    int n_slab;
    int c_lo, c_hi;         // this CTA's run of candidates, in whole mask words
    int survivors, base, fresh;  // of this CTA, of those before it, of all
    int ok;
    unsigned bar_target;
    int64_t tot[2];
    bool searched;          // the level's group ends are in pstart by row (a given start level), not by parent
    bool projected;         // columns are those of (first item, item), over the rows that hold the first item
    bool shared;            // the offsets are in shared memory
};
static_assert(sizeof(State) <= STATE_BYTES && sizeof(DirectArgs) <= STATE_BYTES, "SMEM_BYTES");
__device__ __forceinline__ DirectArgs& args_sh() {  // as parameters of the phases they would go through L1 as well
    return *reinterpret_cast<DirectArgs*>(offsets + (SMEM_WORK + SMEM_COLS + STATE_BYTES) / 4);
}
__device__ __forceinline__ int32_t* map_sh() { return offsets + (SMEM_WORK + SMEM_COLS + 2 * STATE_BYTES) / 4; }
__device__ __forceinline__ State& state_sh() { return *reinterpret_cast<State*>(offsets + (SMEM_WORK + SMEM_COLS) / 4); }

__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ uint64_t time_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Every CTA arrives and waits for the others; false once a wait ran out anywhere.
__device__ __forceinline__ bool grid_barrier(int32_t* scratch) {
    State& S = state_sh();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned* bar = reinterpret_cast<unsigned*>(scratch);
        unsigned* abort_flag = bar + 1;
        const unsigned target = S.bar_target += gridDim.x;
        __threadfence();
        atomicAdd(bar, 1u);
        const uint64_t t0 = time_ns();
        while (load_acquire(bar) < target) {
            if (load_acquire(abort_flag) != 0u) break;
            if (time_ns() - t0 > BARRIER_NS) {
                atomicExch(abort_flag, 1u);
                break;
            }
        }
        S.ok = load_acquire(abort_flag) == 0u;
        __threadfence();
    }
    __syncthreads();
    return S.ok != 0;
}

// Sum over the CTAs of v[0, gridDim.x), and of those before this one; for all threads.
__device__ __forceinline__ int64_t sum_over_ctas(const int64_t* v, int64_t* before) {
    int64_t* tot_sh = state_sh().tot;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        int64_t all = 0, mine = 0;
        for (int c = lane; c < gridDim.x; c += 32) {
            const int64_t x = __ldcg(reinterpret_cast<const long long*>(v) + c);
            all += x;
            if (c < blockIdx.x) mine += x;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            all += __shfl_xor_sync(0xffffffffu, all, d);
            mine += __shfl_xor_sync(0xffffffffu, mine, d);
        }
        if (lane == 0) tot_sh[0] = all, tot_sh[1] = mine;
    }
    __syncthreads();
    const int64_t all = tot_sh[0];
    if (before != nullptr) *before = tot_sh[1];
    __syncthreads();
    return all;
}

// Exclusive scan of one int per thread of the CTA; *total: the sum.
__device__ __forceinline__ int scan_ints(int v, int* total, int* warp_sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += y;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int s = lane < DWARPS ? warp_sums[lane] : 0;
        int si = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, si, d);
            if (lane >= d) si += y;
        }
        if (lane < DWARPS) warp_sums[lane] = si - s;
        if (lane == DWARPS - 1) warp_sums[DWARPS] = si;
    }
    __syncthreads();
    const int out = warp_sums[warp] + inc - v;
    *total = warp_sums[DWARPS];
    __syncthreads();
    return out;
}

// Exclusive scan of two counts per thread of the CTA, packed (high: candidates, low: tiles), in thread order.
__device__ __forceinline__ int64_t scan_pairs(int64_t v, int64_t* total, int64_t* warp_sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += y;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    int64_t before = 0, all = 0;
#pragma unroll
    for (int i = 0; i < DWARPS; i++) {
        const int64_t x = warp_sums[i];
        if (i < warp) before += x;
        all += x;
    }
    *total = all;
    __syncthreads();
    return before + inc - v;
}

// Rows written by other CTAs of this launch are read through L2 (__ldcg): a line of L1 may be older.
__device__ __forceinline__ int item_at(const int32_t* rows, int w, int r, int q) { return __ldcg(rows + (int64_t)r * w + q); }

// Row of the n rows of w items (read by at(row, item)) holding row r's items without item d (d < w) plus `last` at the end, or -1.
template <class F>
__device__ __forceinline__ int find_without(F at, int n, int w, int r, int d, int last) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        int cmp = 0;
        for (int t = 0; t < w && cmp == 0; t++) {
            const int v = t == w - 1 ? last : at(r, t < d ? t : t + 1);
            const int x = at(mid, t);
            cmp = x < v ? -1 : (x > v ? 1 : 0);
        }
        if (cmp == 0) return mid;
        if (cmp < 0) lo = mid + 1;
        else hi = mid;
    }
    return -1;
}

// First index in [0, n] of the non-decreasing off[0..n] with off[i] >= x (n + 1 if none).
__device__ __forceinline__ int lower_bound(const int32_t* off, int n, int x) {
    int lo = 0, hi = n + 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The row r with off[r] <= x < off[r + 1], off[0] = 0, x < off[n].
__device__ __forceinline__ int row_of(const int32_t* off, int n, int x) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

// First candidates (coff) and first tiles (toff) of the rows, n + 1 of each; a group's tiles belong to its first row.
template <class F>
__device__ __forceinline__ auto with_offsets(const DirectArgs& a, bool shared, F f) {
    if (shared) return f(offsets, offsets + SMEM_ROWS + 1);
    return f(a.scratch + a.at.coff, a.scratch + a.at.toff);
}

// End of row r's group.
__device__ __forceinline__ int group_end(const DirectArgs& a, const State& S, int r) {
    if (S.w == 1) return S.n;
    const int32_t* pstart = a.scratch + a.at.pstart;
    return S.searched ? __ldcg(pstart + r) : __ldcg(pstart + __ldcg(a.scratch + a.at.par + r) + 1);
}

__device__ __forceinline__ int row_item(const State& S, int r, int q) {
    return S.rows == nullptr ? r : item_at(S.rows, S.w, r, q);
}

// Word offset of an item's column.
__device__ __forceinline__ int64_t item_column(const DirectArgs& a, const State& S, int it) {
    const int col = S.map == nullptr ? it : S.n_items <= MAP_ITEMS ? map_sh()[it] : __ldcg(S.map + it);
    return (int64_t)col * a.ld;
}

// Counts the tile at tile_cols(); RO: of columns this launch does not write (read-only loads: 88 against 98 us).
template <class V, bool RO>
__device__ __forceinline__ uint2 tile_counts(const uint64_t* bv, int64_t v0, int64_t v1, int plen, bool tri, int ta, int tb) {
    unsigned res[2] = {0u, 0u};
    const int64_t* off = tile_cols();
    const GroupTile t{bv, v0, v1, off + 2 * GB, off, off + GB, plen};
    count_shape<V, RO>(t, threadIdx.x & 31, tri, ta, tb, res);
    return make_uint2(res[0], res[1]);
}

// Counts the level at level_sh(). PROJ: on the columns of (first item, item).
template <class V, bool PROJ>
__device__ __noinline__ void count_units() {
    const DirectArgs& a = args_sh();
    constexpr int VW = sizeof(V) / 8;  // words per vector
    constexpr int LEAD = PROJ ? 1 : 0;  // prefix items whose rows the columns are already cut to
    const State& S = state_sh();
    const int n_slab = S.n_slab, w = S.w;
    const int64_t tiles = S.tiles, units = tiles * n_slab;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.x, G = gridDim.x;
    int64_t* off = tile_cols();
    int32_t* cnt = a.scratch + a.at.cnt;
    // Neighbouring tiles share most columns: a CTA's warps take them side by side, for its L1, from eight units a warp on
    // (400K rows, 6.2M candidates: 1.11 -> 1.06 ms). Below that the last round would fill some CTAs and leave the others
    // empty (33,561 rows, 2,970 units over 2,432 warps: 66 us, spread out 57; a K=2 level of 1M rows 552, 503).
    const bool side_by_side = units >= 8 * (int64_t)G * DWARPS;
    for (int64_t u = side_by_side ? (int64_t)b * DWARPS + warp : (int64_t)b + (int64_t)warp * G; u < units;
         u += (int64_t)G * DWARPS) {
        const int slab = n_slab == 1 ? 0 : (int)(u / tiles), tile = (int)(u - slab * tiles);
        int rest;
        const int first = with_offsets(a, S.shared, [&](const int32_t*, const int32_t* toff) {
            const int r = row_of(toff, S.n, tile);
            rest = tile - toff[r];
            return r;
        });
        const int m = group_end(a, S, first) - first;
        const int nb = (m + GB - 1) / GB;
        int ba = 0;
        while (rest >= nb - ba) rest -= nb - ba++;
        const int a0 = first + ba * GB, b0 = first + (ba + rest) * GB;
        const int na = min(GB, first + m - a0), nbm = min(GB, first + m - b0);
        const int head = PROJ ? row_item(S, first, 0) : 0;
        const int32_t* cols = a.pscratch + a.pat.table + (int64_t)head * S.n_items;
        auto word_of = [&](int it) -> int64_t {
            return PROJ ? 2 * (int64_t)__ldcg(cols + it) : item_column(a, S, it);
        };
        __syncwarp();  // the previous tile is done with the offsets
        if (lane < GB) off[lane] = word_of(row_item(S, a0 + min(lane, na - 1), w - 1));
        else if (lane < 2 * GB) off[lane] = word_of(row_item(S, b0 + min(lane - GB, nbm - 1), w - 1));
        for (int q = lane; q < w - 1 - LEAD; q += 32) off[2 * GB + q] = word_of(row_item(S, first, q + LEAD));
        __syncwarp();
        const int64_t vecs = PROJ ? __ldcg(a.pscratch + a.pat.cw + head) / VW : (a.n_words + VW - 1) / VW;
        const int64_t per = n_slab == 1 ? vecs : (vecs + n_slab - 1) / n_slab;
        const int64_t v0 = min64(vecs, slab * per), v1 = min64(vecs, v0 + per);
        int ta, tb;
        tile_shape(rest == 0, na, nbm, &ta, &tb);
        const uint64_t* bv = PROJ ? reinterpret_cast<const uint64_t*>(a.pscratch + a.pat.proj) : a.bv;
        const uint2 counted = tile_counts<V, !PROJ>(bv, v0, v1, w - 1 - LEAD, rest == 0, ta, tb);
        const unsigned res[2] = {counted.x, counted.y};
        with_offsets(a, S.shared, [&](const int32_t* coff, const int32_t*) {
            emit_tile(lane, rest == 0, ta, tb, na, nbm, res, [&](int i, int j, int32_t c) {
                const int at = coff[a0 + i] + (b0 + j) - (a0 + i) - 1;
                if (n_slab == 1) cnt[at] = c;
                else if (c != 0) atomicAdd(cnt + at, c);
            });
        });
    }
}

// Projection by first item, before K=3: the columns of (first item, item) for the rows {first item, item} of level 2
// whose first item has more than one, holding only the rows of the first item. Every deeper candidate's items share its
// first item, so from here on a column is as long as that item's rows. A column is its segments one after another, each
// filled up to 16 bytes. What bounds it is the instructions of the gather, per member and 32 rows of the first item a
// load, a test, a ballot and a select (20M rows, 1,724 columns of 0.7M rows: 1.57 ms, of which 0.6 ms would be the bytes;
// gathers straight from memory 2.2 ms, with the row numbers read from the list for every member 1.9).
template <class V>
__device__ __noinline__ int project_columns() {
    const DirectArgs& a = args_sh();
    State& S = state_sh();
    const int n = S.n, n_items = S.n_items;
    const int32_t* rows = S.rows;
    __shared__ int64_t pair_sums[DWARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, G = gridDim.x;
    int32_t* gfirst = a.pscratch + a.pat.gfirst;
    int32_t* gsize = a.pscratch + a.pat.gsize;
    int32_t* cw = a.pscratch + a.pat.cw;
    int32_t* table = a.pscratch + a.pat.table;
    uint64_t* proj = reinterpret_cast<uint64_t*>(a.pscratch + a.pat.proj);
    auto item = [&](int r, int q) -> int { return item_at(rows, 2, r, q); };
    auto column = [&](int it) -> int64_t { return item_column(a, S, it); };
    int projected = PROJ_NOT;
    // Each first item's group.
    for (int r = b * DT + tid; r < n; r += G * DT) {
        const int end = group_end(a, S, r), first = item(r, 0);
        if (end - r > 1 && (r == 0 || item(r - 1, 0) != first)) {
            gfirst[first] = r;
            gsize[first] = end - r;
        }
    }
    if (!grid_barrier(a.scratch)) return PROJ_LOST;
    constexpr int SEG = PROJ_SEG, LANE_WORDS = 2 * SEG / 32;  // 32-bit words of a segment by lane
    const int n_seg = (int)((a.n_words + SEG - 1) / SEG);
    int32_t* seg = a.pscratch + a.pat.seg;
    // Words of each first item's rows in each segment, whole 16 bytes.
    for (int64_t u = (int64_t)warp * G + b; u < (int64_t)n_items * n_seg; u += (int64_t)G * DWARPS) {
        const int first = (int)(u / n_seg), sg = (int)(u - (int64_t)first * n_seg);
        if (__ldcg(gsize + first) == 0) continue;
        const uint64_t* x = a.bv + column(first);
        const int64_t w1 = min64(a.n_words, (int64_t)(sg + 1) * SEG);
        int set = 0;
#pragma unroll 8
        for (int64_t v = (int64_t)sg * SEG + lane; v < w1; v += 32) set += __popcll(__ldg(x + v));
        set = __reduce_add_sync(0xffffffffu, set);
        if (lane == 0) seg[u] = (set + 127) / 128 * 2;
    }
    if (!grid_barrier(a.scratch)) return PROJ_LOST;
    for (int first = warp * G + b; first < n_items; first += G * DWARPS) {
        if (__ldcg(gsize + first) == 0) continue;
        int run = 0;
        for (int s0 = 0; s0 < n_seg; s0 += 32) {
            const int v = s0 + lane < n_seg ? __ldcg(seg + (int64_t)first * n_seg + s0 + lane) : 0;
            int inc = v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += y;
            }
            if (s0 + lane < n_seg) seg[(int64_t)first * n_seg + s0 + lane] = run + inc - v;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) cw[first] = run;
    }
    if (!grid_barrier(a.scratch)) return PROJ_LOST;
    // Every CTA: where each first item's columns start, and its runs of PROJ_MEMBERS members.
    int64_t* base = reinterpret_cast<int64_t*>(offsets + SMEM_BUFS / 4);
    int32_t* runs = reinterpret_cast<int32_t*>(base + PROJ_ITEMS);  // n_items + 1
    int64_t words = 0, n_run = 0;
    for (int i0 = 0; i0 < n_items; i0 += DT) {
        const int i = i0 + tid;
        const int m = i < n_items ? __ldcg(gsize + i) : 0;
        const int64_t mine = m == 0 ? 0 : (int64_t)m * __ldcg(cw + i);
        int64_t total;
        const int64_t at = words + scan_pairs(mine, &total, pair_sums);
        words += total;
        const int64_t rat = n_run + scan_pairs((m + PROJ_MEMBERS - 1) / PROJ_MEMBERS, &total, pair_sums);
        n_run += total;
        if (i < n_items) {
            base[i] = at;
            runs[i] = (int)rat;
        }
    }
    if (tid == 0) runs[n_items] = (int)n_run;
    __syncthreads();
    if (words <= a.proj_words && n_run * n_seg <= PROJ_UNITS && words * PROJ_SHARE <= (int64_t)n * a.n_words) {
        for (int r = b * DT + tid; r < n; r += G * DT) {
            const int first = item(r, 0);
            if (__ldcg(gsize + first) != 0)
                table[(int64_t)first * n_items + item(r, 1)] =
                    (int)((base[first] + (int64_t)(r - __ldcg(gfirst + first)) * __ldcg(cw + first)) >> 1);
        }
        uint16_t* list = reinterpret_cast<uint16_t*>(runs + PROJ_ITEMS + 4) + warp * PROJ_LIST;
        V* bufs = reinterpret_cast<V*>(offsets) + warp * PROJ_BUFS * (PROJ_SEG * 8 / sizeof(V));
        // Units cost as their first items' rows, so warps claim them in turn.
        const int64_t units = n_run * n_seg;
        int* claimed = a.scratch + 2;
        int next = 0;
        for (int64_t u = (int64_t)warp * G + b; u < units; u = (int64_t)G * DWARPS + __shfl_sync(0xffffffffu, next, 0)) {
            if (lane == 0) next = atomicAdd(claimed, 1);
            const int sg = (int)(u / n_run), run = (int)(u - (int64_t)sg * n_run);
            const int first = row_of(runs, n_items, run);
            const int c = __ldcg(cw + first), i0 = (run - runs[first]) * PROJ_MEMBERS;
            const int ni = min(PROJ_MEMBERS, __ldcg(gsize + first) - i0);
            const int row0 = __ldcg(gfirst + first) + i0;
            const int64_t w0 = (int64_t)sg * SEG;
            const int len = 2 * (int)min64(SEG, a.n_words - w0);  // 32-bit words
            const uint32_t* x = reinterpret_cast<const uint32_t*>(a.bv + column(first) + w0);
            const int64_t own = column(item(row0 + min(lane, ni - 1), 1)) + w0;  // lane i: member i's column
            const int from = __ldcg(seg + (int64_t)first * n_seg + sg);
            const int out_n = 2 * ((sg + 1 < n_seg ? __ldcg(seg + (int64_t)first * n_seg + sg + 1) : c) - from);
            // A segment without a row of the first item adds no words. It must not reach the copies: only a gather waits
            // for them, and two copies to one buffer that are not waited for between come in any order. Of a unit that
            // has rows the last flush writes at least one word of every member, and its last wait is for all of them.
            if (out_n == 0) continue;
            uint32_t* out = reinterpret_cast<uint32_t*>(proj + base[first] + (int64_t)i0 * c + from);
            // Members' segments are copied to shared memory two ahead of the gathers from them: a gather from memory waits
            // long, and a warp has few in flight. That pays even where a few of a segment's words are wanted (192 columns
            // of 20M rows, a launch: one row a segment 0.58 against 0.65 ms straight from memory, 64 rows 0.81 against
            // 0.88, 1,024 rows 2.16 against 2.66).
            constexpr int PER = PROJ_SEG * 8 / sizeof(V);
            auto copy = [&](int i) {
                const V* y = reinterpret_cast<const V*>(a.bv + __shfl_sync(0xffffffffu, own, i & 31));
                const unsigned to = (unsigned)__cvta_generic_to_shared(bufs + i % PROJ_BUFS * PER);
                if (i < ni) {
#pragma unroll
                    for (int q = lane; q < PER; q += 32)
                        if (q < len * 4 / (int)sizeof(V))
                            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to + q * (unsigned)sizeof(V)),
                                         "l"(y + q), "n"(sizeof(V)) : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            int held = 0, done = 0;  // rows in the list; 32-bit words written
            __syncwarp();  // the previous unit is done with the buffers
            copy(0);
            copy(1);
            // Writes n_out words of every member from the list's rows (held of them; zero past those). A lane keeps its
            // rows of PROJ_WORDS words, as a word and a bit of it, over all members: a word of 32 rows is then a
            // load, a test, a ballot and a select by each lane, which is what bounds this loop.
            auto flush = [&](int n_out) {
                __syncwarp();
                for (int q0 = 0; q0 < n_out; q0 += PROJ_WORDS) {
                    uint32_t at[PROJ_WORDS], bit[PROJ_WORDS];
#pragma unroll
                    for (int q = 0; q < PROJ_WORDS; q++) {
                        const int j = (q0 + q) * 32 + lane;
                        const uint32_t row = j < held ? list[j] : 0u;
                        at[q] = row >> 5;
                        bit[q] = j < held ? 1u << (row & 31) : 0u;
                    }
                    if (done + q0 != 0) {
                        copy(0);
                        copy(1);
                    }
                    const int nq = min(PROJ_WORDS, n_out - q0);
                    auto gather = [&](const uint32_t* y, uint32_t* o) {
#pragma unroll
                        for (int b0 = 0; b0 < PROJ_WORDS; b0 += 8) {
                            if (b0 >= nq) break;
                            uint32_t w8[8];
#pragma unroll
                            for (int q = 0; q < 8; q++) w8[q] = y[at[b0 + q]];
#pragma unroll
                            for (int q = 0; q < 8; q++) w8[q] = __ballot_sync(0xffffffffu, (w8[q] & bit[b0 + q]) != 0u);
#pragma unroll
                            for (int d = 1; d < 8; d *= 2)
#pragma unroll
                                for (int q = 0; q < 8; q += 2 * d) w8[q] = (lane & d) != 0 ? w8[q + d] : w8[q];
                            if (lane < 8 && b0 + lane < nq) o[b0 + lane] = w8[0];
                        }
                    };
                    for (int i = 0; i < ni; i++) {
                        __syncwarp();
                        copy(i + 2);
                        asm volatile("cp.async.wait_group 2;" ::: "memory");
                        __syncwarp();
                        gather(reinterpret_cast<const uint32_t*>(bufs + i % PROJ_BUFS * PER),
                               out + (int64_t)i * 2 * c + done + q0);
                    }
                    __syncwarp();
                }
                done += n_out;
            };
            // Each lane takes 16 words in a row (one where so many rows could pass the list), so that a piece needs one
            // scan of their sums.
            const int per_lane = 32 * out_n <= PROJ_LIST ? LANE_WORDS : 1;
            for (int p0 = 0; p0 < len; p0 += 32 * per_lane) {
                const int v0 = p0 + lane * per_lane;
                uint32_t word[LANE_WORDS];
                int set = 0;
#pragma unroll
                for (int q = 0; q < LANE_WORDS; q += 2) {
                    uint2 two = make_uint2(0u, 0u);
                    if (per_lane == 1) {
                        if (q == 0 && v0 < len) two.x = __ldg(x + v0);
                    } else if (v0 + q < len) {
                        two = __ldg(reinterpret_cast<const uint2*>(x + v0 + q));
                    }
                    word[q] = two.x;
                    word[q + 1] = two.y;
                }
#pragma unroll
                for (int q = 0; q < LANE_WORDS; q++) set += __popc(word[q]);
                int inc = set;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, inc, d);
                    if (lane >= d) inc += y;
                }
                const int total = __shfl_sync(0xffffffffu, inc, 31);
                if (total == 0) continue;
                if (held + total > PROJ_LIST) {
                    // Whole words out; the rows left over move to the front.
                    const int n_out = held / 32;
                    flush(n_out);
                    const int left = held - 32 * n_out;
                    const uint16_t keep = lane < left ? list[32 * n_out + lane] : (uint16_t)0;
                    __syncwarp();
                    if (lane < left) list[lane] = keep;
                    held = left;
                    __syncwarp();
                }
                int to = held + inc - set;
#pragma unroll
                for (int q = 0; q < LANE_WORDS; q++)
                    for (uint32_t rest = word[q]; rest != 0u; rest &= rest - 1u)
                        list[to++] = (uint16_t)((v0 + q) * 32 + __ffs(rest) - 1);
                held += total;
            }
            flush(out_n - done);
        }
        projected = PROJ_DONE;
    }
    return grid_barrier(a.scratch) ? projected : PROJ_LOST;
}
// The candidates and tiles of the next level: its offsets, T, tiles, groups, work. Up to SMEM_ROWS rows every CTA scans
// them all, which costs less than a barrier, and holds the offsets in shared memory; past it each CTA scans its part,
// and the offsets lie in memory. False: a wait gave up.
__device__ __noinline__ bool scan_level() {
    const DirectArgs& a = args_sh();
    __shared__ int64_t pair_sums[DWARPS];
    State& S = state_sh();
    const int tid = threadIdx.x, lane = tid & 31, b = blockIdx.x, G = gridDim.x;
    const int n = S.n, w = S.w;
    const bool shared = n <= SMEM_ROWS;
    const int r_lo = shared ? 0 : (int)((int64_t)n * b / G), r_hi = shared ? n : (int)((int64_t)n * (b + 1) / G);
    int32_t* partial = a.scratch + a.at.partial;
    int64_t* sums = reinterpret_cast<int64_t*>(partial + MAX_GRID);  // [3][MAX_GRID]: candidates, tiles, work
    if (tid == 0) {
        S.groups = S.survivors = S.base = S.fresh = 0;
        S.work = 0;
        S.shared = shared;
    }
    __syncthreads();
    int groups = 0;
    int64_t T = 0, tiles = 0, work = 0;
    // Scans the rows from T candidates and tiles on; writes their offsets, or sums up groups and work.
    auto scan_rows = [&](int32_t* coff, int32_t* toff, bool sum_up) {
        for (int r0 = r_lo; r0 < r_hi; r0 += DT) {
            const int r = r0 + tid;
            int cands = 0, nt = 0;
            if (r < r_hi) {
                const int end = group_end(a, S, r);
                cands = min(end - 1 - r, ROW_CANDS);
                if (cands > 0) {
                    if (r == 0 || (w > 1 && group_end(a, S, r - 1) == r)) {
                        const int nb = (min(end - r, ROW_CANDS) + GB - 1) / GB;
                        nt = nb * (nb + 1) / 2;
                        groups += 1;
                    }
                    if (sum_up && S.projected) work += (int64_t)cands * __ldcg(a.pscratch + a.pat.cw + row_item(S, r, 0));
                }
            }
            int64_t total;
            const int64_t at = scan_pairs(((int64_t)cands << 32) + nt, &total, pair_sums);
            if (coff != nullptr && r < r_hi) {
                coff[r] = (int)(T + (at >> 32));
                toff[r] = (int)(tiles + (at & 0xffffffff));
            }
            T += total >> 32;
            tiles += total & 0xffffffff;
        }
    };
    if (shared) scan_rows(offsets, offsets + SMEM_ROWS + 1, true);
    else scan_rows(nullptr, nullptr, true);
    groups = __reduce_add_sync(0xffffffffu, groups);
    if (lane == 0 && groups != 0) atomicAdd(&S.groups, groups);
    if (work != 0) atomicAdd(&S.work, (unsigned long long)work);
    __syncthreads();
    if (!shared) {
        if (tid == 0) {
            sums[b] = T;
            sums[MAX_GRID + b] = tiles;
            sums[2 * MAX_GRID + b] = (int64_t)S.work;
            partial[b] = S.groups;
        }
        if (!grid_barrier(a.scratch)) return false;
        int64_t t_before, tile_before;
        const int64_t t_all = sum_over_ctas(sums, &t_before), tile_all = sum_over_ctas(sums + MAX_GRID, &tile_before);
        const int64_t work_all = sum_over_ctas(sums + 2 * MAX_GRID, nullptr);
        if (tid == 0) {
            S.work = (unsigned long long)work_all;
            S.groups = 0;
        }
        __syncthreads();
        for (int c = tid; c < G; c += DT) atomicAdd(&S.groups, __ldcg(partial + c));
        T = t_before;
        tiles = tile_before;
        if (t_all <= a.cap_cands) scan_rows(a.scratch + a.at.coff, a.scratch + a.at.toff, false);
        T = t_all;
        tiles = tile_all;
    }
    if (tid == 0) {
        S.T = T;
        S.tiles = tiles;
        if (T <= a.cap_cands) {
            // Slabs: for units enough, and for warps that run side by side to read the same words of the columns.
            const int mean = S.projected ? (int)(S.work / (unsigned)max((int)T, 1)) : (int)a.n_words;  // of a column
            S.n_slab = max(min(max(mean / SLAB_MIN, 1), 2 * G * DWARPS / max((int)tiles, 1)), (mean + SLAB_MAX - 1) / SLAB_MAX);
            if (S.n_slab < 1) S.n_slab = 1;
            const int words = ((int)T + 31) / 32;
            S.c_lo = words * b / G * 32;
            S.c_hi = min((int)T, words * (b + 1) / G * 32);
            if (shared) {
                offsets[n] = (int)T;
                offsets[SMEM_ROWS + 1 + n] = (int)tiles;
            } else if (b == G - 1) {
                a.scratch[a.at.coff + n] = (int)T;
                a.scratch[a.at.toff + n] = (int)tiles;
            }
        }
    }
    __syncthreads();
    return true;
}

// Marks and counts the survivors of this CTA's candidates.
__device__ __noinline__ void select_level() {
    const DirectArgs& a = args_sh();
    State& S = state_sh();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c_lo = S.c_lo, c_hi = S.c_hi;
    const int32_t* cnt = a.scratch + a.at.cnt;
    uint32_t* mask = reinterpret_cast<uint32_t*>(a.scratch + a.at.mask);
    // The free-set prune looks rows up by search: in shared memory, where they fit in the tiles' place.
    int32_t* rows_sh = offsets + SMEM_ROWS + 1;
    const bool held = a.prune && S.rows != nullptr && S.shared && (int64_t)S.n * S.w <= SMEM_ROWS;
    if (held) {
        for (int i = threadIdx.x; i < S.n * S.w; i += DT) rows_sh[i] = __ldcg(S.rows + i);
        __syncthreads();
    }
    for (int c0 = c_lo + 32 * warp; c0 < c_hi; c0 += DT) {
        const int c = c0 + lane;
        const int v = c < c_hi ? __ldcg(cnt + c) : -1;
        bool keep = v >= a.min_count;
        if (a.prune && keep) {
            // Free: every (k-1)-subset is a generator with a larger count.
            int j;
            const int r = with_offsets(a, S.shared, [&](const int32_t* coff, const int32_t*) {
                const int at = row_of(coff, S.n, c);
                j = at + 1 + (c - coff[at]);
                return at;
            });
            keep = __ldcg(S.counts + r) != v && __ldcg(S.counts + j) != v;
            const int last = row_item(S, j, S.w - 1);
            for (int d = 0; d + 1 < S.w && keep; d++) {
                const int f = held ? find_without([&](int i, int q) { return rows_sh[i * S.w + q]; }, S.n, S.w, r, d, last)
                                   : find_without([&](int i, int q) { return item_at(S.rows, S.w, i, q); }, S.n, S.w, r, d,
                                                  last);
                keep = f >= 0 && __ldcg(S.counts + f) != v;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) {
            mask[c0 >> 5] = m;
            if (m != 0u) atomicAdd(&S.survivors, __popc(m));
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) a.scratch[a.at.partial + blockIdx.x] = S.survivors;
}

// Writes the survivors of this CTA's candidates as rows of the next level, with their parents. False: they do not fit.
__device__ __noinline__ bool compact_level() {
    const DirectArgs& a = args_sh();
    __shared__ int warp_sums[DWARPS + 1];
    __shared__ int chunk_off[DT];
    State& S = state_sh();
    const int tid = threadIdx.x, lane = tid & 31, b = blockIdx.x, G = gridDim.x;
    const int n = S.n, w = S.w, k = w + 1, c_lo = S.c_lo, c_hi = S.c_hi;
    const int32_t* cnt = a.scratch + a.at.cnt;
    const uint32_t* mask = reinterpret_cast<const uint32_t*>(a.scratch + a.at.mask);
    int32_t* par = a.scratch + a.at.par;
    int32_t* pstart = a.scratch + a.at.pstart;
    const bool few = !a.prune && S.T <= FEW_CANDS;
    if (few) {
        int before = 0, all = 0;
#pragma unroll 4
        for (int c = tid; c < (int)S.T; c += DT) {
            const int keep = __ldcg(cnt + c) >= a.min_count;
            all += keep;
            if (c < c_lo) before += keep;
        }
        before = __reduce_add_sync(0xffffffffu, before);
        all = __reduce_add_sync(0xffffffffu, all);
        if (lane == 0) {
            atomicAdd(&S.base, before);
            atomicAdd(&S.fresh, all);
        }
    } else if (tid < 32) {
        int before = 0, all = 0;
        for (int c = lane; c < G; c += 32) {
            const int v = __ldcg(a.scratch + a.at.partial + c);
            all += v;
            if (c < b) before += v;
        }
        before = __reduce_add_sync(0xffffffffu, before);
        all = __reduce_add_sync(0xffffffffu, all);
        if (lane == 0) {
            S.base = before;
            S.fresh = all;
        }
    }
    __syncthreads();
    const int n_new = S.fresh;
    if (n_new > a.cap_rows || S.rows_used + (int64_t)n_new * k > a.rows_cap || S.counts_used + n_new > a.counts_cap)
        return false;
    // No CTA reads the parents (par, pstart) of the level being extended any more; its rows are still read, and the new
    // level goes to memory of its own.
    int32_t* new_rows = a.out_rows + S.rows_used;
    int32_t* new_counts = a.out_counts + S.counts_used;
    auto write = [&](const int32_t* coff, const int32_t*) {
        int run = S.base;
        for (int c0 = c_lo; c0 < c_hi; c0 += DT) {
            const int c = c0 + tid;
            const bool keep = c < c_hi && (few ? __ldcg(cnt + c) >= a.min_count
                                               : ((__ldcg(mask + (c >> 5)) >> (c & 31)) & 1u) != 0u);
            int total;
            const int at = run + scan_ints(keep ? 1 : 0, &total, warp_sums);
            chunk_off[tid] = at;
            if (keep) {
                const int r = row_of(coff, n, c);
                int32_t* o = new_rows + (int64_t)at * k;
                for (int t = 0; t < w; t++) o[t] = row_item(S, r, t);
                o[w] = row_item(S, r + 1 + (c - coff[r]), w - 1);
                new_counts[at] = __ldcg(cnt + c);
                par[at] = r;
            }
            __syncthreads();
            // First new row of every parent whose first candidate lies in this chunk.
            const int c1 = min(c0 + DT, c_hi);
            for (int r = lower_bound(coff, n, c0) + tid; r <= n && coff[r] < c1; r += DT)
                pstart[r] = chunk_off[coff[r] - c0];
            run += total;
            __syncthreads();
        }
        if (b == G - 1)  // rows past the last candidate
            for (int r = lower_bound(coff, n, (int)S.T) + tid; r <= n; r += DT) pstart[r] = n_new;
        return 0;
    };
    with_offsets(a, S.shared, write);
    if (b == 0 && tid == 0) {
        a.header[8 + 4 * k] = n_new;
        a.header[8 + 4 * k + 1] = S.T;
        a.header[8 + 4 * k + 2] = S.groups;
    }
    return true;
}

// The first level: K=1 from the columns' counts, or the given one. False: nothing follows.
__device__ __noinline__ bool first_level() {
    const DirectArgs& a = args_sh();
    __shared__ int warp_sums[DWARPS + 1];
    State& S = state_sh();
    const int tid = threadIdx.x, b = blockIdx.x, G = gridDim.x;
    int32_t* pstart = a.scratch + a.at.pstart;
    if (tid == 0) {
        S.rows = a.rows;
        S.counts = a.counts;
        S.map = nullptr;
        S.rows_used = S.counts_used = 0;
        S.n = a.n;
        S.w = a.width;
        S.n_items = (int)a.n_cols;
        S.bar_target = 0;
        S.searched = false;
        S.projected = a.projected != 0;
    }
    __syncthreads();
    if (a.proj_words > 0 && !a.projected && b == 0)
        for (int i = tid; i < PROJ_ITEMS && i < a.n_cols; i += DT) a.pscratch[a.pat.gsize + i] = 0;
    if (a.col_counts != nullptr) {
        // K=1: the frequent columns (under the free-set prune, those short of every row), ascending.
        if (b == 0) {
            int run = 0;
            for (int64_t c0 = 0; c0 < a.n_cols; c0 += DT) {
                const int64_t c = c0 + tid;
                const int64_t v = c < a.n_cols ? a.col_counts[c] : 0;
                const bool keep = c < a.n_cols && v >= a.min_count && (!a.prune || v < a.n_rows);
                int total;
                const int at = run + scan_ints(keep ? 1 : 0, &total, warp_sums);
                if (keep && at < a.cap_rows) {
                    a.out_rows[at] = (int32_t)c;
                    a.out_counts[at] = (int32_t)v;
                }
                run += total;
            }
            if (tid == 0) pstart[0] = run;
        }
        if (!grid_barrier(a.scratch)) return false;
        const int n = __ldcg(pstart);
        if (n > a.cap_rows) {
            if (b == 0 && tid == 0) a.header[0] = ETM_DIRECT_LIMIT, a.header[1] = 0;
            return false;
        }
        if (n <= MAP_ITEMS)
            for (int i = tid; i < n; i += DT) map_sh()[i] = __ldcg(a.out_rows + i);
        if (tid == 0) {
            S.n = S.n_items = n;
            S.w = 1;
            S.map = a.out_rows;
            S.rows = nullptr;
            S.counts = a.out_counts;
            S.rows_used = S.counts_used = n;
            if (b == 0) {
                a.header[8 + 4] = n;
                a.header[8 + 5] = a.n_cols;
                a.header[8 + 6] = 0;
            }
        }
    } else {
        // Group ends of the given level: the last row sharing row r's first w - 1 items, by binary search.
        const int n = a.n, w = a.width;
        for (int r = b * DT + tid; r < n; r += G * DT) {
            int lo = r, hi = n;  // rows[lo] shares the prefix, rows[hi] does not
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                bool same = true;
                for (int t = 0; t < w - 1 && same; t++) same = item_at(a.rows, w, mid, t) == item_at(a.rows, w, r, t);
                if (same) lo = mid;
                else hi = mid;
            }
            pstart[r] = hi;
        }
        if (tid == 0) S.searched = true;
        if (!grid_barrier(a.scratch)) return false;
    }
    __syncthreads();
    return true;
}

template <class V>
__global__ void __launch_bounds__(DT, 1) direct_mine_kernel(const __grid_constant__ DirectArgs a) {
    State& S = state_sh();
    const int tid = threadIdx.x;
    if (tid == 0) args_sh() = a;
    __syncthreads();
    if (!first_level()) return;
    bool may_project = a.proj_words > 0 && S.n_items <= PROJ_ITEMS && a.col_counts == nullptr && a.width == 2 && !a.projected;
    int status = ETM_DIRECT_DONE, full = 0;
    for (;;) {
        if (S.w + 1 > a.max_k || S.n < S.w + 1) break;
        if (!scan_level()) return;
        const int64_t T = S.T;
        if (may_project && S.w == 2 && T <= a.cap_cands && T * a.n_words >= PROJ_WORK) {
            // Once, before K=3; then the scan again: the projection used the offsets' memory and changes the work.
            may_project = false;
            const int done = project_columns<V>();
            if (done == PROJ_LOST) return;
            if (tid == 0) S.projected = done == PROJ_DONE;
            __syncthreads();
            continue;
        }
        if (T > a.cap_cands || (S.projected ? (int64_t)S.work : T * a.n_words) >
                                   (S.projected || S.w == 1 ? a.work_limit : a.deep_limit)) {
            status = ETM_DIRECT_LIMIT;
            full = T > a.cap_cands ? ETM_DIRECT_CANDS_FULL : 0;
            break;
        }
        if (!S.shared || S.n_slab > 1) {
            if (S.n_slab > 1)
                for (int c = S.c_lo + tid; c < S.c_hi; c += DT) a.scratch[a.at.cnt + c] = 0;
            if (!grid_barrier(a.scratch)) return;
        }
        if (S.projected) count_units<V, true>();
        else count_units<V, false>();
        if (!grid_barrier(a.scratch)) return;
        // Few candidates are not selected in a phase of their own: every CTA reads all counts for less than a barrier.
        if (a.prune || T > FEW_CANDS) {
            select_level();
            if (!grid_barrier(a.scratch)) return;
        }
        if (!compact_level()) {
            status = ETM_DIRECT_LIMIT;
            full = ETM_DIRECT_ROWS_FULL;
            break;
        }
        if (!grid_barrier(a.scratch)) return;
        if (tid == 0) {
            const int k = S.w + 1, n_new = S.fresh;
            S.rows = a.out_rows + S.rows_used;
            S.counts = a.out_counts + S.counts_used;
            S.rows_used += (int64_t)n_new * k;
            S.counts_used += n_new;
            S.n = n_new;
            S.w = k;
            S.searched = false;
        }
        __syncthreads();
        if (S.n == 0) break;
    }
    if (blockIdx.x == 0 && tid == 0) {
        a.header[1] = S.w;
        a.header[2] = full;
        a.header[3] = S.projected;
        a.header[0] = status;
    }
}

}  // namespace

extern "C" int etm_direct_scratch_words(int32_t cap_rows, int32_t cap_cands, int64_t n_cols, int64_t n_words,
                                        int64_t proj_words, int64_t* out, int64_t* proj_out) {
    ETM_REQUIRE(cap_rows >= 1 && cap_rows <= ETM_DIRECT_ROWS && cap_cands >= 1 && cap_cands <= ETM_DIRECT_CANDS &&
                    n_cols >= 0 && n_words >= 0 && proj_words >= 0 && proj_words <= ETM_DIRECT_PROJ,
                ETM_EINVAL, "etm_direct_scratch_words: bad sizes");
    *out = scratch_layout(cap_rows, cap_cands).words;
    *proj_out = proj_layout(n_cols, n_words, proj_words).words;
    return ETM_OK;
}

namespace {

struct Event {
    cudaEvent_t e = nullptr;
    ~Event() {
        if (e != nullptr) cudaEventDestroy(e);
    }
};

}  // namespace

// A launch's header and the start of its outputs to page-locked host memory with one wait: a copy and a wait each took
// 30 us a mine, of 0.33 ms for the smallest. keep: the same counts and rows for the caller to hold on to, copied on the
// device after the wait's copies, so that it is not waited for (made before them it took 15 us of 0.29 ms).
extern "C" int etm_direct_take(const int64_t* header, const int32_t* counts, int64_t n_counts, const int32_t* rows,
                               int64_t n_rows, int32_t* host, int32_t* keep, void* stream) {
    ETM_REQUIRE(n_counts >= 0 && n_rows >= 0, ETM_EINVAL, "etm_direct_take: negative size");
    constexpr int64_t HEAD = 8 + 4 * (ETM_DIRECT_LEVELS + 1);
    cudaStream_t s = as_stream(stream);
    Event done;
    if (keep != nullptr) ETM_CUDA(cudaEventCreateWithFlags(&done.e, cudaEventDisableTiming));
    const bool joined = counts == reinterpret_cast<const int32_t*>(header + HEAD);  // as they are on the host
    ETM_CUDA(cudaMemcpyAsync(host, header, HEAD * 8 + (joined ? (size_t)n_counts * 4 : 0), cudaMemcpyDeviceToHost, s));
    if (!joined) ETM_CUDA(cudaMemcpyAsync(host + 2 * HEAD, counts, (size_t)n_counts * 4, cudaMemcpyDeviceToHost, s));
    ETM_CUDA(cudaMemcpyAsync(host + 2 * HEAD + n_counts, rows, (size_t)n_rows * 4, cudaMemcpyDeviceToHost, s));
    if (keep == nullptr) {
        ETM_CUDA(cudaStreamSynchronize(s));
        return ETM_OK;
    }
    ETM_CUDA(cudaEventRecord(done.e, s));
    ETM_CUDA(cudaMemcpyAsync(keep, counts, (size_t)n_counts * 4, cudaMemcpyDeviceToDevice, s));
    ETM_CUDA(cudaMemcpyAsync(keep + n_counts, rows, (size_t)n_rows * 4, cudaMemcpyDeviceToDevice, s));
    ETM_CUDA(cudaEventSynchronize(done.e));
    return ETM_OK;
}

extern "C" int etm_direct_fetch(const int64_t* header, const int32_t* counts, int64_t n_counts, const int32_t* rows,
                                int64_t n_rows, int32_t* host, void* stream) {
    return etm_direct_take(header, counts, n_counts, rows, n_rows, host, nullptr, stream);
}

extern "C" int etm_mine_direct(const uint64_t* bv, int64_t ld, int64_t n_words, int64_t n_cols,
                               const int64_t* col_counts, int64_t n_rows, int32_t min_count, int32_t prune,
                               int32_t max_k, int64_t work_limit, int64_t deep_limit, const int32_t* start_rows,
                               const int32_t* start_counts, int64_t start_n, int32_t start_width, int64_t* header,
                               int32_t* out_counts, int64_t counts_cap, int32_t* out_rows, int64_t rows_cap,
                               int32_t cap_rows, int32_t cap_cands, int64_t proj_words, int32_t projected,
                               int32_t* scratch, int64_t scratch_words, int32_t* proj_scratch,
                               int64_t proj_scratch_words, void* stream) {
    ETM_REQUIRE(n_words >= 0 && ld >= n_words && n_cols >= 0 && work_limit >= 0 && deep_limit >= 0, ETM_EINVAL, "etm_mine_direct: bad sizes");
    ETM_REQUIRE(max_k >= 1 && max_k <= ETM_DIRECT_LEVELS, ETM_EINVAL, "etm_mine_direct: max_k %d out of range", max_k);
    ETM_REQUIRE(cap_rows >= 1 && cap_rows <= ETM_DIRECT_ROWS && cap_cands >= 1 && cap_cands <= ETM_DIRECT_CANDS &&
                    proj_words >= 0 && proj_words <= ETM_DIRECT_PROJ,
                ETM_EINVAL, "etm_mine_direct: bad capacities");
    const Scratch at = scratch_layout(cap_rows, cap_cands);
    const ProjScratch pat = proj_layout(n_cols, n_words, proj_words);
    ETM_REQUIRE(proj_words == 0 || (proj_scratch_words >= pat.words && (reinterpret_cast<uintptr_t>(proj_scratch) & 15) == 0),
                ETM_ENOSPACE, "etm_mine_direct: projection scratch of %lld words (16-byte aligned), need %lld",
                (long long)proj_scratch_words, (long long)pat.words);
    ETM_REQUIRE(!projected || (proj_words > 0 && col_counts == nullptr), ETM_EINVAL,
                "etm_mine_direct: projected columns without their scratch or a start level");
    ETM_REQUIRE(scratch_words >= at.words && (reinterpret_cast<uintptr_t>(scratch) & 15) == 0, ETM_ENOSPACE,
                "etm_mine_direct: scratch of %lld words (16-byte aligned), need %lld", (long long)scratch_words,
                (long long)at.words);
    if (col_counts != nullptr)
        ETM_REQUIRE(rows_cap >= cap_rows && counts_cap >= cap_rows, ETM_ENOSPACE, "etm_mine_direct: outputs below %d rows",
                    cap_rows);
    else
        ETM_REQUIRE(start_rows != nullptr && start_counts != nullptr && start_n >= 1 && start_n <= cap_rows &&
                        start_width >= 2 && start_width < ETM_DIRECT_LEVELS,
                    ETM_EINVAL, "etm_mine_direct: the start level needs 1..%d rows of 2 items or more", cap_rows);
    cudaStream_t s = as_stream(stream);
    const bool vec = ld % 2 == 0 && n_words % 2 == 0 && (reinterpret_cast<uintptr_t>(bv) & 15) == 0;
    const void* kernel = vec ? (const void*)direct_mine_kernel<ulonglong2> : (const void*)direct_mine_kernel<uint64_t>;
    ETM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    ETM_CUDA(cudaMemsetAsync(header, 0xFF, sizeof(int64_t), s));
    ETM_CUDA(cudaMemsetAsync(scratch, 0, 3 * sizeof(int32_t), s));
    DirectArgs a{bv,         ld,           n_words, n_cols,     col_counts, n_rows,     min_count,
                 prune,      max_k,        work_limit, deep_limit, start_rows, start_counts, (int)start_n, start_width,
                 header,     out_counts,   counts_cap, out_rows,   rows_cap,   scratch,    at,
                 proj_scratch, pat,        cap_rows, cap_cands,  proj_words, projected};
    void* args[] = {&a};
    const int grid = min(MAX_GRID, max(1, sm_count()));
    ETM_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(DT), args, (size_t)SMEM_BYTES, s));
    ETM_LAUNCHED("mine_direct");
    return ETM_OK;
}
