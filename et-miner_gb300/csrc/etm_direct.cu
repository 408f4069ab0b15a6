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
// Every CTA computes the candidate and tile offsets of a level itself (ordered scans over the rows, in shared memory),
// which costs less than a further barrier. The kernel stops, and says so, before a level past its limits (rows,
// candidates, candidate words) and the caller goes on from the last complete level.
//
// Measured per mine, general path against this kernel: 10,000 rows (108 frequent items, 5 levels) 3.1 -> 0.32 ms, of
// which 0.06 ms on the device; 33,333 rows under the free-set prune 7.6 -> 2.1 ms; 1M rows (267 frequent items, 6
// levels, 7.8e8 candidate words) 4.7 -> 1.0 ms. The caller's limit of 2^30 candidate words a level (about 0.6 ms)
// lies where the general path's launches and its tensor-core Gram take as long.
//
// The grid barriers hold only while every CTA is resident, hence the cooperative launch; their waits are bounded in
// time (%globaltimer), after which every CTA leaves and the header keeps the value the caller set it to.
#include "etm_tile.cuh"

namespace {

using namespace etm;

constexpr int DT = 512;                   // threads per CTA: 128 registers each, for the tiles
constexpr int DWARPS = DT / 32;
constexpr int CAP_ROWS = ETM_DIRECT_ROWS; // rows of a level
constexpr int CAP_CANDS = 1 << 22;        // candidates of a level
constexpr int SLAB_MIN = 256;             // words of a slab at least
constexpr int MAXW = ETM_DIRECT_LEVELS;
constexpr int MAX_GRID = 256;
constexpr uint64_t BARRIER_NS = 2000000000ull;

// Scratch layout, in 32-bit words.
constexpr int64_t S_BAR = 0;                               // barrier counter, abort flag
constexpr int64_t S_PARTIAL = 64;                          // survivors of each CTA
constexpr int64_t S_PAR = S_PARTIAL + MAX_GRID;            // parent row of each row of the level being written / read
constexpr int64_t S_PSTART = S_PAR + CAP_ROWS;             // first new row of each parent
constexpr int64_t S_MASK = S_PSTART + CAP_ROWS + 64;       // survivor bits, by candidate
constexpr int64_t S_COUNT = S_MASK + CAP_CANDS / 32;       // counts, by candidate
constexpr int64_t S_WORDS = S_COUNT + CAP_CANDS;

struct DirectArgs {
    const uint64_t* bv;  // columns [.][ld]
    int64_t ld;
    int64_t n_words, n_cols;
    const int64_t* col_counts;  // K=1 start: counts of the n_cols columns (nullptr: start from `rows`)
    int64_t n_rows;
    int min_count, prune, max_k;
    int64_t work_limit;         // candidate words of a level at most
    const int32_t* rows;        // start level [n][width] over the columns of bv
    const int32_t* counts;
    int n, width;
    int64_t* header;
    int32_t* out_counts;
    int64_t counts_cap;
    int32_t* out_rows;
    int64_t rows_cap;
    int32_t* scratch;
};

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
__device__ bool grid_barrier(int32_t* scratch, unsigned* target, int* ok_sh) {
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned* bar = reinterpret_cast<unsigned*>(scratch + S_BAR);
        unsigned* abort_flag = bar + 1;
        *target += gridDim.x;
        __threadfence();
        atomicAdd(bar, 1u);
        const uint64_t t0 = time_ns();
        while (load_acquire(bar) < *target) {
            if (load_acquire(abort_flag) != 0u) break;
            if (time_ns() - t0 > BARRIER_NS) {
                atomicExch(abort_flag, 1u);
                break;
            }
        }
        *ok_sh = load_acquire(abort_flag) == 0u;
        __threadfence();
    }
    __syncthreads();
    return *ok_sh != 0;
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

// Rows written by other CTAs of this launch are read through L2 (__ldcg): a line of L1 may be older.
__device__ __forceinline__ int item_at(const int32_t* rows, int w, int r, int q) { return __ldcg(rows + (int64_t)r * w + q); }

// Row of rows[n][w] holding row r's items without item d (d < w) plus `last` at the end, or -1.
__device__ int find_without(const int32_t* rows, int n, int w, int r, int d, int last) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        int cmp = 0;
        for (int t = 0; t < w && cmp == 0; t++) {
            const int v = t == w - 1 ? last : item_at(rows, w, r, t < d ? t : t + 1);
            const int x = item_at(rows, w, mid, t);
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

template <class V>
__global__ void __launch_bounds__(DT, 1) direct_mine_kernel(DirectArgs a) {
    extern __shared__ int32_t offsets[];
    int32_t* coff = offsets;                 // CAP_ROWS + 1: first candidate of each row
    int32_t* toff = offsets + CAP_ROWS + 1;  // CAP_ROWS + 1: first tile of each row (tiles belong to a group's first row)
    __shared__ int64_t tile_cols[DWARPS][2 * GB + MAXW];
    __shared__ int warp_sums[DWARPS + 1];
    __shared__ int chunk_off[DT];
    __shared__ int ok_sh, survivors_sh, base_sh, new_sh, groups_sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, G = gridDim.x;
    unsigned bar_target = 0;
    int32_t* par = a.scratch + S_PAR;
    int32_t* pstart = a.scratch + S_PSTART;
    uint32_t* mask = reinterpret_cast<uint32_t*>(a.scratch + S_MASK);
    int32_t* cnt = a.scratch + S_COUNT;
    constexpr int VW = sizeof(V) / 8;  // words per vector
    const int64_t n_vec = (a.n_words + VW - 1) / VW;  // 16-byte vectors: n_words is even

    const int32_t* map = nullptr;  // column of an item (nullptr: the item)
    const int32_t* rows = a.rows;
    const int32_t* counts = a.counts;
    int n = a.n, w = a.width;
    int64_t rows_used = 0, counts_used = 0;
    bool searched = false;  // the level's group ends are in pstart by row (a given start level), not by parent
    int status = ETM_DIRECT_DONE, level = w;

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
                if (keep && at < CAP_ROWS) {
                    a.out_rows[at] = (int32_t)c;
                    a.out_counts[at] = (int32_t)v;
                }
                run += total;
            }
            if (tid == 0) pstart[0] = run;
        }
        if (!grid_barrier(a.scratch, &bar_target, &ok_sh)) return;
        n = __ldcg(pstart);
        w = 1;
        level = 1;
        if (n > CAP_ROWS) {
            if (b == 0 && tid == 0) a.header[0] = ETM_DIRECT_LIMIT, a.header[1] = 0;
            return;
        }
        map = a.out_rows;
        rows = nullptr;  // row r of level 1 is item r
        counts = a.out_counts;
        rows_used = n;
        counts_used = n;
        if (b == 0 && tid == 0) {
            a.header[8 + 4] = n;
            a.header[8 + 5] = a.n_cols;
            a.header[8 + 6] = 0;
        }
    } else if (w > 1) {
        // Group ends of the given level: the last row sharing row r's first w - 1 items, by binary search.
        for (int r = b * DT + tid; r < n; r += G * DT) {
            int lo = r, hi = n;  // rows[lo] shares the prefix, rows[hi] does not
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                bool same = true;
                for (int t = 0; t < w - 1 && same; t++) same = item_at(rows, w, mid, t) == item_at(rows, w, r, t);
                if (same) lo = mid;
                else hi = mid;
            }
            pstart[r] = hi;
        }
        searched = true;
        if (!grid_barrier(a.scratch, &bar_target, &ok_sh)) return;
    }
    // End of row r's group.
    auto group_end = [&](int r) -> int {
        if (w == 1) return n;
        return searched ? __ldcg(pstart + r) : __ldcg(pstart + __ldcg(par + r) + 1);
    };
    auto item = [&](int r, int q) -> int { return rows == nullptr ? r : item_at(rows, w, r, q); };
    auto column = [&](int it) -> int64_t {  // its word offset
        return (map == nullptr ? (int64_t)it : (int64_t)__ldcg(map + it)) * a.ld;
    };

    for (;;) {
        const int k = w + 1;
        if (k > a.max_k || n < k) break;
        // ---- candidates and tiles of the level, by every CTA ----
        if (tid == 0) groups_sh = survivors_sh = 0;
        __syncthreads();
        int groups = 0, T = 0, tiles = 0;  // at most CAP_ROWS^2 / 2 candidates
        for (int r0 = 0; r0 < n; r0 += DT) {
            const int r = r0 + tid;
            const int end = r < n ? group_end(r) : 0;
            int nt = 0;
            if (r < n && end - r > 1 && (r == 0 || (w > 1 && group_end(r - 1) == r))) {
                const int nb = (end - r + GB - 1) / GB;
                nt = nb * (nb + 1) / 2;
                groups += 1;
            }
            int total;
            const int at = T + scan_ints(r < n ? end - 1 - r : 0, &total, warp_sums);
            T += total;
            const int tat = tiles + scan_ints(nt, &total, warp_sums);
            tiles += total;
            if (r < n) {
                coff[r] = at;
                toff[r] = tat;
            }
        }
        if (tid == 0) {
            coff[n] = T;
            toff[n] = tiles;
        }
        groups = __reduce_add_sync(0xffffffffu, groups);
        if (lane == 0 && groups != 0) atomicAdd(&groups_sh, groups);
        __syncthreads();
        if (T > CAP_CANDS || T * a.n_words > a.work_limit) {
            status = ETM_DIRECT_LIMIT;
            break;
        }
        // This CTA's run of candidates, in whole mask words.
        const int words = (T + 31) / 32;
        const int c_lo = (int)((int64_t)words * b / G) * 32, c_hi = min(T, (int)((int64_t)words * (b + 1) / G) * 32);
        // ---- count ----
        const int max_slab = (int)max64(1, a.n_words / SLAB_MIN);
        const int n_slab = max(1, min(max_slab, (2 * G * DWARPS) / max(1, tiles)));
        if (n_slab > 1) {
            for (int c = c_lo + tid; c < c_hi; c += DT) cnt[c] = 0;
            if (!grid_barrier(a.scratch, &bar_target, &ok_sh)) return;
        }
        const int64_t per = (n_vec + n_slab - 1) / n_slab;
        int64_t* off = tile_cols[warp];
        for (int64_t u = (int64_t)b + (int64_t)warp * G; u < (int64_t)tiles * n_slab; u += (int64_t)G * DWARPS) {
            const int slab = (int)(u / tiles), tile = (int)(u - (int64_t)slab * tiles);
            const int first = row_of(toff, n, tile);
            const int m = group_end(first) - first;
            const int nb = (m + GB - 1) / GB;
            int rest = tile - toff[first], ba = 0;
            while (rest >= nb - ba) rest -= nb - ba++;
            const int a0 = first + ba * GB, b0 = first + (ba + rest) * GB;
            const int na = min(GB, first + m - a0), nbm = min(GB, first + m - b0);
            __syncwarp();  // the previous tile is done with the offsets
            if (lane < GB) off[lane] = column(item(a0 + min(lane, na - 1), w - 1));
            else if (lane < 2 * GB) off[lane] = column(item(b0 + min(lane - GB, nbm - 1), w - 1));
            for (int q = lane; q < w - 1; q += 32) off[2 * GB + q] = column(item(first, q));
            __syncwarp();
            const GroupTile t{a.bv, slab * per, min64(n_vec, (slab + 1) * per), off + 2 * GB, off, off + GB, w - 1};
            count_any_tile<V>(t, lane, rest == 0, na, nbm, [&](int i, int j, int32_t c) {
                const int at = coff[a0 + i] + (b0 + j) - (a0 + i) - 1;
                if (n_slab == 1) cnt[at] = c;
                else if (c != 0) atomicAdd(cnt + at, c);
            });
        }
        if (!grid_barrier(a.scratch, &bar_target, &ok_sh)) return;
        // ---- select ----
        for (int c0 = c_lo + 32 * warp; c0 < c_hi; c0 += DT) {
            const int c = c0 + lane;
            const int v = c < c_hi ? __ldcg(cnt + c) : -1;
            bool keep = v >= a.min_count;
            if (a.prune && keep) {
                // Free: every (k-1)-subset is a generator with a larger count.
                const int r = row_of(coff, n, c);
                const int j = r + 1 + (c - coff[r]);
                keep = __ldcg(counts + r) != v && __ldcg(counts + j) != v;
                const int last = item(j, w - 1);
                for (int d = 0; d + 1 < w && keep; d++) {
                    const int f = find_without(rows, n, w, r, d, last);
                    keep = f >= 0 && __ldcg(counts + f) != v;
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) {
                mask[c0 >> 5] = m;
                if (m != 0u) atomicAdd(&survivors_sh, __popc(m));
            }
        }
        __syncthreads();
        if (tid == 0) a.scratch[S_PARTIAL + b] = survivors_sh;
        if (!grid_barrier(a.scratch, &bar_target, &ok_sh)) return;
        // ---- compact ----
        if (warp == 0) {
            int before = 0, all = 0;
            for (int c = lane; c < G; c += 32) {
                const int v = __ldcg(a.scratch + S_PARTIAL + c);
                all += v;
                if (c < b) before += v;
            }
            before = __reduce_add_sync(0xffffffffu, before);
            all = __reduce_add_sync(0xffffffffu, all);
            if (lane == 0) {
                base_sh = before;
                new_sh = all;
            }
        }
        __syncthreads();
        const int n_new = new_sh;
        if (n_new > CAP_ROWS || rows_used + (int64_t)n_new * k > a.rows_cap || counts_used + n_new > a.counts_cap) {
            status = ETM_DIRECT_LIMIT;
            break;
        }
        // No CTA reads the parents (par, pstart) of the level being extended any more; its rows are still read, and
        // the new level goes to memory of its own.
        int32_t* new_rows = a.out_rows + rows_used;
        int32_t* new_counts = a.out_counts + counts_used;
        int run = base_sh;
        for (int c0 = c_lo; c0 < c_hi; c0 += DT) {
            const int c = c0 + tid;
            const bool keep = c < c_hi && ((__ldcg(mask + (c >> 5)) >> (c & 31)) & 1u) != 0u;
            int total;
            const int at = run + scan_ints(keep ? 1 : 0, &total, warp_sums);
            chunk_off[tid] = at;
            if (keep) {
                const int r = row_of(coff, n, c);
                int32_t* o = new_rows + (int64_t)at * k;
                for (int t = 0; t < w; t++) o[t] = item(r, t);
                o[w] = item(r + 1 + (c - coff[r]), w - 1);
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
            for (int r = lower_bound(coff, n, T) + tid; r <= n; r += DT) pstart[r] = n_new;
        if (b == 0 && tid == 0) {
            a.header[8 + 4 * k] = n_new;
            a.header[8 + 4 * k + 1] = T;
            a.header[8 + 4 * k + 2] = groups_sh;
        }
        if (!grid_barrier(a.scratch, &bar_target, &ok_sh)) return;
        rows = new_rows;
        counts = new_counts;
        rows_used += (int64_t)n_new * k;
        counts_used += n_new;
        n = n_new;
        w = k;
        level = k;
        searched = false;
        if (n_new == 0) break;
    }
    if (b == 0 && tid == 0) {
        a.header[1] = level;
        a.header[0] = status;
    }
}

}  // namespace

extern "C" int etm_direct_scratch_words(void) { return (int)S_WORDS; }

extern "C" int etm_mine_direct(const uint64_t* bv, int64_t ld, int64_t n_words, int64_t n_cols,
                               const int64_t* col_counts, int64_t n_rows, int32_t min_count, int32_t prune,
                               int32_t max_k, int64_t work_limit, const int32_t* start_rows,
                               const int32_t* start_counts, int64_t start_n, int32_t start_width, int64_t* header,
                               int32_t* out_counts, int64_t counts_cap, int32_t* out_rows, int64_t rows_cap,
                               int32_t* scratch, int64_t scratch_words, void* stream) {
    ETM_REQUIRE(n_words >= 0 && ld >= n_words && n_cols >= 0 && work_limit >= 0, ETM_EINVAL, "etm_mine_direct: bad sizes");
    ETM_REQUIRE(max_k >= 1 && max_k <= ETM_DIRECT_LEVELS, ETM_EINVAL, "etm_mine_direct: max_k %d out of range", max_k);
    ETM_REQUIRE(scratch_words >= S_WORDS, ETM_ENOSPACE, "etm_mine_direct: scratch of %lld words, need %lld",
                (long long)scratch_words, (long long)S_WORDS);
    if (col_counts != nullptr)
        ETM_REQUIRE(rows_cap >= CAP_ROWS && counts_cap >= CAP_ROWS, ETM_ENOSPACE,
                    "etm_mine_direct: outputs below %d rows", CAP_ROWS);
    else
        ETM_REQUIRE(start_rows != nullptr && start_counts != nullptr && start_n >= 1 && start_n <= CAP_ROWS &&
                        start_width >= 2 && start_width < ETM_DIRECT_LEVELS,
                    ETM_EINVAL, "etm_mine_direct: the start level needs 1..%d rows of 2 items or more", CAP_ROWS);
    cudaStream_t s = as_stream(stream);
    constexpr int smem = 2 * (CAP_ROWS + 1) * 4;
    const bool vec = ld % 2 == 0 && n_words % 2 == 0 && (reinterpret_cast<uintptr_t>(bv) & 15) == 0;
    const void* kernel = vec ? (const void*)direct_mine_kernel<ulonglong2> : (const void*)direct_mine_kernel<uint64_t>;
    ETM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    ETM_CUDA(cudaMemsetAsync(header, 0xFF, sizeof(int64_t), s));
    ETM_CUDA(cudaMemsetAsync(scratch + S_BAR, 0, 2 * sizeof(int32_t), s));
    DirectArgs a{bv,         ld,           n_words, n_cols,     col_counts, n_rows,     min_count,
                 prune,      max_k,        work_limit, start_rows, start_counts, (int)start_n, start_width,
                 header,     out_counts,   counts_cap, out_rows,   rows_cap,   scratch};
    void* args[] = {&a};
    const int grid = min(MAX_GRID, max(1, sm_count()));
    ETM_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(DT), args, (size_t)smem, s));
    ETM_LAUNCHED("mine_direct");
    return ETM_OK;
}
