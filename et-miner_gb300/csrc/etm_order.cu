// Levels from the order they are counted in to the order they are returned in.
//
// The engine numbers the generators by ascending support while it counts: the prefix of a candidate is then its rarest
// items, so prefix groups hold few rows. A level comes out over that numbering, its rows sorted over it; the caller
// gets the columns' own order: every row's items renumbered and sorted, and the rows sorted lexicographically.
//
// A row becomes a key of `bits` bits per item, first item highest, in as many 64-bit words as its items take. Up to
// RANK_ROWS rows a row's place is the number of smaller keys, counted over all keys (two launches for any length). Up to
// MERGE_ROWS tiles are sorted in shared memory and a row's place is its own there and those of its key in the other tiles,
// found by search: three launches for any length, where a radix sort takes five per digit, and the same time however the
// keys are spread (41,000 rows of 6 items: 54 us, by radix 270; 65,536 rows of 11 items that share their first nine, so
// that every comparison reads a second word: 140 us, where counting within buckets of the leading bits took 12.8 ms; that
// took 57 us for rows of random items, this 55). Past that a least-significant-digit radix sort moves (key, payload) pairs 8 bits at a time: counts
// per digit and tile, their scan, and a stable scatter through shared memory so that each digit's run is written
// contiguously. It is bound by HBM: 8 bytes read for the counts and 24 moved per row and digit. Measured on 74.7M rows
// of 3 items (36 bits, 5 digits): 4.9 ms, against the 230 ms that counting over ascending supports takes off the mine
// (dense 2M x 4,096: 515 -> 278 ms; 1M x 2,048: 47.8 -> 28.7 ms; 20M deep sparse 16.6 -> 11.1 ms).
#include "etm_scan.cuh"

namespace {

using namespace etm;

constexpr int RANK_ROWS = 2048;
constexpr int MERGE_ROWS = 65536;  // 32 tiles: a search in each of the others is up to 341 steps a row
constexpr int TILE_ROWS = 2048;
constexpr int TILE_THREADS = TILE_ROWS / 2;
constexpr int RANK_THREADS = 256;
constexpr int MAX_ITEMS = 64;
constexpr int RX_THREADS = 512;
constexpr int RX_WARPS = RX_THREADS / 32;
constexpr int RX_ITEMS = 16;
constexpr int RX_TILE = RX_THREADS * RX_ITEMS;
constexpr int RX_BITS = 8;
constexpr int RX_BINS = 1 << RX_BITS;
constexpr int RX_SMEM = RX_TILE * 12;

// Key words of row t: its items renumbered by `perm` and sorted, per_word of them packed into each word (the last
// word's first), word q at keys[q n + t]. K > 0: the row's length at compile time.
template <int K>
__global__ void __launch_bounds__(256) order_keys_kernel(const int32_t* __restrict__ rows, int64_t n, int k_rt,
                                                         const int32_t* __restrict__ perm, int bits, int per_word,
                                                         uint64_t* __restrict__ keys, const int32_t* __restrict__ counts,
                                                         uint32_t* __restrict__ payload) {
    const int k = K > 0 ? K : k_rt;
    int32_t it[K > 0 ? K : MAX_ITEMS];
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int q = 0; q < k; q++) {
            const int32_t v = __ldg(perm + rows[t * k + q]);
            int p = q;
            if (K > 0) {
                it[q] = v;
            } else {
                while (p > 0 && it[p - 1] > v) {
                    it[p] = it[p - 1];
                    --p;
                }
                it[p] = v;
            }
        }
        if (K > 0) {
#pragma unroll
            for (int a = 0; a < k; a++)
#pragma unroll
                for (int c = 0; c + 1 < k - a; c++) {
                    const int32_t lo = min(it[c], it[c + 1]), hi = max(it[c], it[c + 1]);
                    it[c] = lo;
                    it[c + 1] = hi;
                }
        }
        uint64_t word = 0;
        int in = 0;
        int64_t w = 0;
#pragma unroll
        for (int q = 0; q < k; q++) {
            word = (word << bits) | (uint32_t)it[q];
            if (++in == per_word || q + 1 == k) {
                keys[w * n + t] = word;
                word = 0;
                in = 0;
                ++w;
            }
        }
        if (payload != nullptr) payload[t] = counts != nullptr ? (uint32_t)counts[t] : (uint32_t)t;
    }
}

// Row `at` of the output from the key words of input row t.
__device__ __forceinline__ void unpack_row(const uint64_t* __restrict__ keys, int64_t n, int64_t t, int k, int bits,
                                           int per_word, int32_t* __restrict__ out) {
    const uint64_t mask = (1ULL << bits) - 1ULL;
    for (int q0 = 0, w = 0; q0 < k; q0 += per_word, w++) {
        const int in = min(per_word, k - q0);
        const uint64_t word = keys[(int64_t)w * n + t];
        for (int q = 0; q < in; q++) out[q0 + q] = (int32_t)((word >> (bits * (in - 1 - q))) & mask);
    }
}

// Up to RANK_ROWS rows: a warp's lanes share a row and count the smaller keys among every 32nd (keys differ: the rows
// of a level are distinct itemsets).
__global__ void __launch_bounds__(RANK_THREADS) order_rank_kernel(const uint64_t* __restrict__ keys, int n, int nw,
                                                                  const int32_t* __restrict__ counts, int k, int bits,
                                                                  int per_word, int32_t* __restrict__ out_rows,
                                                                  int32_t* __restrict__ out_counts) {
    const int lane = threadIdx.x & 31;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n; t += n_warps) {
        const uint64_t mine = keys[t];
        int below = 0;
        for (int j = lane; j < n; j += 32) {
            uint64_t a = keys[j], b = mine;
            for (int w = 1; a == b && w < nw; w++) {
                a = keys[(int64_t)w * n + j];
                b = keys[(int64_t)w * n + t];
            }
            below += a < b ? 1 : 0;
        }
        below = __reduce_add_sync(0xffffffffu, below);
        if (lane == 0) {
            unpack_row(keys, n, t, k, bits, per_word, out_rows + (int64_t)below * k);
            out_counts[below] = counts[t];
        }
    }
}

// Whether the row of key (first word x, row t) sorts before that of (y, u). Rows past the level (NO_ROW) are last.
constexpr uint32_t NO_ROW = 0xFFFFFFFFu;
__device__ __forceinline__ bool key_less(uint64_t x, uint32_t t, uint64_t y, uint32_t u, const uint64_t* __restrict__ keys,
                                         int64_t n, int nw) {
    if (x != y) return x < y;
    if (nw == 1 || t == NO_ROW || u == NO_ROW) return t != NO_ROW && u == NO_ROW;
    uint64_t a = 0, b = 0;
    for (int w = 1; a == b && w < nw; w++) {
        a = keys[w * n + t];
        b = keys[w * n + u];
    }
    return a < b;
}

// Tiles of TILE_ROWS rows, each sorted (bitonic, in shared memory): first key words and row numbers.
__global__ void __launch_bounds__(TILE_THREADS) tile_sort_kernel(const uint64_t* __restrict__ keys, int n, int nw,
                                                                 uint64_t* __restrict__ sorted, uint32_t* __restrict__ idx) {
    __shared__ uint64_t x[TILE_ROWS];
    __shared__ uint32_t id[TILE_ROWS];
    const int base = blockIdx.x * TILE_ROWS;
    for (int i = threadIdx.x; i < TILE_ROWS; i += TILE_THREADS) {
        x[i] = base + i < n ? keys[base + i] : ~0ULL;
        id[i] = base + i < n ? (uint32_t)(base + i) : NO_ROW;
    }
    __syncthreads();
    for (int k = 2; k <= TILE_ROWS; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int t = threadIdx.x, i = 2 * t - (t & (j - 1)), p = i + j;
            const uint64_t a = x[i], b = x[p];
            const uint32_t ia = id[i], ib = id[p];
            if (key_less(b, ib, a, ia, keys, n, nw) == ((i & k) == 0)) {
                x[i] = b;
                x[p] = a;
                id[i] = ib;
                id[p] = ia;
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < TILE_ROWS && base + i < n; i += TILE_THREADS) {
        sorted[base + i] = x[i];
        idx[base + i] = id[i];
    }
}

// 32 rows in a row of a tile by a block: each row's place in its own tile, and by searches in the others, which the warps
// share out. A warp's lanes are neighbours in order, so that their searches of a tile take nearly the same way and
// read the same few words (a lane per tile instead: 32 words a step, 65,536 rows 101 us).
__global__ void __launch_bounds__(RANK_THREADS) tile_rank_kernel(const uint64_t* __restrict__ keys, int n, int nw,
                                                                 const uint64_t* __restrict__ sorted,
                                                                 const uint32_t* __restrict__ idx,
                                                                 const int32_t* __restrict__ counts, int k, int bits,
                                                                 int per_word, int32_t* __restrict__ out_rows,
                                                                 int32_t* __restrict__ out_counts) {
    __shared__ int place[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane, n_tiles = (n + TILE_ROWS - 1) / TILE_ROWS;
    const uint64_t mine = p < n ? sorted[p] : 0ULL;
    const uint32_t t = p < n ? idx[p] : NO_ROW;
    if (warp == 0) place[lane] = p % TILE_ROWS;
    __syncthreads();
    int below = 0;
    for (int tile = warp; tile < n_tiles; tile += RANK_THREADS / 32) {
        if (tile == p / TILE_ROWS || p >= n) continue;
        const int first = tile * TILE_ROWS;
        int lo = first, hi = min(first + TILE_ROWS, n);
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (key_less(sorted[mid], nw == 1 ? 0u : idx[mid], mine, t, keys, n, nw)) lo = mid + 1;
            else hi = mid;
        }
        below += lo - first;
    }
    if (below != 0) atomicAdd(place + lane, below);
    __syncthreads();
    const uint64_t mask = (1ULL << bits) - 1ULL;
    for (int r = warp; r < 32 && blockIdx.x * 32 + r < n; r += RANK_THREADS / 32) {
        const uint32_t row = idx[blockIdx.x * 32 + r];
        const int at = place[r];
        for (int q = lane; q < k; q += 32) {
            const int w = q / per_word, in = min(per_word, k - w * per_word);
            out_rows[(int64_t)at * k + q] =
                (int32_t)((keys[(int64_t)w * n + row] >> (bits * (in - 1 - (q - w * per_word)))) & mask);
        }
        if (lane == 0) out_counts[at] = counts[row];
    }
}

__device__ __forceinline__ int digit_of(uint64_t key, int shift, uint32_t mask) { return (int)((uint32_t)(key >> shift) & mask); }

// Elements of each digit in each tile: table[digit n_tiles + tile].
__global__ void __launch_bounds__(RX_THREADS) radix_count_kernel(const uint64_t* __restrict__ keys, int64_t n, int shift,
                                                                 uint32_t mask, int64_t n_tiles,
                                                                 uint32_t* __restrict__ table) {
    __shared__ uint32_t hist[RX_BINS];
    for (int i = threadIdx.x; i < RX_BINS; i += RX_THREADS) hist[i] = 0u;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * RX_TILE;
#pragma unroll 4
    for (int i = 0; i < RX_ITEMS; i++) {
        const int64_t t = base + i * RX_THREADS + threadIdx.x;
        if (t < n) atomicAdd(&hist[digit_of(keys[t], shift, mask)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < RX_BINS; i += RX_THREADS) table[i * n_tiles + blockIdx.x] = hist[i];
}

struct TableVal {
    const uint32_t* table;
    __device__ int64_t operator()(int64_t i) const { return table[i]; }
};
struct TablePut {
    uint32_t* table;
    __device__ void operator()(int64_t i, int64_t off) const { table[i] = (uint32_t)off; }
};

// Stable scatter of a tile by one digit. Each warp owns RX_ITEMS x 32 consecutive elements and takes them 32 at a time
// in order; the lanes of a digit find each other by one ballot per bit, and the warp's count of the digit so far is
// kept in shared memory. The tile is put in order in shared memory and written out from there.
__global__ void __launch_bounds__(RX_THREADS) radix_scatter_kernel(const uint64_t* __restrict__ keys,
                                                                   const uint32_t* __restrict__ payload, int64_t n,
                                                                   int shift, uint32_t mask, int n_bits,
                                                                   int64_t n_tiles, const uint32_t* __restrict__ offsets,
                                                                   uint64_t* __restrict__ out_keys,
                                                                   uint32_t* __restrict__ out_payload) {
    extern __shared__ uint64_t sorted[];  // RX_TILE keys, then RX_TILE payloads
    uint32_t* sorted_p = reinterpret_cast<uint32_t*>(sorted + RX_TILE);
    __shared__ uint32_t hist[RX_WARPS][RX_BINS];
    __shared__ uint32_t start[RX_BINS];   // first place of the digit in the tile
    __shared__ uint32_t to[RX_BINS];      // its first place in the output, less `start`
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < RX_WARPS * RX_BINS; i += RX_THREADS) (&hist[0][0])[i] = 0u;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * RX_TILE;
    const int live = (int)min64(RX_TILE, n - base);
    uint64_t key[RX_ITEMS];
    uint32_t pay[RX_ITEMS], place[RX_ITEMS];
#pragma unroll
    for (int i = 0; i < RX_ITEMS; i++) {
        const int e = warp * (RX_ITEMS * 32) + i * 32 + lane;
        key[i] = e < live ? keys[base + e] : ~0ULL;
        pay[i] = e < live ? payload[base + e] : 0u;
    }
#pragma unroll
    for (int i = 0; i < RX_ITEMS; i++) {
        const int e = warp * (RX_ITEMS * 32) + i * 32 + lane;
        const int d = digit_of(key[i], shift, mask);
        unsigned peers = __ballot_sync(0xffffffffu, e < live);
        for (int q = 0; q < n_bits; q++) {
            const unsigned bal = __ballot_sync(0xffffffffu, (d >> q) & 1);
            peers &= ((d >> q) & 1) ? bal : ~bal;
        }
        uint32_t before = 0;
        if (e < live) before = hist[warp][d];
        __syncwarp();
        const unsigned below = peers & ((1u << lane) - 1u);
        place[i] = before + __popc(below);
        if (e < live && below == 0u) hist[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Per digit: the warps' counts to offsets within the digit, then the digits' starts in the tile.
    if (threadIdx.x < RX_BINS) {
        uint32_t run = 0;
        for (int w = 0; w < RX_WARPS; w++) {
            const uint32_t c = hist[w][threadIdx.x];
            hist[w][threadIdx.x] = run;
            run += c;
        }
        start[threadIdx.x] = run;
    }
    __syncthreads();
    int64_t total;
    const int64_t ex = block_exclusive_scan(threadIdx.x < RX_BINS ? start[threadIdx.x] : 0, &total);
    if (threadIdx.x < RX_BINS) {
        start[threadIdx.x] = (uint32_t)ex;
        to[threadIdx.x] = offsets[threadIdx.x * n_tiles + blockIdx.x] - (uint32_t)ex;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RX_ITEMS; i++) {
        const int e = warp * (RX_ITEMS * 32) + i * 32 + lane;
        if (e >= live) continue;
        const int d = digit_of(key[i], shift, mask);
        const uint32_t p = start[d] + hist[warp][d] + place[i];
        sorted[p] = key[i];
        sorted_p[p] = pay[i];
    }
    __syncthreads();
    for (int p = threadIdx.x; p < live; p += RX_THREADS) {
        const uint64_t x = sorted[p];
        const uint32_t at = to[digit_of(x, shift, mask)] + p;  // modulo 2^32: the sum is the place, below 2^32
        out_keys[at] = x;
        out_payload[at] = sorted_p[p];
    }
}

// Key word of the rows in the order of idx.
__global__ void __launch_bounds__(256) gather_keys_kernel(const uint64_t* __restrict__ words,
                                                          const uint32_t* __restrict__ idx, int64_t n,
                                                          uint64_t* __restrict__ out) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        out[t] = words[idx[t]];
}

// The sorted rows: from their keys with the counts as payload (idx nullptr), or from the key words of input row idx[t].
__global__ void __launch_bounds__(256) order_emit_kernel(const uint64_t* __restrict__ keys, int64_t n, int k, int bits,
                                                         int per_word, const uint32_t* __restrict__ payload,
                                                         const int32_t* __restrict__ counts,
                                                         int32_t* __restrict__ out_rows,
                                                         int32_t* __restrict__ out_counts) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t src = counts == nullptr ? t : (int64_t)payload[t];
        unpack_row(keys, n, src, k, bits, per_word, out_rows + t * k);
        out_counts[t] = counts == nullptr ? (int32_t)payload[t] : counts[src];
    }
}

// Candidates C(m, 2) and prefix groups of two rows or more of a sorted level: out[0] and out[1], added.
__global__ void __launch_bounds__(256) group_totals_kernel(const int32_t* __restrict__ rows, int64_t n, int width,
                                                           unsigned long long* __restrict__ out) {
    unsigned long long cands = 0;
    unsigned groups = 0;
    auto same = [&](int64_t a, int64_t b) {
        for (int c = 0; c < width - 1; c++)
            if (__ldg(rows + a * width + c) != __ldg(rows + b * width + c)) return false;
        return true;
    };
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        if (t > 0 && same(t - 1, t)) continue;
        // The first row of a prefix: the last row sharing it, by doubling steps and bisection.
        int64_t lo = t, hi = n, step = 1;
        while (lo + step < n) {
            if (!same(t, lo + step)) {
                hi = lo + step;
                break;
            }
            lo += step;
            step *= 2;
        }
        while (hi - lo > 1) {
            const int64_t mid = lo + ((hi - lo) >> 1);
            if (same(t, mid)) lo = mid;
            else hi = mid;
        }
        const int64_t m = lo + 1 - t;
        if (m >= 2) {
            cands += (unsigned long long)pairs_of(m);
            groups += 1;
        }
    }
    for (int d = 16; d > 0; d >>= 1) cands += __shfl_xor_sync(0xffffffffu, cands, d);
    groups = __reduce_add_sync(0xffffffffu, groups);
    if ((threadIdx.x & 31) == 0 && cands != 0) {
        atomicAdd(out, cands);
        atomicAdd(out + 1, (unsigned long long)groups);
    }
}

int grid_of(int64_t n, int threads) {
    return (int)max64(1, min64(ceil_div<int64_t>(n, threads), (int64_t)max(1, sm_count()) * 16));
}

struct OrderPlan {
    int per_word, nw;
    int64_t n_tiles, keys, idx, table, ws, bytes;  // byte offsets of the scratch's parts: key words at 0
};

OrderPlan order_plan(int64_t n, int k, int bits) {
    OrderPlan p;
    p.per_word = 64 / bits;
    p.nw = (k + p.per_word - 1) / p.per_word;
    p.n_tiles = ceil_div<int64_t>(n, RX_TILE);
    auto up = [](int64_t b) { return (b + 255) & ~(int64_t)255; };
    const bool big = n > MERGE_ROWS;
    p.keys = up(n * 8 * p.nw);                               // two key buffers (one where the words are the first)
    p.idx = p.keys + (big ? up(n * 8) * (p.nw > 1 ? 2 : 1) : 0);
    p.table = p.idx + (big ? 2 * up(n * 4) : 0);
    p.ws = p.table + (big ? up(RX_BINS * p.n_tiles * 4) : 0);
    p.bytes = p.ws + (big ? up(scan_workspace_words(RX_BINS * p.n_tiles) * 8) : 0);
    if (!big && n > RANK_ROWS) {
        p.idx = p.keys + up(n * 8);                          // sorted tiles: first key words, row numbers
        p.bytes = p.idx + up(n * 4);
    }
    return p;
}

}  // namespace

extern "C" int etm_order_level_bytes(int64_t n, int32_t k, int32_t bits, int64_t* out_bytes) {
    ETM_REQUIRE(n >= 0 && k >= 1 && k <= MAX_ITEMS && bits >= 1 && bits <= 31 && out_bytes != nullptr, ETM_EINVAL,
                "etm_order_level_bytes: bad sizes");
    *out_bytes = order_plan(n, k, bits).bytes;
    return ETM_OK;
}

extern "C" int etm_order_level_launches(int64_t n, int32_t k, int32_t bits) {
    if (n <= 0 || k < 1 || k > MAX_ITEMS || bits < 1 || bits > 31) return 0;
    if (n <= MERGE_ROWS) return n <= RANK_ROWS ? 2 : 3;
    const OrderPlan p = order_plan(n, k, bits);
    int launches = 2;  // the keys and the sorted rows; a word's gather, and a digit's counts, their scan and its scatter
    for (int w = 0; w < p.nw; w++)
        launches += (p.nw > 1 ? 1 : 0) + 5 * ((bits * min(p.per_word, k - w * p.per_word) + RX_BITS - 1) / RX_BITS);
    return launches;
}

extern "C" int etm_order_level(const int32_t* rows, const int32_t* counts, int64_t n, int32_t k, const int32_t* perm,
                               int32_t bits, int32_t* out_rows, int32_t* out_counts, uint8_t* scratch,
                               int64_t scratch_bytes, void* stream) {
    ETM_REQUIRE(n >= 0 && n < (1LL << 31) && k >= 1 && k <= MAX_ITEMS && bits >= 1 && bits <= 31, ETM_EINVAL,
                "etm_order_level: bad sizes");
    if (n == 0) return ETM_OK;
    const OrderPlan p = order_plan(n, k, bits);
    ETM_REQUIRE(scratch_bytes >= p.bytes, ETM_ENOSPACE, "etm_order_level: scratch of %lld bytes, need %lld",
                (long long)scratch_bytes, (long long)p.bytes);
    ETM_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 15) == 0, ETM_EINVAL, "etm_order_level: unaligned scratch");
    cudaStream_t s = as_stream(stream);
    uint64_t* words = reinterpret_cast<uint64_t*>(scratch);
    const bool big = n > MERGE_ROWS;
    const int64_t key_step = (n * 8 + 255) & ~(int64_t)255, idx_step = (n * 4 + 255) & ~(int64_t)255;
    uint64_t* kb[2] = {p.nw > 1 ? reinterpret_cast<uint64_t*>(scratch + p.keys) : words,
                       reinterpret_cast<uint64_t*>(scratch + p.keys + (p.nw > 1 ? key_step : 0))};
    uint32_t* pb[2] = {reinterpret_cast<uint32_t*>(scratch + p.idx), reinterpret_cast<uint32_t*>(scratch + p.idx + idx_step)};
    const int grid = grid_of(n, 256);
    const int32_t* pay_counts = p.nw == 1 ? counts : nullptr;  // one word: the counts travel with their keys
    uint32_t* pay = big ? pb[0] : nullptr;
    if (k == 2) order_keys_kernel<2><<<grid, 256, 0, s>>>(rows, n, k, perm, bits, p.per_word, words, pay_counts, pay);
    else if (k == 3) order_keys_kernel<3><<<grid, 256, 0, s>>>(rows, n, k, perm, bits, p.per_word, words, pay_counts, pay);
    else if (k == 4) order_keys_kernel<4><<<grid, 256, 0, s>>>(rows, n, k, perm, bits, p.per_word, words, pay_counts, pay);
    else order_keys_kernel<0><<<grid, 256, 0, s>>>(rows, n, k, perm, bits, p.per_word, words, pay_counts, pay);
    ETM_LAUNCHED("order_keys");
    if (!big && n > RANK_ROWS) {
        uint64_t* sorted = reinterpret_cast<uint64_t*>(scratch + p.keys);
        tile_sort_kernel<<<(unsigned)ceil_div<int64_t>(n, TILE_ROWS), TILE_THREADS, 0, s>>>(words, (int)n, p.nw, sorted, pb[0]);
        ETM_LAUNCHED("tile_sort");
        tile_rank_kernel<<<(unsigned)ceil_div<int64_t>(n, 32), RANK_THREADS, 0, s>>>(
            words, (int)n, p.nw, sorted, pb[0], counts, k, bits, p.per_word, out_rows, out_counts);
        ETM_LAUNCHED("tile_rank");
        return ETM_OK;
    }
    if (!big) {
        order_rank_kernel<<<grid_of(n * 32, RANK_THREADS), RANK_THREADS, 0, s>>>(words, (int)n, p.nw, counts, k, bits,
                                                                                 p.per_word, out_rows, out_counts);
        ETM_LAUNCHED("order_rank");
        return ETM_OK;
    }
    ETM_CUDA(cudaFuncSetAttribute(radix_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RX_SMEM));
    uint32_t* table = reinterpret_cast<uint32_t*>(scratch + p.table);
    int64_t* ws = reinterpret_cast<int64_t*>(scratch + p.ws);
    int cur = 0;  // buffers holding the current order
    for (int w = p.nw - 1; w >= 0; w--) {
        if (p.nw > 1) {
            gather_keys_kernel<<<grid, 256, 0, s>>>(words + (int64_t)w * n, pb[cur], n, kb[cur]);
            ETM_LAUNCHED("gather_keys");
        }
        const int word_bits = bits * min(p.per_word, k - w * p.per_word);
        for (int shift = 0; shift < word_bits; shift += RX_BITS) {
            const int nb = min(RX_BITS, word_bits - shift);
            const uint32_t mask = (1u << nb) - 1u;
            radix_count_kernel<<<(unsigned)p.n_tiles, RX_THREADS, 0, s>>>(kb[cur], n, shift, mask, p.n_tiles, table);
            ETM_LAUNCHED("radix_count");
            const int st = scan_apply((int64_t)(mask + 1u) * p.n_tiles, TableVal{table}, TablePut{table}, ws,
                                      scan_workspace_words(RX_BINS * p.n_tiles), nullptr, s);
            if (st) return st;
            radix_scatter_kernel<<<(unsigned)p.n_tiles, RX_THREADS, RX_SMEM, s>>>(
                kb[cur], pb[cur], n, shift, mask, nb, p.n_tiles, table, kb[cur ^ 1], pb[cur ^ 1]);
            ETM_LAUNCHED("radix_scatter");
            cur ^= 1;
        }
    }
    order_emit_kernel<<<grid, 256, 0, s>>>(p.nw > 1 ? words : kb[cur], n, k, bits, p.per_word, pb[cur],
                                           p.nw > 1 ? counts : nullptr, out_rows, out_counts);
    ETM_LAUNCHED("order_emit");
    return ETM_OK;
}

// One call for the levels of a launch: a small level is two or three launches of a few microseconds each, and the calls,
// allocations and bookkeeping of the caller took 0.15 ms a level.
extern "C" int etm_order_levels(const int32_t* rows, const int32_t* counts, const int64_t* sizes, int32_t n_levels,
                                int32_t k0, const int32_t* perm, int32_t bits, const int32_t* prev_rows, int64_t prev_n,
                                int32_t* out_rows, int32_t* out_counts, int64_t* totals, uint8_t* scratch,
                                int64_t scratch_bytes, void* stream) {
    ETM_REQUIRE(n_levels >= 0 && k0 >= 2 && k0 + n_levels <= MAX_ITEMS + 1 && prev_n >= 0, ETM_EINVAL,
                "etm_order_levels: bad sizes");
    for (int i = 0; i < n_levels; i++) {
        const int k = k0 + i;
        ETM_REQUIRE(sizes[i] >= 0, ETM_EINVAL, "etm_order_levels: negative size");
        if (prev_rows != nullptr) {
            const int st = etm_group_totals(prev_rows, prev_n, k - 1, totals + 2 * i, stream);
            if (st) return st;
        }
        const int st = etm_order_level(rows, counts, sizes[i], k, perm, bits, out_rows, out_counts, scratch,
                                       scratch_bytes, stream);
        if (st) return st;
        prev_rows = out_rows;
        prev_n = sizes[i];
        rows += sizes[i] * k;
        out_rows += sizes[i] * k;
        counts += sizes[i];
        out_counts += sizes[i];
    }
    return ETM_OK;
}

extern "C" int etm_group_totals(const int32_t* rows, int64_t n, int32_t width, int64_t* out, void* stream) {
    ETM_REQUIRE(n >= 0 && width >= 1, ETM_EINVAL, "etm_group_totals: bad sizes");
    cudaStream_t s = as_stream(stream);
    ETM_CUDA(cudaMemsetAsync(out, 0, 2 * sizeof(int64_t), s));
    if (n == 0) return ETM_OK;
    group_totals_kernel<<<grid_of(n, 256), 256, 0, s>>>(rows, n, width, reinterpret_cast<unsigned long long*>(out));
    ETM_LAUNCHED("group_totals");
    return ETM_OK;
}
