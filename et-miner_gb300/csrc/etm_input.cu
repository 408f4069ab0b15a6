// The device input layer: the item coding of a transaction CSR without sorting (a presence bitmap over the
// id span ranks every id; rows are checked to be canonical; a histogram of the ranks gives the supports),
// the lex row order (sort keys that gather the rows sharing their most frequent columns, and the CSR
// permuted into that order), and the tile occupancy (per column one bit per 32-word tile holding a row of
// it, which lets the prefix and per-candidate kernels skip tiles).
//
// HBM-bound integer work: warps over rows / occupancy words, grids a multiple of the SM count.
#include "etm_scan.cuh"

namespace {

using namespace etm;

constexpr int IN_THREADS = 256;

__device__ inline uint64_t warp_or64(uint64_t x) {
    const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)x);
    const unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(x >> 32));
    return ((uint64_t)hi << 32) | lo;
}

// One warp per row. A row holding the column of rank r (ranks by descending support) sets bit 63 - r of its
// high key for r < 64 and bit 127 - r of its low key for 64 <= r < 128 (the key of
// gpu/kernels/_src/csr_to_bitvec.cu:75-104). Both keys are stored with their top bit flipped, so that an
// ascending signed sort orders them as unsigned values.
__global__ void __launch_bounds__(IN_THREADS) row_order_keys_kernel(const int64_t* __restrict__ row_ptr,
                                                                    const int32_t* __restrict__ cols, int64_t n_rows,
                                                                    const int32_t* __restrict__ rank_of_col,
                                                                    int64_t n_cols, int64_t* __restrict__ key_hi,
                                                                    int64_t* __restrict__ key_lo) {
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_rows; r += n_warps) {
        const int64_t e1 = row_ptr[r + 1];
        uint64_t hi = 0, lo = 0;
        for (int64_t e = row_ptr[r] + lane; e < e1; e += 32) {
            const int32_t c = cols[e];
            if (c < 0 || c >= n_cols) continue;
            const int32_t k = rank_of_col[c];
            if (k >= 0 && k < 64) hi |= 1ULL << (63 - k);
            else if (k >= 64 && k < 128) lo |= 1ULL << (127 - k);
        }
        hi = warp_or64(hi);
        lo = warp_or64(lo);
        if (lane == 0) {
            key_hi[r] = (int64_t)(hi ^ (1ULL << 63));
            key_lo[r] = (int64_t)(lo ^ (1ULL << 63));
        }
    }
}

// One warp per output row p: input row order[p]'s entries copied to new_ptr[p] onwards. A row whose source
// index or destination range falls outside the arrays is skipped and reported in *bad.
__global__ void __launch_bounds__(IN_THREADS) permute_rows_kernel(const int64_t* __restrict__ row_ptr,
                                                                  const int32_t* __restrict__ cols, int64_t nnz,
                                                                  const int64_t* __restrict__ order, int64_t n_rows,
                                                                  const int64_t* __restrict__ new_ptr,
                                                                  int32_t* __restrict__ new_cols, int* bad) {
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < n_rows; p += n_warps) {
        const int64_t src = order[p];
        if (src < 0 || src >= n_rows) {
            if (lane == 0) atomicExch(bad, 1);
            continue;
        }
        const int64_t e0 = row_ptr[src], n = row_ptr[src + 1] - e0, d0 = new_ptr[p];
        if (e0 < 0 || n < 0 || e0 + n > nnz || d0 < 0 || d0 + n > nnz) {
            if (lane == 0) atomicExch(bad, 1);
            continue;
        }
        for (int64_t i = lane; i < n; i += 32) new_cols[d0 + i] = cols[e0 + i];
    }
}

// occ[c][ow], bit b: tile t = 64 ow + b of column c (words [32 t, 32 t + 32) below n_words) holds a set bit
// (the occupancy of gpu/kernels/occupancy.py:37-58). One warp per occupancy word, 32 steps of two words per
// lane: lanes 0-15 read tile 2 i of step i, lanes 16-31 tile 2 i + 1; one 16-byte load per lane when every
// column starts 16-byte aligned (VEC), else two 8-byte loads.
template <bool VEC>
__global__ void __launch_bounds__(IN_THREADS) tile_occupancy_kernel(const uint64_t* __restrict__ bv, int64_t n_cols,
                                                                    int64_t n_words, int64_t ld,
                                                                    uint64_t* __restrict__ occ, int64_t occ_ld) {
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t total = n_cols * occ_ld;
    for (int64_t u = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < total; u += n_warps) {
        const int64_t c = u / occ_ld, ow = u - c * occ_ld;
        const uint64_t* col = bv + c * ld;
        const int64_t w0 = ow * (64 * ETM_OCC_TILE_WORDS) + 2 * lane;
        uint64_t bits = 0;
#pragma unroll 8
        for (int i = 0; i < 32; i++) {
            const int64_t w = w0 + 64 * i;
            uint64_t x = 0;
            if (w + 1 < n_words) {
                if (VEC) {
                    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(col + w));
                    x = v.x | v.y;
                } else {
                    x = __ldg(col + w) | __ldg(col + w + 1);
                }
            } else if (w < n_words) {
                x = __ldg(col + w);
            }
            const unsigned b = __ballot_sync(0xffffffffu, x != 0ULL);
            bits |= (uint64_t)((b & 0xFFFFu) != 0u) << (2 * i);
            bits |= (uint64_t)((b >> 16) != 0u) << (2 * i + 1);
        }
        if (lane == 0) occ[u] = bits;
    }
}

// ---- item coding of a transaction CSR: ids to ranks among the distinct ids, without sorting ----

// Bit (id - lo) of the bitmap for every entry with lo <= id < lo + span; an id outside sets *bad. A bit already
// set is not OR-ed again, so a frequent id costs a read, not an atomic. SMEM: the bitmap fits a block's shared memory
// (spans up to PRESENCE_SMEM_WORDS words): it is collected there and merged once. Else the reads go through L1, where a
// stale word costs an OR too many, not a wrong bit. Read through L2, the few sectors of a small vocabulary serialised
// the reads of every SM: 24M entries of 2,000 ids 1.40 -> 0.04 ms.
constexpr int PRESENCE_SMEM_WORDS = 8192;
template <bool SMEM>
__global__ void __launch_bounds__(IN_THREADS) id_presence_kernel(const int64_t* __restrict__ ids, int64_t nnz,
                                                                 int64_t lo, int64_t span, uint32_t* bitmap,
                                                                 int* bad) {
    extern __shared__ uint32_t seen[];
    const int n_w = (int)ceil_div<int64_t>(span, 32);
    if (SMEM) {
        for (int i = threadIdx.x; i < n_w; i += blockDim.x) seen[i] = 0u;
        __syncthreads();
    }
    volatile uint32_t* map = SMEM ? seen : bitmap;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 4
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += stride) {
        const uint64_t v = (uint64_t)ids[e] - (uint64_t)lo;
        if (v >= (uint64_t)span) {
            atomicExch(bad, 1);
            continue;
        }
        const unsigned bit = 1u << (v & 31);
        const unsigned w = SMEM ? map[v >> 5] : *reinterpret_cast<const uint32_t*>(bitmap + (v >> 5));
        if ((w & bit) == 0u) atomicOr((SMEM ? seen : bitmap) + (v >> 5), bit);
    }
    if (SMEM) {
        __syncthreads();
        for (int i = threadIdx.x; i < n_w; i += blockDim.x) {
            const uint32_t x = seen[i];
            if (x != 0u && (__ldcg(bitmap + i) & x) != x) atomicOr(bitmap + i, x);
        }
    }
}

// One block: word_rank[w] = set bits in words [0, w) of the bitmap, word_rank[n] = the distinct ids.
__global__ void __launch_bounds__(1024) bitmap_rank_kernel(const uint32_t* __restrict__ bitmap, int64_t n,
                                                           int64_t* __restrict__ word_rank) {
    int64_t carry = 0;  // the same in every thread
    for (int64_t w0 = 0; w0 < n; w0 += blockDim.x) {
        const int64_t w = w0 + threadIdx.x;
        int64_t total;
        const int64_t ex = block_exclusive_scan(w < n ? __popc(bitmap[w]) : 0, &total);
        if (w < n) word_rank[w] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) word_rank[n] = carry;
}

// Each entry's code, the rank of its id among the distinct ids (word_rank[w] plus the set bits below it in word w), a
// thread per entry; *order is raised by the entries whose id does not exceed the one before, and by those outside.
__global__ void __launch_bounds__(IN_THREADS) code_entries_kernel(const int64_t* __restrict__ ids, int64_t nnz,
                                                                  int64_t lo, int64_t span,
                                                                  const uint32_t* __restrict__ bitmap,
                                                                  const int64_t* __restrict__ word_rank,
                                                                  int32_t* __restrict__ codes, unsigned* order) {
    unsigned down = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 4
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += stride) {
        const int64_t id = ids[e];
        const uint64_t v = (uint64_t)id - (uint64_t)lo;
        int32_t code = -1;
        if (v < (uint64_t)span) code = (int32_t)(word_rank[v >> 5] + __popc(bitmap[v >> 5] & ((1u << (v & 31)) - 1u)));
        codes[e] = code;
        down += (e > 0 && ids[e - 1] >= id ? 1u : 0u) + (code < 0 ? 1u : 0u);
    }
    down = __reduce_add_sync(0xffffffffu, down);
    if ((threadIdx.x & 31) == 0 && down != 0u) atomicAdd(order, down);
}

// *order lowered by the rows that start with an id not above the entry before them. A row whose ids do not strictly
// ascend (unsorted, or with a repeated id) holds such an entry past its start, so *order ends at zero exactly when the
// rows are canonical (fewer than 2^32 entries; more are told apart by no count that matters: the caller sorts then).
__global__ void __launch_bounds__(IN_THREADS) row_starts_kernel(const int64_t* __restrict__ row_ptr,
                                                                const int64_t* __restrict__ ids, int64_t n_rows,
                                                                unsigned* order) {
    unsigned down = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += stride) {
        const int64_t e0 = row_ptr[r], e1 = row_ptr[r + 1];
        down += e0 < e1 && e0 > 0 && ids[e0 - 1] >= ids[e0] ? 1u : 0u;
    }
    down = __reduce_add_sync(0xffffffffu, down);
    if ((threadIdx.x & 31) == 0 && down != 0u) atomicSub(order, down);
}

__global__ void order_status_kernel(int* status) { *status = *status != 0 ? 1 : 0; }

// Each row's codes sorted and without repeats, in place: the places behind the distinct codes hold -1, which every
// reader of codes takes for no entry. Rows of up to 32 entries by a warp, from registers; up to SORT_ROW_MAX by a block,
// in shared memory; a longer row sets *too_long and stays as it is.
constexpr int SORT_ROW_MAX = 2048;
__global__ void __launch_bounds__(IN_THREADS) sort_short_rows_kernel(const int64_t* __restrict__ row_ptr, int64_t n_rows,
                                                                     int32_t* __restrict__ codes) {
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_rows; r += n_warps) {
        const int64_t e0 = row_ptr[r];
        const int len = (int)min64(row_ptr[r + 1] - e0, 33);
        if (len < 2 || len > 32) continue;  // warp-uniform
        uint32_t x = lane < len ? (uint32_t)codes[e0 + lane] : 0xFFFFFFFFu;
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
                const bool up = ((lane & k) == 0) == ((lane & j) == 0);  // keeps the smaller
                x = up ? min(x, y) : max(x, y);
            }
        }
        const uint32_t prev = __shfl_up_sync(0xffffffffu, x, 1);
        const bool keep = x != 0xFFFFFFFFu && (lane == 0 || prev != x);
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        if (keep) codes[e0 + __popc(kept & ((1u << lane) - 1u))] = (int32_t)x;
        if (lane < len && lane >= __popc(kept)) codes[e0 + lane] = -1;
    }
}

__global__ void __launch_bounds__(IN_THREADS) sort_long_rows_kernel(const int64_t* __restrict__ row_ptr, int64_t n_rows,
                                                                    int32_t* __restrict__ codes, int* too_long) {
    __shared__ uint32_t x[SORT_ROW_MAX];
    for (int64_t r = blockIdx.x; r < n_rows; r += gridDim.x) {
        const int64_t e0 = row_ptr[r], n64 = row_ptr[r + 1] - e0;
        if (n64 <= 32) continue;  // block-uniform
        if (n64 > SORT_ROW_MAX) {
            if (threadIdx.x == 0) atomicExch(too_long, 1);
            continue;
        }
        const int len = (int)n64;
        int n = 64;
        while (n < len) n <<= 1;
        for (int i = threadIdx.x; i < n; i += IN_THREADS) x[i] = i < len ? (uint32_t)codes[e0 + i] : 0xFFFFFFFFu;
        __syncthreads();
        for (int k = 2; k <= n; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = threadIdx.x; i < n; i += IN_THREADS) {
                    const int p = i ^ j;
                    if (p > i) {
                        const uint32_t a = x[i], b = x[p];
                        if ((a > b) == ((i & k) == 0)) {
                            x[i] = b;
                            x[p] = a;
                        }
                    }
                }
                __syncthreads();
            }
        }
        int64_t base = 0;
        for (int i0 = 0; i0 < n; i0 += IN_THREADS) {
            const int i = i0 + threadIdx.x;
            const bool keep = i < n && x[i] != 0xFFFFFFFFu && (i == 0 || x[i - 1] != x[i]);
            int64_t total;
            const int64_t at = base + block_exclusive_scan(keep ? 1 : 0, &total);
            if (keep) codes[e0 + at] = (int32_t)x[i];
            base += total;
        }
        for (int i = (int)base + threadIdx.x; i < len; i += IN_THREADS) codes[e0 + i] = -1;
        __syncthreads();  // the next row rewrites x
    }
}

// Block-private counters in shared memory: up to 48 KB by several blocks an SM, up to 216 KB by one block of 1,024
// threads an SM where the entries are many times the counters to merge (1M rows over 50,000 ids 0.38 -> 0.05 ms).
constexpr int HIST_SMEM_BINS = 12288;
constexpr int HIST_WIDE_BINS = 55296;
constexpr int HIST_WIDE_THREADS = 1024;

// Occurrences of each code in [0, n_bins) (others ignored): block-private shared counters when the bins fit,
// added to the global counts once per non-zero bin; global atomics otherwise.
template <bool SMEM>
__global__ void __launch_bounds__(HIST_WIDE_THREADS) code_histogram_kernel(const int32_t* __restrict__ codes, int64_t nnz,
                                                                    int64_t n_bins,
                                                                    unsigned long long* __restrict__ counts) {
    extern __shared__ uint32_t hist[];
    if (SMEM) {
        for (int64_t i = threadIdx.x; i < n_bins; i += blockDim.x) hist[i] = 0u;
        __syncthreads();
    }
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += stride) {
        const int32_t c = codes[e];
        if (c < 0 || c >= n_bins) continue;
        if (SMEM) atomicAdd(hist + c, 1u);
        else atomicAdd(counts + c, 1ULL);
    }
    if (SMEM) {
        __syncthreads();
        for (int64_t i = threadIdx.x; i < n_bins; i += blockDim.x)
            if (hist[i] != 0u) atomicAdd(counts + i, (unsigned long long)hist[i]);
    }
}

// The distinct ids in ascending order: lo + 32 w + b for every set bit b of word w, at out[word_rank[w]] on.
__global__ void __launch_bounds__(IN_THREADS) bitmap_values_kernel(const uint32_t* __restrict__ bitmap, int64_t n,
                                                                   const int64_t* __restrict__ word_rank, int64_t lo,
                                                                   int64_t* __restrict__ out) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n; w += stride) {
        uint32_t x = bitmap[w];
        int64_t at = word_rank[w];
        while (x) {
            const int b = __ffs(x) - 1;
            out[at++] = lo + 32 * w + b;
            x &= x - 1u;
        }
    }
}

// out[0]: the sum over the rows of L (L - 1) / 2, L its entries whose code maps to a column; out[1]: the most entries of a
// row, mapped or not. Eight lanes per row.
__global__ void __launch_bounds__(IN_THREADS) row_pairs_kernel(const int64_t* __restrict__ row_ptr,
                                                               const int32_t* __restrict__ codes, int64_t n_rows,
                                                               const int32_t* __restrict__ lut, int64_t lut_size,
                                                               unsigned long long* __restrict__ out) {
    const int lane = threadIdx.x & 31, sub = lane & 7;
    const unsigned mask = 0xFFu << (lane & 24);
    const int64_t n_subs = ((int64_t)gridDim.x * blockDim.x) >> 3;
    unsigned long long sum = 0, longest = 0;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3; r < n_rows; r += n_subs) {
        const int64_t e0 = row_ptr[r], e1 = row_ptr[r + 1];
        longest = max(longest, (unsigned long long)(e1 - e0));
        unsigned n = 0;
        for (int64_t e = e0 + sub; e < e1; e += 8) {
            const int32_t c = codes[e];
            n += (c >= 0 && c < lut_size && __ldg(lut + c) >= 0) ? 1u : 0u;
        }
        n = __reduce_add_sync(mask, n);
        if (sub == 0 && n > 1u) sum += (unsigned long long)n * (n - 1u) / 2u;
    }
    for (int d = 16; d > 0; d >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, d);
        longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, d));
    }
    if (lane == 0 && sum != 0ULL) atomicAdd(out, sum);
    if (lane == 0 && longest != 0ULL) atomicMax(out + 1, longest);
}

// out[0]: the largest of the ids with their sign bit flipped, as unsigned; out[1]: the largest of those values inverted.
__global__ void __launch_bounds__(IN_THREADS) id_range_kernel(const int64_t* __restrict__ ids, int64_t n,
                                                              unsigned long long* __restrict__ out) {
    unsigned long long hi = 0, lo = 0;
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long u = (unsigned long long)__ldg(reinterpret_cast<const long long*>(ids) + i) ^ (1ULL << 63);
        hi = max(hi, u);
        lo = max(lo, ~u);
    }
    for (int d = 16; d > 0; d >>= 1) {
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
        lo = max(lo, __shfl_xor_sync(0xffffffffu, lo, d));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out, hi);
        atomicMax(out + 1, lo);
    }
}

struct FrequentCode {
    const int64_t* counts;
    int64_t min_count;
    int32_t* col_of;
    __device__ int64_t operator()(int64_t i) const {
        const bool keep = counts[i] >= min_count;
        if (!keep) col_of[i] = -1;
        return keep ? 1 : 0;
    }
};
struct PutColumn {
    int32_t* col_of;
    __device__ void operator()(int64_t i, int64_t off) const { col_of[i] = (int32_t)off; }
};

// One warp per row: its entries whose code maps to a column (0 <= code < lut_size and lut[code] >= 0).
__global__ void __launch_bounds__(IN_THREADS) kept_lengths_kernel(const int64_t* __restrict__ row_ptr,
                                                                  const int32_t* __restrict__ codes, int64_t n_rows,
                                                                  const int32_t* __restrict__ lut, int64_t lut_size,
                                                                  int64_t* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_rows; r += n_warps) {
        unsigned n = 0;
        for (int64_t e = row_ptr[r] + lane; e < row_ptr[r + 1]; e += 32) {
            const int32_t c = codes[e];
            n += (c >= 0 && c < lut_size && lut[c] >= 0) ? 1u : 0u;
        }
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) out[r] = n;
    }
}

int in_grid(int64_t units_of_warps) {
    const int64_t cap = (int64_t)max(1, sm_count()) * 8;
    return (int)max64(1, min64(cap, ceil_div<int64_t>(units_of_warps, IN_THREADS / 32)));
}

// Grid of a pass with a thread per element, four elements a thread or more.
int wide_grid(int64_t n) {
    return (int)max64(1, min64((int64_t)max(1, sm_count()) * 8, ceil_div<int64_t>(n, 4 * IN_THREADS)));
}

}  // namespace

extern "C" int etm_row_order_keys(const int64_t* row_ptr, const int32_t* cols, int64_t n_rows,
                                  const int32_t* rank_of_col, int64_t n_cols, int64_t* key_hi, int64_t* key_lo,
                                  void* stream) {
    ETM_REQUIRE(n_rows >= 0 && n_cols >= 0, ETM_EINVAL, "etm_row_order_keys: negative size");
    if (n_rows == 0) return ETM_OK;
    row_order_keys_kernel<<<in_grid(n_rows), IN_THREADS, 0, as_stream(stream)>>>(row_ptr, cols, n_rows, rank_of_col,
                                                                                 n_cols, key_hi, key_lo);
    ETM_LAUNCHED("row_order_keys");
    return ETM_OK;
}

extern "C" int etm_permute_rows(const int64_t* row_ptr, const int32_t* cols, int64_t nnz, const int64_t* order,
                                int64_t n_rows, const int64_t* new_row_ptr, int32_t* new_cols, int32_t* status,
                                void* stream) {
    ETM_REQUIRE(n_rows >= 0 && nnz >= 0, ETM_EINVAL, "etm_permute_rows: negative size");
    ETM_REQUIRE(status != nullptr, ETM_EINVAL, "etm_permute_rows: status is required");
    cudaStream_t s = as_stream(stream);
    ETM_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), s));
    if (n_rows == 0) return ETM_OK;
    permute_rows_kernel<<<in_grid(n_rows), IN_THREADS, 0, s>>>(row_ptr, cols, nnz, order, n_rows, new_row_ptr,
                                                               new_cols, reinterpret_cast<int*>(status));
    ETM_LAUNCHED("permute_rows");
    return ETM_OK;
}

extern "C" int etm_tile_occupancy(const uint64_t* bv, int64_t n_cols, int64_t n_words, int64_t ld, uint64_t* occ,
                                  int64_t occ_ld, void* stream) {
    ETM_REQUIRE(n_cols >= 0 && n_words >= 0 && ld >= n_words, ETM_EINVAL, "etm_tile_occupancy: bad sizes");
    ETM_REQUIRE((reinterpret_cast<uintptr_t>(bv) & 7) == 0, ETM_EINVAL, "etm_tile_occupancy: bv must be 8-byte aligned");
    const int64_t tiles = ceil_div<int64_t>(n_words, ETM_OCC_TILE_WORDS);
    ETM_REQUIRE(occ_ld >= ceil_div<int64_t>(tiles, 64) && occ_ld >= 1, ETM_EINVAL,
                "etm_tile_occupancy: occ_ld %lld < ceil(tiles / 64)", (long long)occ_ld);
    if (n_cols == 0) return ETM_OK;
    const int grid = in_grid(n_cols * occ_ld);
    if (ld % 2 == 0 && (reinterpret_cast<uintptr_t>(bv) & 15) == 0)
        tile_occupancy_kernel<true><<<grid, IN_THREADS, 0, as_stream(stream)>>>(bv, n_cols, n_words, ld, occ, occ_ld);
    else
        tile_occupancy_kernel<false><<<grid, IN_THREADS, 0, as_stream(stream)>>>(bv, n_cols, n_words, ld, occ, occ_ld);
    ETM_LAUNCHED("tile_occupancy");
    return ETM_OK;
}

extern "C" int etm_item_codes(const int64_t* row_ptr, const int64_t* ids, int64_t nnz, int64_t n_rows, int64_t lo,
                              int64_t span, uint32_t* bitmap, int64_t* word_rank, int32_t* codes, int32_t* status,
                              void* stream) {
    ETM_REQUIRE(nnz >= 0 && n_rows >= 0 && span >= 1 && span <= ETM_CODE_SPAN_MAX, ETM_EINVAL,
                "etm_item_codes: span %lld outside [1, 2^26] or negative size", (long long)span);
    ETM_REQUIRE(status != nullptr, ETM_EINVAL, "etm_item_codes: status is required");
    cudaStream_t s = as_stream(stream);
    const int64_t n_w = ceil_div<int64_t>(span, 32);
    ETM_CUDA(cudaMemsetAsync(status, 0, 2 * sizeof(int32_t), s));
    ETM_CUDA(cudaMemsetAsync(bitmap, 0, (size_t)n_w * 4, s));
    int* st = reinterpret_cast<int*>(status);
    unsigned* order = reinterpret_cast<unsigned*>(st + 1);
    if (nnz > 0) {
        const int blocks = (int)max64(1, min64((int64_t)max(1, sm_count()) * 8, ceil_div<int64_t>(nnz, 4 * IN_THREADS)));
        if (n_w <= PRESENCE_SMEM_WORDS)
            id_presence_kernel<true><<<blocks, IN_THREADS, (size_t)n_w * 4, s>>>(ids, nnz, lo, span, bitmap, st);
        else
            id_presence_kernel<false><<<blocks, IN_THREADS, 0, s>>>(ids, nnz, lo, span, bitmap, st);
        ETM_LAUNCHED("id_presence");
    }
    bitmap_rank_kernel<<<1, 1024, 0, s>>>(bitmap, n_w, word_rank);
    ETM_LAUNCHED("bitmap_rank");
    if (nnz > 0) {
        code_entries_kernel<<<wide_grid(nnz), IN_THREADS, 0, s>>>(ids, nnz, lo, span, bitmap, word_rank, codes, order);
        ETM_LAUNCHED("code_entries");
    }
    if (n_rows > 0) {
        row_starts_kernel<<<wide_grid(n_rows), IN_THREADS, 0, s>>>(row_ptr, ids, n_rows, order);
        ETM_LAUNCHED("row_starts");
    }
    order_status_kernel<<<1, 1, 0, s>>>(st + 1);
    ETM_LAUNCHED("order_status");
    return ETM_OK;
}

extern "C" int etm_sort_rows(const int64_t* row_ptr, int64_t n_rows, int32_t* codes, int32_t* status, void* stream) {
    ETM_REQUIRE(n_rows >= 0, ETM_EINVAL, "etm_sort_rows: negative size");
    ETM_REQUIRE(status != nullptr, ETM_EINVAL, "etm_sort_rows: status is required");
    cudaStream_t s = as_stream(stream);
    ETM_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), s));
    if (n_rows == 0) return ETM_OK;
    sort_short_rows_kernel<<<in_grid(n_rows), IN_THREADS, 0, s>>>(row_ptr, n_rows, codes);
    ETM_LAUNCHED("sort_short_rows");
    sort_long_rows_kernel<<<(int)min64(n_rows, (int64_t)max(1, sm_count()) * 8), IN_THREADS, 0, s>>>(
        row_ptr, n_rows, codes, reinterpret_cast<int*>(status));
    ETM_LAUNCHED("sort_long_rows");
    return ETM_OK;
}

extern "C" int etm_row_pairs(const int64_t* row_ptr, const int32_t* codes, int64_t n_rows, const int32_t* lut,
                             int64_t lut_size, int64_t* out, void* stream) {
    ETM_REQUIRE(n_rows >= 0 && lut_size >= 0, ETM_EINVAL, "etm_row_pairs: negative size");
    cudaStream_t s = as_stream(stream);
    ETM_CUDA(cudaMemsetAsync(out, 0, 2 * sizeof(int64_t), s));
    if (n_rows == 0) return ETM_OK;
    row_pairs_kernel<<<in_grid(ceil_div<int64_t>(n_rows, 4)), IN_THREADS, 0, s>>>(
        row_ptr, codes, n_rows, lut, lut_size, reinterpret_cast<unsigned long long*>(out));
    ETM_LAUNCHED("row_pairs");
    return ETM_OK;
}

// The bounds of the ids and the columns of the codes in a launch or three of their own: as array operations (minimum and
// maximum, stack; compare, widen, scan, subtract, invert, place) they were fourteen launches and three waits, 0.3 ms of
// the 1.2 ms call over 60,000 transactions.
extern "C" int etm_id_range(const int64_t* ids, int64_t n, int64_t* out, void* stream) {
    ETM_REQUIRE(n >= 0, ETM_EINVAL, "etm_id_range: negative size");
    cudaStream_t s = as_stream(stream);
    ETM_CUDA(cudaMemsetAsync(out, 0, 2 * sizeof(int64_t), s));
    if (n == 0) return ETM_OK;
    const int grid = (int)max64(1, min64((int64_t)max(1, sm_count()) * 8, ceil_div<int64_t>(n, 4 * IN_THREADS)));
    id_range_kernel<<<grid, IN_THREADS, 0, s>>>(ids, n, reinterpret_cast<unsigned long long*>(out));
    ETM_LAUNCHED("id_range");
    return ETM_OK;
}

extern "C" int etm_code_columns(const int64_t* counts, int64_t n, int64_t min_count, int32_t* col_of, int64_t* ws,
                                int64_t ws_words, void* stream) {
    ETM_REQUIRE(n >= 0 && n < (1LL << 31), ETM_EINVAL, "etm_code_columns: bad size");
    if (n == 0) return ETM_OK;
    return scan_apply(n, FrequentCode{counts, min_count, col_of}, PutColumn{col_of}, ws, ws_words, nullptr,
                      as_stream(stream));
}

extern "C" int etm_code_histogram(const int32_t* codes, int64_t nnz, int64_t n_bins, int64_t* counts, void* stream) {
    ETM_REQUIRE(nnz >= 0 && n_bins >= 0, ETM_EINVAL, "etm_code_histogram: negative size");
    cudaStream_t s = as_stream(stream);
    if (n_bins == 0) return ETM_OK;
    ETM_CUDA(cudaMemsetAsync(counts, 0, (size_t)n_bins * 8, s));
    if (nnz == 0) return ETM_OK;
    auto* out = reinterpret_cast<unsigned long long*>(counts);
    const int grid = (int)max64(1, min64((int64_t)max(1, sm_count()) * 4, ceil_div<int64_t>(nnz, IN_THREADS)));
    if (n_bins <= HIST_SMEM_BINS) {
        code_histogram_kernel<true><<<grid, IN_THREADS, (size_t)n_bins * 4, s>>>(codes, nnz, n_bins, out);
    } else if (n_bins <= HIST_WIDE_BINS && nnz >= n_bins * (int64_t)max(1, sm_count())) {
        ETM_CUDA(cudaFuncSetAttribute(code_histogram_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      HIST_WIDE_BINS * 4));
        code_histogram_kernel<true><<<max(1, sm_count()), HIST_WIDE_THREADS, (size_t)n_bins * 4, s>>>(codes, nnz, n_bins,
                                                                                                      out);
    } else {
        code_histogram_kernel<false><<<grid, IN_THREADS, 0, s>>>(codes, nnz, n_bins, out);
    }
    ETM_LAUNCHED("code_histogram");
    return ETM_OK;
}

extern "C" int etm_bitmap_values(const uint32_t* bitmap, int64_t span, const int64_t* word_rank, int64_t lo,
                                 int64_t* out, void* stream) {
    ETM_REQUIRE(span >= 1 && span <= ETM_CODE_SPAN_MAX, ETM_EINVAL, "etm_bitmap_values: span out of range");
    const int64_t n_w = ceil_div<int64_t>(span, 32);
    bitmap_values_kernel<<<(int)min64((int64_t)max(1, sm_count()) * 8, ceil_div<int64_t>(n_w, IN_THREADS)), IN_THREADS,
                           0, as_stream(stream)>>>(bitmap, n_w, word_rank, lo, out);
    ETM_LAUNCHED("bitmap_values");
    return ETM_OK;
}

extern "C" int etm_kept_lengths(const int64_t* row_ptr, const int32_t* codes, int64_t n_rows, const int32_t* lut,
                                int64_t lut_size, int64_t* out_lengths, void* stream) {
    ETM_REQUIRE(n_rows >= 0 && lut_size >= 0, ETM_EINVAL, "etm_kept_lengths: negative size");
    if (n_rows == 0) return ETM_OK;
    kept_lengths_kernel<<<in_grid(n_rows), IN_THREADS, 0, as_stream(stream)>>>(row_ptr, codes, n_rows, lut, lut_size,
                                                                              out_lengths);
    ETM_LAUNCHED("kept_lengths");
    return ETM_OK;
}
