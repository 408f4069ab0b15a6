// The result frame's arrays from a level: item ids, offsets and supports, where the result's other levels leave off.
#include "etm_common.cuh"

namespace {

using namespace etm;

constexpr int FR_THREADS = 256;

// What bounds it is the writes, 8 (k + 2) bytes an itemset. One pass over the level where the array operations it takes
// the place of (widen the rows, look the ids up, widen and divide the counts, count the offsets up, concatenate) wrote
// each of these two or three times and took nine launches a level: 164,130 itemsets of eleven levels 1.29 -> 0.34 ms with the copy
// back, 1.1M itemsets of four 0.90 -> 0.52.
__global__ void __launch_bounds__(FR_THREADS) frame_level_kernel(
    const int32_t* __restrict__ rows, const int32_t* __restrict__ counts, int64_t n, int k,
    const int64_t* __restrict__ table, double n_rows, int64_t row0, int64_t value0, int64_t* __restrict__ values,
    int64_t* __restrict__ offsets, double* __restrict__ support) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t0 == 0 && row0 == 0) offsets[0] = 0;
    for (int64_t e = t0; e < n * k; e += step) {
        values[value0 + e] = __ldg(table + (rows == nullptr ? e : (int64_t)rows[e]));
        if (e < n) {
            offsets[row0 + e + 1] = value0 + (e + 1) * k;
            support[row0 + e] = (double)counts[e] / n_rows;
        }
    }
}

}  // namespace

extern "C" int etm_frame_level(const int32_t* rows, const int32_t* counts, int64_t n, int32_t k, const int64_t* table,
                               int64_t n_rows, int64_t row0, int64_t value0, int64_t* values, int64_t* offsets,
                               double* support, void* stream) {
    ETM_REQUIRE(n >= 0 && k >= 1 && n_rows >= 1 && row0 >= 0 && value0 >= 0, ETM_EINVAL, "etm_frame_level: bad sizes");
    if (n == 0) return ETM_OK;
    ETM_REQUIRE(rows != nullptr || k == 1, ETM_EINVAL, "etm_frame_level: only single items come without rows");
    const int64_t grid = max64(1, min64((int64_t)max(1, sm_count()) * 16, ceil_div<int64_t>(n * k, FR_THREADS)));
    frame_level_kernel<<<(unsigned)grid, FR_THREADS, 0, as_stream(stream)>>>(rows, counts, n, k, table, (double)n_rows,
                                                                             row0, value0, values, offsets, support);
    ETM_LAUNCHED("frame_level");
    return ETM_OK;
}
