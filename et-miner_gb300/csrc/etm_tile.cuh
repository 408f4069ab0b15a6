// Pair counts of a tile of a prefix group's members by one warp, each column read once.
#pragma once

#include "etm_common.cuh"

namespace etm {

constexpr int GB = 8;  // members per tile side

struct GroupTile {
    const uint64_t* fbv;
    int64_t v0, v1;           // vectors (16 or 8 bytes) of the slab
    const int64_t* off_pre;   // shared: word offsets of the prefix columns,
    const int64_t* off_a;     // of block a's members
    const int64_t* off_b;     // and of block b's (block a's again for a triangle); past the group: a member again
    int plen;
};

__device__ __forceinline__ ulonglong2 bits_and(const ulonglong2& x, const ulonglong2& y) {
    return make_ulonglong2(x.x & y.x, x.y & y.y);
}
__device__ __forceinline__ uint64_t bits_and(uint64_t x, uint64_t y) { return x & y; }
__device__ __forceinline__ int bits_set(const ulonglong2& x) { return __popcll(x.x) + __popcll(x.y); }
__device__ __forceinline__ int bits_set(uint64_t x) { return __popcll(x); }
template <class V>
__device__ __forceinline__ V bits_all();
template <>
__device__ __forceinline__ ulonglong2 bits_all<ulonglong2>() { return make_ulonglong2(~0ULL, ~0ULL); }
template <>
__device__ __forceinline__ uint64_t bits_all<uint64_t>() { return ~0ULL; }
// RO: the words are not written by this launch.
template <bool RO, class V>
__device__ __forceinline__ V load_bits(const V* p) { return RO ? __ldg(p) : *p; }

// Counts the pairs of NA x NB members (TRI: a < b of NA members) over the slab; lane (p % 32) gets pair p's count in
// res[p / 32], pairs in a-major order. V: ulonglong2 where every column starts 16-byte aligned, else uint64_t.
template <class V, bool RO, int NA, int NB, bool TRI>
__device__ __forceinline__ void count_tile(const GroupTile& t, int lane, unsigned* res) {
    constexpr int NP = TRI ? NA * (NA - 1) / 2 : NA * NB;
    unsigned acc[NP];
#pragma unroll
    for (int p = 0; p < NP; p++) acc[p] = 0;
    auto at = [&](int64_t off, int64_t v) { return load_bits<RO>(reinterpret_cast<const V*>(t.fbv + off) + v); };
    for (int64_t v = t.v0 + lane; v < t.v1; v += 32) {
        V a[NA];
#pragma unroll
        for (int i = 0; i < NA; i++) a[i] = at(t.off_a[i], v);
        V m = bits_all<V>();
        for (int q = 0; q < t.plen; q++) m = bits_and(m, at(t.off_pre[q], v));
#pragma unroll
        for (int i = 0; i < NA; i++) a[i] = bits_and(a[i], m);
        if (TRI) {
            int p = 0;
#pragma unroll
            for (int i = 0; i < NA; i++) {
#pragma unroll
                for (int j = i + 1; j < NA; j++) acc[p++] += bits_set(bits_and(a[i], a[j]));
            }
        } else {
            // Block b in parts of BP members: all of it at a time, beside 64 sums, would not fit the registers.
            constexpr int BP = NB < 4 ? NB : 4;
#pragma unroll
            for (int j0 = 0; j0 < NB; j0 += BP) {
                V b[BP];
#pragma unroll
                for (int j = 0; j < BP; j++) b[j] = at(t.off_b[j0 + j], v);
#pragma unroll
                for (int i = 0; i < NA; i++) {
#pragma unroll
                    for (int j = 0; j < BP; j++) acc[i * NB + j0 + j] += bits_set(bits_and(a[i], b[j]));
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const unsigned s = __reduce_add_sync(0xffffffffu, acc[p]);
        if ((p & 31) == lane) res[p >> 5] = s;
    }
}

// The smallest counted shape that covers a tile of na x nb members (tri: the pairs of na members).
__device__ __forceinline__ void tile_shape(bool tri, int na, int nb, int* ta, int* tb) {
    *ta = tri ? (na <= 2 ? 2 : na <= 4 ? na : na <= 6 ? 6 : GB) : GB;
    *tb = tri ? *ta : (nb <= 2 ? 2 : nb <= 4 ? 4 : GB);
}

// Counts a tile of a shape that tile_shape gave.
template <class V, bool RO>
__device__ __forceinline__ void count_shape(const GroupTile& t, int lane, bool tri, int ta, int tb, unsigned* res) {
    if (tri) {
        if (ta == 2) count_tile<V, RO, 2, 2, true>(t, lane, res);
        else if (ta == 3) count_tile<V, RO, 3, 3, true>(t, lane, res);
        else if (ta == 4) count_tile<V, RO, 4, 4, true>(t, lane, res);
        else if (ta == 6) count_tile<V, RO, 6, 6, true>(t, lane, res);
        else count_tile<V, RO, 8, 8, true>(t, lane, res);
    } else {
        if (tb == 2) count_tile<V, RO, GB, 2, false>(t, lane, res);
        else if (tb == 4) count_tile<V, RO, GB, 4, false>(t, lane, res);
        else count_tile<V, RO, GB, 8, false>(t, lane, res);
    }
}

// Calls emit(a, b, count) for every pair of a counted tile, on the lane that holds it.
template <class Emit>
__device__ __forceinline__ void emit_tile(int lane, bool tri, int ta, int tb, int na, int nb, const unsigned* res,
                                          Emit emit) {
    const int np = tri ? ta * (ta - 1) / 2 : ta * tb;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int p = lane + 32 * h;
        if (p >= np) continue;
        int a, b;
        if (tri) {
            int r = p;
            a = 0;
            while (r >= ta - 1 - a) r -= ta - 1 - a++;
            b = a + 1 + r;
        } else {
            a = p / tb;
            b = p - a * tb;
        }
        if (a < na && b < nb) emit(a, b, (int32_t)res[h]);
    }
}

// Counts a tile of na x nb members (tri: the pairs of the na members) with the smallest shape that covers it and calls
// emit(a, b, count) for every pair, on the lane that holds it.
template <class V, class Emit>
__device__ __forceinline__ void count_any_tile(const GroupTile& t, int lane, bool tri, int na, int nb, Emit emit) {
    unsigned res[2] = {0u, 0u};
    int ta, tb;
    tile_shape(tri, na, nb, &ta, &tb);
    count_shape<V, true>(t, lane, tri, ta, tb, res);
    emit_tile(lane, tri, ta, tb, na, nb, res, emit);
}

}  // namespace etm
