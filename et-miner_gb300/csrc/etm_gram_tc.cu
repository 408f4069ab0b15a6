// Exact 0/1 Gram of prefix-group suffixes on the tcgen05 tensor cores.
//
// For a group whose members are bit rows x_0..x_{m-1} (projected suffix
// words, or for K=2 the frequent columns themselves), the pair counts are
// C[i][j] = popcount(x_i & x_j) = sum_r x_i[r] * x_j[r]: the Gram matrix X X^T
// of a 0/1 matrix. One persistent kernel (one CTA per SM) computes it by
// block pairs: the members are cut into blocks of T, and a CTA takes a whole
// block pair (ua <= ub) at a time. As follows for any operand format and
// row-major or blocked member rows (gram_kernel); packed e2m1 over blocked
// rows has a kernel of its own (gram_blocked_kernel, below).
//
//   producers  512 threads, one operand row each (thread t < 256: row t of
//              block ua, else row t - 256 of block ub): per stage they load
//              the row's next bits (prefetched PF stages ahead into
//              registers), expand them into 128 bytes of operand elements
//              in the 128-byte swizzled K-major layout the MMA reads
//              (SWIZZLE_128B), then fence.proxy.async and an mbarrier
//              arrive. A diagonal block pair stages only the B rows and
//              reads A from them.
//   MMA        one thread issues, per 32-byte K step, two M = 128 MMAs that
//              share the B tile (A halves: the first and last T/2 rows of
//              block ua) into two f32 accumulators in tensor memory;
//              tcgen05.commit frees each stage and finally signals the
//              epilogue.
//   epilogue   the producer warps read the accumulators back with
//              tcgen05.ld and emit the i < j pair counts at their
//              lexicographic candidate slots: every count (dense), or only
//              the counts reaching min_count plus a survivor bit each
//              (fused threshold).
//
// Operand formats (the element a set bit becomes, and what a product is):
//
//   FMT 1  e4m3 under kind::f8f6f4, T = 256, 128 bits per stage row:
//          0x01 = 2^-9, products 2^-18.
//   FMT 2  f16 under kind::f16, T = 256, 64 bits per stage row:
//          0x0001 = 2^-24, products 2^-48.
//   FMT 4  packed e2m1 under kind::mxf4 (block scale 2X, every ue8m0 scale
//          factor 127 = 1.0), T = 240, 256 bits per stage row: 0b0001 =
//          0.5, products 0.25. The two 240-column accumulators take TMEM
//          columns 0-479 and the scale factors 480-511, so a block holds
//          240 members (each A half 120 rows of a 128-row MMA; rows 120-127
//          are not read back).
//
// Exactness: every product is one power of two s and every partial sum is
// c * s with an integer c below 2^24 (the caller sends only groups of at
// most 2^24 rows here): exact in f32, and scaled back exactly to c.
//
// Bit expansion: the order of the transactions along K does not change a
// Gram entry, as long as every row uses the same order. So a 32-bit piece v
// of a row is spread by shifts: word q of an output chunk is (v >> q) & M
// with M = 0x11111111 (e2m1 nibbles), 0x01010101 (e4m3 bytes) or
// 0x00010001 (f16 halves); two operations per output word, the same
// permutation in every row.
//
// Every mbarrier wait is bounded in time (%globaltimer): after the limit the
// block raises an abort flag, every thread leaves its loop, the MMA thread
// waits (bounded) for its issued MMAs, TMEM is freed, and the kernel records
// ETM_ETIMEOUT in its status word instead of hanging.
#include <cstdlib>
#include <mutex>

#include "etm_count.cuh"

namespace {

using namespace etm;

constexpr int PRODUCERS = 512;                 // thread t < 256: A row t; else B row t - 256
constexpr int THREADS = PRODUCERS + 32;
constexpr int MMA_WARP = PRODUCERS / 32;
constexpr int STAGES = 3;
constexpr int HALF_BYTES = 128 * 128;          // one 128-row operand tile of 128-byte rows
constexpr int SLOT_BYTES = 4 * HALF_BYTES;     // A (two 128-row halves), then B (256 rows)
constexpr int SMEM_BYTES = STAGES * SLOT_BYTES + 1024;
// Packed e2m1 over blocked rows: operand slots of 240 A rows and 240 B rows of 128 bytes, each followed by eight more
// rows (the first of them ones); three of them in flight.
constexpr int BK_OPS = 3;
constexpr int BK_TILE = 248 * 128;
constexpr int BK_SLOT = 2 * BK_TILE;            // A rows, then B rows
constexpr int BK_AHEAD = 4;                     // stages whose raw words a producer holds in registers
constexpr int BK_PRODUCERS = 480;               // thread t < 240: A row t; else B row t - 240
constexpr int BK_THREADS = BK_PRODUCERS + 32;   // and the MMA warp: 16 warps of 128 registers a thread
constexpr int BK_MMA_WARP = BK_PRODUCERS / 32;
constexpr int BK_SMEM = BK_OPS * BK_SLOT + 1024;
static_assert(BK_SMEM <= 227 * 1024 - 8192 && BK_TILE % 1024 == 0, "operand slots");
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t SF_COL = 480;               // FMT 4: scale factors in TMEM columns 480-511
constexpr uint64_t WAIT_NS = 2000000000ull;    // every bounded wait: 2 s

template <int FMT>
struct Fmt;
template <>
struct Fmt<1> {  // e4m3
    static constexpr int T = 256, WORDS = 2, PF = 4;
    static constexpr float SCALE = 262144.0f;  // 2^18
};
template <>
struct Fmt<2> {  // f16
    static constexpr int T = 256, WORDS = 1, PF = 4;
    static constexpr float SCALE = 281474976710656.0f;  // 2^48
};
template <>
struct Fmt<4> {  // e2m1, block-scaled with unit scales
    static constexpr int T = 240, WORDS = 4, PF = 2;
    static constexpr float SCALE = 4.0f;
};

__device__ int g_tc_status;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// try_wait suspends the thread in hardware until the phase completes or a short time-out passes.
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for the phase of `parity` to complete; false if the block aborts or `limit_ns` passes first
// (then the abort flag is raised). A limit of 0 gives up at once: the give-up path's test hook.
__device__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint64_t limit_ns) {
    if (limit_ns == 0) {
        *abort_flag = 1;
        return false;
    }
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = now_ns();
    while (!mbar_try(bar, parity)) {
        if (*abort_flag) return false;
        if (now_ns() - t0 > limit_ns) {
            *abort_flag = 1;
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, SWIZZLE_128B, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;                  // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;        // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1 << 46;                  // descriptor version for tcgen05
    d |= (uint64_t)2 << 61;                  // SWIZZLE_128B
    return d;
}

// Instruction descriptor, M = 128, N = T, both operands K-major.
//   FMT 1, 2: D f32 (bits 4-5 = 1), A/B format 0 (e4m3 under kind::f8f6f4, f16 under kind::f16).
//   FMT 4 (block-scaled): A/B format 1 (e2m1 under kind::mxf4) in bits 7-9 / 10-12, scale factors ue8m0
//   (bit 23), scale-factor ids 0 (bits 4-5, 29-30).
template <int FMT>
__host__ __device__ constexpr uint32_t instr_desc() {
    constexpr uint32_t n_m = ((uint32_t)(Fmt<FMT>::T >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    if constexpr (FMT == 4) return n_m | (1u << 7) | (1u << 10) | (1u << 23);
    else return n_m | (1u << 4);
}

// D (TMEM) += A x B, both from shared-memory descriptors.
template <int FMT>
__device__ __forceinline__ void mma_ss(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t acc, uint32_t tmem_sf) {
    if constexpr (FMT == 2) {
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
            "l"(a), "l"(b), "r"(instr_desc<FMT>()), "r"(acc));
    } else if constexpr (FMT == 1) {
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
            "l"(a), "l"(b), "r"(instr_desc<FMT>()), "r"(acc));
    } else {
        // Scale factors of A at tmem_sf, of B 16 columns on; every byte of those columns is 127 (2^0).
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%6], p;\n}\n" ::"r"(
                tmem_d),
            "l"(a), "l"(b), "r"(instr_desc<FMT>()), "r"(acc), "r"(tmem_sf), "r"(tmem_sf + 16));
    }
}

// The packed e2m1 MMA with a run-time instruction descriptor (its N).
__device__ __forceinline__ void mma_mxf4(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc,
                                         uint32_t tmem_sf) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%6], p;\n}\n" ::"r"(
            tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(tmem_sf), "r"(tmem_sf + 16));
}

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// One operand row of the stage: Fmt::WORDS words of the row's bits, expanded into the eight 16-byte
// chunks of row r of a SWIZZLE_128B tile (logical chunk c lives at chunk c ^ (r % 8)).
template <int FMT>
__device__ __forceinline__ void store_row(uint8_t* tile, int r, const uint64_t* x) {
    uint8_t* row = tile + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        uint32_t v, mask;
        int q0;
        if constexpr (FMT == 4) {  // chunk c: the 32 bits of piece c as 32 nibbles
            v = (uint32_t)(x[c >> 1] >> (32 * (c & 1)));
            q0 = 0;
            mask = 0x11111111u;
        } else if constexpr (FMT == 1) {  // chunks 2p, 2p + 1: the 32 bits of piece p as 32 bytes
            v = (uint32_t)(x[c >> 2] >> (32 * ((c >> 1) & 1)));
            q0 = 4 * (c & 1);
            mask = 0x01010101u;
        } else {  // chunks 4p .. 4p + 3: the 32 bits of piece p as 32 halves
            v = (uint32_t)(x[0] >> (32 * (c >> 2)));
            q0 = 4 * (c & 3);
            mask = 0x00010001u;
        }
        const uint4 o = make_uint4((v >> q0) & mask, (v >> (q0 + 1)) & mask, (v >> (q0 + 2)) & mask,
                                   (v >> (q0 + 3)) & mask);
        *reinterpret_cast<uint4*>(row + ((c ^ (r & 7)) << 4)) = o;
    }
}

template <int FMT>
__global__ void __launch_bounds__(THREADS, 1) gram_kernel(
    const uint64_t* __restrict__ src, const int64_t* __restrict__ cbase, const int64_t* __restrict__ cwords,
    const int64_t* __restrict__ cld, const int32_t* __restrict__ grp_size, const int64_t* __restrict__ cand_off,
    const int64_t* __restrict__ work_groups, const int64_t* __restrict__ work_off, int64_t n_work, int64_t chunk_base,
    const uint8_t* __restrict__ cls, int32_t min_count, int32_t* __restrict__ out, uint32_t* __restrict__ surv,
    unsigned long long* __restrict__ work_counter, uint64_t first_wait_ns, bool blocked) {
    constexpr int T = Fmt<FMT>::T;
    constexpr int TH = T / 2;  // A rows per accumulator
    constexpr int WORDS = Fmt<FMT>::WORDS;
    constexpr int PF = Fmt<FMT>::PF;
    constexpr int BW = PF * WORDS;
    constexpr int NST = STAGES;  // operand stages
    extern __shared__ uint8_t dsmem[];
    __shared__ __align__(8) uint64_t full_bar[NST];
    __shared__ __align__(8) uint64_t empty_bar[NST];
    __shared__ __align__(8) uint64_t acc_bar;
    __shared__ __align__(8) uint64_t drain_bar;
    __shared__ uint32_t tmem_sh;
    __shared__ int abort_sh;
    // Member row offsets of the block pair.
    __shared__ int64_t off_a[256];
    __shared__ int64_t off_b[256];
    __shared__ int64_t next_sh;

    uint8_t* slots = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dsmem) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int s = 0; s < NST; s++) {
            mbar_init(&full_bar[s], PRODUCERS);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_bar, 1);
        mbar_init(&drain_bar, 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_sh;
    volatile int* abort_flag = &abort_sh;
    if constexpr (FMT == 4) {
        // Unit scale factors: warp w (w < 4) fills lanes 32 w .. 32 w + 31 of columns 480-511 with 127s.
        if (warp < 4) {
            const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + SF_COL;
            const uint32_t u = 0x7F7F7F7Fu;
            asm volatile(
                "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
                "%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
                "r"(u)
                : "memory");
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }

    const int64_t total = work_off[n_work];
    int64_t gstage = 0;
    uint32_t tile_iter = 0;
    // Block pairs in work-list order; with a work counter each CTA takes the next unclaimed one
    // (dynamic balance across groups of different lengths), else every gridDim.x-th.
    auto next_item = [&](int64_t tp) -> int64_t {
        if (tid == 0)
            next_sh = work_counter != nullptr ? (int64_t)gridDim.x + (int64_t)atomicAdd(work_counter, 1ULL)
                                               : tp + gridDim.x;
        __syncthreads();
        return next_sh;
    };
    for (int64_t tp = blockIdx.x; tp < total; tp = next_item(tp)) {
        const int64_t wi = upper_find(work_off, n_work, tp);
        const int64_t g = work_groups[wi];
        const int64_t m = grp_size[g];
        const int64_t nb = ceil_div<int64_t>(m, T);
        int64_t ua, ub1;
        tri_decode(tp - work_off[wi], nb + 1, &ua, &ub1);
        const int64_t ub = ub1 - 1;
        const bool diag = ua == ub;
        const int64_t a0 = ua * T, b0 = ub * T;
        const int64_t cb = cand_off[g] - chunk_base;
        const int64_t words = cwords[wi];
        const int64_t n_stages = ceil_div<int64_t>(words, WORDS);
        if (tid < 256) {
            const int64_t ia = a0 + tid, ib = b0 + tid;
            // Row-major rows: member i at cbase + i cld. Blocked rows (blocks of T members stored 4-word chunk
            // by chunk, each chunk as two 2-word halves, so a stage's words of one block are one run): member i
            // at cbase + (i / T) T cld + 2 (i % T).
            const int64_t cw = cld[wi];
            off_a[tid] = tid < T && ia < m ? cbase[wi] + (blocked ? ua * T * cw + 2 * tid : ia * cw) : -1;
            off_b[tid] = tid < T && ib < m ? cbase[wi] + (blocked ? ub * T * cw + 2 * tid : ib * cw) : -1;
        }
        int any = cls == nullptr;
        if (!any && tid < T) {
            const int64_t i = a0 + tid;
            for (int c = 0; c < T && !any; c++) {
                const int64_t j = b0 + c;
                any = i < j && j < m && cls[cb + tri_index(i, j, m)] == ETM_CAND_COUNT;
            }
        }
        if (!__syncthreads_or(any)) continue;

        if (warp < MMA_WARP) {
            // ---- producers ----
            const bool is_b = tid >= 256;
            const int prow = is_b ? tid - 256 : tid;
            const bool idle = prow >= T || (!is_b && diag);  // on a diagonal block pair the A rows are B rows
            const int64_t off = idle ? -1 : (is_b ? off_b[prow] : off_a[prow]);
            // B row r: row r of the 256-row B tile; A row r: row r % TH of A half r / TH.
            const int dst = is_b ? 2 * HALF_BYTES : (prow / TH) * HALF_BYTES;
            const int hrow = is_b ? prow : prow % TH;
            {
                uint64_t cur[BW], nxt[BW];
                // Words past the row's last stage are not read (they may lie past the buffer).
                const int64_t lim = n_stages * WORDS;
                auto load_batch = [&](int64_t s0, uint64_t* x) {
    #pragma unroll
                    for (int q = 0; q < BW; q += 2) {
                        const int64_t w = s0 * WORDS + q;
                        ulonglong2 v = make_ulonglong2(0, 0);
                        const int64_t at = off + (blocked ? (w >> 2) * (4 * T) + ((w >> 1) & 1) * (2 * T) + (w & 1) : w);
                        if (off >= 0 && w + 1 < lim) v = __ldg(reinterpret_cast<const ulonglong2*>(src + at));
                        else if (off >= 0 && w < lim) v.x = __ldg(src + at);
                        x[q] = v.x;
                        x[q + 1] = v.y;
                    }
                };
                if (n_stages > 0) load_batch(0, cur);
                for (int64_t s0 = 0; s0 < n_stages && !*abort_flag; s0 += PF) {
                    if (s0 + PF < n_stages) load_batch(s0 + PF, nxt);
    #pragma unroll
                    for (int j = 0; j < PF; j++) {
                        const int64_t s = s0 + j;
                        if (s >= n_stages) break;
                        const int64_t G = gstage + s;
                        const int slot = (int)(G % STAGES);
                        const uint32_t use = (uint32_t)(G / STAGES);
                        if (!mbar_wait(&empty_bar[slot], (use & 1u) ^ 1u, abort_flag, WAIT_NS)) break;
                        if (off >= 0) {
                            store_row<FMT>(slots + slot * SLOT_BYTES + dst, hrow, cur + j * WORDS);
                            fence_proxy_async();
                        }
                        mbar_arrive(&full_bar[slot]);
                    }
    #pragma unroll
                    for (int q = 0; q < BW; q++) cur[q] = nxt[q];
                }
            }
            // ---- epilogue: warp w reads lanes 32 (w % 4) .. of accumulator w / 8, columns 128 ((w / 4) % 2) .. ----
            // Every lane observes the accumulator barrier itself (its own acquire before its tcgen05 fence), and
            // the warp takes one decision, as the tcgen05.ld below needs the whole warp.
            const bool got_acc = n_stages == 0 || mbar_wait(&acc_bar, tile_iter & 1u, abort_flag, WAIT_NS);
            const bool ok = __all_sync(0xffffffffu, got_acc);
            if (ok) {
                tc_fence_after();
                const int lane_base = (warp & 3) * 32;
                const int accn = warp >> 3;
                const int64_t i = a0 + accn * TH + lane_base + lane;
                const bool row_ok = lane_base + lane < TH && i < m;
                for (int q = 0; q < 4; q++) {
                    const int col0 = ((warp >> 2) & 1) * 128 + q * 32;
                    if (col0 >= T) break;  // warp-uniform
                    uint32_t v[32];
                    if (n_stages > 0) {
                        const uint32_t taddr = tmem + ((uint32_t)lane_base << 16) + (uint32_t)(accn * T + col0);
                        asm volatile(
                            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
                            "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                              "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
                              "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
                              "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                            : "r"(taddr));
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    } else {
#pragma unroll
                        for (int c = 0; c < 32; c++) v[c] = 0u;
                    }
                    if (!row_ok) continue;
                    const int64_t j0 = b0 + col0;
                    const int64_t t0 = cb + tri_index(i, j0, m);  // slot of (i, j0 + c) is t0 + c when j0 + c > i
                    uint32_t bits = 0;
#pragma unroll
                    for (int c = 0; c < 32; c++) {
                        const int64_t j = j0 + c;
                        if (i < j && j < m && col0 + c < T) {
                            const int64_t t = t0 + c;
                            if (cls == nullptr || cls[t] == ETM_CAND_COUNT) {
                                const int32_t cnt =
                                    n_stages > 0 ? __float2int_rn(__uint_as_float(v[c]) * Fmt<FMT>::SCALE) : 0;
                                if (surv == nullptr) {
                                    out[t] = cnt;
                                } else if (cnt >= min_count) {
                                    out[t] = cnt;
                                    bits |= 1u << c;
                                }
                            }
                        }
                    }
                    if (bits != 0u) {
                        // Survivor bits of slots t0 + c, c in the mask: at most two words of the bitmask.
                        const int c1 = __ffs(bits) - 1;
                        const int64_t t1 = t0 + c1;
                        const uint32_t sh = (uint32_t)(t1 & 31);
                        const uint32_t mb = bits >> c1;
                        atomicOr(surv + (t1 >> 5), mb << sh);
                        if (sh != 0u && (mb >> (32u - sh)) != 0u) atomicOr(surv + (t1 >> 5) + 1, mb >> (32u - sh));
                    }
                }
            }
            tc_fence_before();
        } else if (warp == MMA_WARP && lane == 0) {
            // ---- MMA issuer: two M = 128 MMAs per K step, sharing the B tile ----
            tc_fence_after();
            for (int64_t s = 0; s < n_stages; s++) {
                const int64_t G = gstage + s;
                const int slot = (int)(G % NST);
                const uint32_t use = (uint32_t)(G / NST);
                if (!mbar_wait(&full_bar[slot], use & 1u, abort_flag, first_wait_ns)) break;
                tc_fence_after();
                const uint32_t base = smem_u32(slots + slot * SLOT_BYTES);
                const uint32_t b_addr = base + 2 * HALF_BYTES;
                // A half h: rows h TH .. of block ua; on a diagonal block pair, rows of the B tile.
                const uint32_t a_lo = diag ? b_addr : base;
                const uint32_t a_hi = diag ? b_addr + TH * 128 : base + HALF_BYTES;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t acc = (s > 0 || k > 0) ? 1u : 0u;
                    const uint64_t bd = smem_desc(b_addr + 32 * k);
                    mma_ss<FMT>(tmem, smem_desc(a_lo + 32 * k), bd, acc, tmem + SF_COL);
                    mma_ss<FMT>(tmem + T, smem_desc(a_hi + 32 * k), bd, acc, tmem + SF_COL);
                }
                mma_commit(&empty_bar[slot]);
            }
            // A block pair without stages (an empty prefix) issues no MMA and commits nothing: its producers do
            // not wait for the accumulator, and acc_bar's phases stay one per block pair with stages, so a
            // later pair's epilogue can never take an earlier phase for its own.
            if (n_stages > 0) mma_commit(&acc_bar);
        }
        gstage += n_stages;
        if (n_stages > 0) tile_iter += 1;  // one acc_bar phase per block pair with stages
        __syncthreads();
        if (*abort_flag) break;
    }

    if (warp == MMA_WARP) {
        if (lane == 0 && *abort_flag) {
            // Wait (bounded) for every MMA this CTA issued before its tensor memory is freed.
            mma_commit(&drain_bar);
            const uint64_t t0 = now_ns();
            while (!mbar_test(&drain_bar, 0) && now_ns() - t0 < WAIT_NS) __nanosleep(256);
        }
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
    if (tid == 0 && *abort_flag) atomicExch(&g_tc_status, ETM_ETIMEOUT);
}

// ---- packed e2m1 over blocked rows ---------------------------------------------------------------------------
//
// The form the engine runs: 15 producer warps, a row a thread, load the raw bits (32 bytes a row and stage, a warp's 16-byte
// halves contiguous in the blocked layout) BK_AHEAD stages ahead into registers and expand them into BK_OPS operand
// slots; one thread of the sixteenth warp issues the MMAs; all sixteen read the accumulators.
//
// What bounds it: shared memory. A stage of 256 rows stores 480 rows of 128 bytes and its 8 MMAs read 736 (B for each A
// half), 1,216 wavefronts of 128 bytes, 0.59 us at 2,070 MHz; the MMAs alone take 0.49 us. Measured 0.70 us a stage
// (2,400 members; 0.88 with raw stages copied through shared memory and two operand slots). A slot's way round
// (expansion, fence, arrival, the MMAs, their commit and the wake-ups between) is about three times its MMAs, hence
// three slots, and hence the raw words in registers, which leave the room for them. Rings are walked by counters (a
// 64-bit division by the ring size in every thread and stage costs more than the expansion), a warp arrives once for its
// 32 rows, and the MMA warp decodes the next work item while its last MMAs run.
//
// Roles of the blocks: the columns of the accumulators are the members i of block ua (the B tile, N of them), the
// lanes the members j of block ub (two A halves of TH rows). Candidate (i, j) lies at consecutive slots for
// consecutive j, so a warp's 32 lanes store 32 consecutive counts and one ballot makes their survivor bits. The MMAs
// run over the block's members only: N is the members of ua rounded up to 16, the second A half is left out where
// ub ends within the first, and on a diagonal pair the first half (j < TH) meets only the columns i < TH.
//
// A work item is one part of the rows of one block pair (parts[wi] parts per pair of work entry wi, one without
// `parts`): a level of few block pairs over many rows still fills the SMs. Items of a pair cut in parts add their
// counts into `out` (zeroed by the caller, who takes a threshold pass over it); f32 holds the sums of a part of at
// most 2^24 rows exactly. Measured on 20M rows: the Grams of K=3 and K=4 (171 and 281 groups, 3 block pairs at most)
// 48.1 -> 2.1 ms, K=2 of 426 columns 15.5 ms on popcount tiles (past 2^24 rows) -> 0.9 ms; K=2 of 267 columns over
// 1M rows 3.6 -> 0.08 ms. On levels of many pairs (630M candidates over 1M rows) the kernel takes what the
// one-arrive-per-thread, one-count-per-lane form took, less the K=2 level (5.4 -> 2.0 ms in blocked rows).
struct GramItem {
    int64_t wi;       // work entry, -1: no more items
    int64_t pair_ua, pair_ub;
    int64_t s0, s1;   // stages of the part
    bool split;       // one of several parts: counts are added
};

// Item tp, decoded by a whole warp (every lane gets it): the work entry by a search over 32 places at a time.
__device__ __forceinline__ GramItem gram_item(int64_t tp, int64_t total, const int64_t* __restrict__ work_off,
                                              int64_t n_work, const int64_t* __restrict__ parts,
                                              const int64_t* __restrict__ work_groups,
                                              const int32_t* __restrict__ grp_size,
                                              const int64_t* __restrict__ cwords) {
    GramItem it;
    it.wi = -1;
    if (tp >= total) return it;
    const int lane = threadIdx.x & 31;
    int64_t lo = 0, hi = n_work;  // work_off[lo] <= tp < work_off[hi]
    while (hi - lo > 1) {
        const int64_t step = ceil_div<int64_t>(hi - lo, 33);
        const int64_t at = lo + (lane + 1) * step;
        const unsigned below = __ballot_sync(0xffffffffu, at < hi && work_off[at] <= tp);
        const int n = __popc(below);  // the offsets do not decrease: the lanes below are the first ones
        hi = min64(hi, lo + (n + 1) * step);
        lo += n * step;
    }
    it.wi = lo;
    const int64_t m = grp_size[work_groups[it.wi]];
    const int64_t nb = ceil_div<int64_t>(m, Fmt<4>::T);
    const int64_t np = parts != nullptr ? max64(1, parts[it.wi]) : 1;
    int64_t pair = (tp - work_off[it.wi]) / np;
    const int64_t part = (tp - work_off[it.wi]) - pair * np;
    int64_t ua = 0;
    while (pair >= nb - ua) pair -= nb - ua++;
    it.pair_ua = ua;
    it.pair_ub = ua + pair;
    const int64_t n_stages = ceil_div<int64_t>(cwords[it.wi], Fmt<4>::WORDS);
    const int64_t per = ceil_div<int64_t>(n_stages, np);
    it.s0 = min64(n_stages, part * per);
    it.s1 = min64(n_stages, it.s0 + per);
    it.split = np > 1;
    return it;
}

// 32 accumulator columns of the warp's lanes.
__device__ __forceinline__ void tmem_ld32(uint32_t (&v)[32], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Items are checked on the way where the members' row counts are given: member i of the rarer block has so many rows
// of the prefix, of which so many have passed; once no pair's count so far plus what its member i has left reaches
// min_count, none of the item's candidates is frequent and the rest of its rows need not be counted. With the
// generators numbered by ascending support most block pairs of a level over independent items end that way. A check
// drains the operand slots, reads the accumulators and refills the ring, about as long as CHECK_COST stages; the next
// one is put a little past where the pairs' paces say it will succeed, and none where it would save less than it
// costs.
constexpr int CHECK_STAGES = 32;  // items checked at all
constexpr int CHECK_COST = 6;

__device__ __forceinline__ int next_check(float at, int done, int n_stages) {
    int s = max(done + 2 * CHECK_COST, (int)((at + 0.01f) * (float)n_stages) + 1);
    s = (s + BK_AHEAD - 1) / BK_AHEAD * BK_AHEAD;  // the producers' registers go on where they were
    return s + 2 * CHECK_COST < n_stages ? s : n_stages;
}

// A ring position: slot and the parity of its current use.
template <int N>
struct Ring {
    int slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next() {
        if (++slot == N) {
            slot = 0;
            phase ^= 1u;
        }
    }
};

__global__ void __launch_bounds__(BK_THREADS, 1) gram_blocked_kernel(
    const uint64_t* __restrict__ src, const int64_t* __restrict__ cbase, const int64_t* __restrict__ cwords,
    const int64_t* __restrict__ cld, const int32_t* __restrict__ grp_size, const int64_t* __restrict__ cand_off,
    const int64_t* __restrict__ work_groups, const int64_t* __restrict__ work_off, const int64_t* __restrict__ parts,
    int64_t n_work, int64_t chunk_base, const uint8_t* __restrict__ cls, int32_t min_count, int32_t* __restrict__ out,
    uint32_t* __restrict__ surv, const int64_t* __restrict__ grp_first, const int32_t* __restrict__ row_counts,
    unsigned long long* __restrict__ work_counter, uint64_t first_wait_ns) {
    constexpr int T = Fmt<4>::T;
    constexpr int TH = T / 2;
    constexpr int WORDS = Fmt<4>::WORDS;
    static_assert((T + 8) * 128 == BK_TILE && TH % 8 == 0 && TH <= 120 && T % 16 == 0, "block shape");
    extern __shared__ uint8_t dsmem[];
    __shared__ __align__(8) uint64_t full_bar[BK_OPS];
    __shared__ __align__(8) uint64_t empty_bar[BK_OPS];
    __shared__ __align__(8) uint64_t acc_bar;
    __shared__ __align__(8) uint64_t drain_bar;
    __shared__ uint32_t tmem_sh;
    __shared__ int abort_sh;
    __shared__ GramItem items[2];
    __shared__ int32_t left_sh[T];        // rows of member i yet to come
    __shared__ int most_i, most_j;        // largest row counts of the two blocks
    __shared__ unsigned next_sh[2];       // where the next check pays, in 65536ths of the item (0: it is decided)

    uint8_t* slots = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dsmem) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int64_t total = work_off[n_work];

    if (tid == 0) {
        for (int s = 0; s < BK_OPS; s++) {
            mbar_init(&full_bar[s], BK_MMA_WARP);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_bar, 1);
        mbar_init(&drain_bar, 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (row_counts != nullptr && tid < 16 * BK_OPS) {
        // A row of ones behind the members' in the A and in the B tile of every slot: it is row TH of the second A half
        // (of a diagonal pair's too), whose lane TH then counts the rows of each member i.
        uint8_t* to = slots + (tid >> 4) * BK_SLOT + ((tid >> 3) & 1) * BK_TILE + T * 128 + (tid & 7) * 16;
        *reinterpret_cast<uint4*>(to) = make_uint4(0x11111111u, 0x11111111u, 0x11111111u, 0x11111111u);
        fence_proxy_async();
    }
    if (warp == BK_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    if (warp == 0) {
        const GramItem first = gram_item(blockIdx.x, total, work_off, n_work, parts, work_groups, grp_size, cwords);
        if (lane == 0) items[0] = first;
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_sh;
    volatile int* abort_flag = &abort_sh;
    // Unit scale factors: warp w (w < 4) fills lanes 32 w .. 32 w + 31 of columns 480-511 with 127s.
    if (warp < 4) {
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + SF_COL;
        const uint32_t u = 0x7F7F7F7Fu;
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
            "%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
            "r"(u)
            : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    Ring<BK_OPS> op;  // producers and MMA thread: the next operand stage
    uint32_t acc_phase = 0;
    int64_t tp = blockIdx.x;  // MMA warp: the item last decoded
    // The next item, claimed and decoded by the MMA warp into the other descriptor.
    auto next_item = [&](int cur) {
        if (work_counter != nullptr) {
            unsigned long long c = 0;
            if (lane == 0) c = atomicAdd(work_counter, 1ULL);
            tp = (int64_t)gridDim.x + (int64_t)__shfl_sync(0xffffffffu, c, 0);
        } else {
            tp += gridDim.x;
        }
        const GramItem next = gram_item(tp, total, work_off, n_work, parts, work_groups, grp_size, cwords);
        if (lane == 0) items[cur ^ 1] = next;
    };
    for (int cur = 0; items[cur].wi >= 0; cur ^= 1) {
        const GramItem it = items[cur];
        const int64_t g = work_groups[it.wi];
        const int64_t m = grp_size[g];
        const bool diag = it.pair_ua == it.pair_ub;
        const int64_t i0 = it.pair_ua * T, j0 = it.pair_ub * T;  // first member of the B columns / of the A lanes
        const int n_i = (int)min64(T, m - i0), n_j = (int)min64(T, m - j0);
        const int64_t cb = cand_off[g] - chunk_base;
        const int n_stages = (int)(it.s1 - it.s0);
        bool live = n_stages > 0 || !it.split;  // an empty part adds nothing
        if (live && cls != nullptr) {
            // A block pair none of whose candidates needs a count is skipped: lanes over j, warps over i.
            int any = 0;
            for (int a = warp; a < n_i && !any; a += BK_THREADS / 32) {
                const int64_t i = i0 + a, row = cb + tri_index(i, 0, m);
                int hit = 0;
                for (int b = lane; b < n_j; b += 32) {
                    const int64_t j = j0 + b;
                    hit |= i < j && cls[row + j] == ETM_CAND_COUNT;
                }
                any = __any_sync(0xffffffffu, hit);
            }
            live = __syncthreads_or(any) != 0;
        }
        if (!live) {
            if (warp == BK_MMA_WARP) next_item(cur);
            __syncthreads();
            continue;
        }
        // Second A half in use; columns of its MMAs, and of the first half's.
        const bool two = n_j > TH;
        const int n_hi = (n_i + 15) & ~15;
        const int n_lo = diag ? min(n_hi, (TH + 15) & ~15) : n_hi;
        // Checks on the way (see CHECK_STAGES): the stage of the next one, n_stages for none.
        int check = n_stages;
        if (row_counts != nullptr && surv != nullptr && !it.split && n_stages >= CHECK_STAGES) {
            const int32_t* tot = row_counts + grp_first[g];
            if (tid == 0) most_i = most_j = 0;
            __syncthreads();
            if (tid < T) {
                const int v = tid < n_i ? tot[i0 + tid] : 0;
                if (v != 0) atomicMax(&most_i, v);
            } else if (tid < T + n_j) {
                atomicMax(&most_j, tot[j0 + tid - T]);
            }
            __syncthreads();
            // Members independent of each other would meet in most_i most_j / rows of the prefix's rows.
            const float mi = (float)min(most_i, most_j), mj = (float)max(most_i, most_j);
            const float meet = mi * mj / (256.f * (float)n_stages);
            if (meet < (float)min_count && mi > (float)min_count)
                check = next_check((mi - (float)min_count) / (mi - meet), 0, n_stages);
            else if (mi <= (float)min_count)
                check = next_check(0.f, 0, n_stages);
        }
        int done = 0, n_checks = 0;  // stages behind the latest check
        // Producer of row `prow` of the A tile or of the B tile. On a diagonal pair the A rows are rows of the B tile.
        // With one A half the row behind it takes the place of the row of ones.
        const bool is_b = tid >= T;
        const int prow = is_b ? tid - T : tid;
        const bool ones = !two && prow == TH && is_b == diag;
        const bool reads = warp < BK_MMA_WARP && (is_b ? prow < n_i : (!diag && prow < n_j));
        const uint4* rsrc = prow + reinterpret_cast<const uint4*>(
            src + cbase[it.wi] + (is_b ? it.pair_ua : it.pair_ub) * T * cld[it.wi] + it.s0 * WORDS * T);
        uint4 ahead[BK_AHEAD][2];
        auto load = [&](int s, uint4 (&x)[2]) {  // words 0-1 and 2-3 of the row's stage s
            const uint4* r = rsrc + (int64_t)s * (WORDS * T / 2);
            x[0] = __ldg(r);
            x[1] = __ldg(r + T);
        };
#pragma unroll
        for (int p = 0; p < BK_AHEAD; p++) {
            ahead[p][0] = ahead[p][1] = make_uint4(~0u, ~0u, ~0u, ~0u);
            if (reads && p < n_stages) load(p, ahead[p]);
        }
        for (;;) {
            const int s_end = min(check, n_stages);
            if (tid == 0) next_sh[n_checks & 1] = 0u;
            if (warp < BK_MMA_WARP) {
                // ---- producers ----
                uint8_t* dst = slots + (is_b ? BK_TILE : 0);
                bool going = true;
                for (int s0 = done; s0 < s_end && going; s0 += BK_AHEAD) {
#pragma unroll
                    for (int p = 0; p < BK_AHEAD; p++) {
                        const int s = s0 + p;
                        if (s >= s_end || !going) continue;
                        going = __all_sync(0xffffffffu,
                                           mbar_wait(&empty_bar[op.slot], op.phase ^ 1u, abort_flag, WAIT_NS));
                        if (!going) continue;
                        if (reads || ones) {
                            const uint4 &v0 = ahead[p][0], &v1 = ahead[p][1];
                            const uint64_t x[4] = {
                                (uint64_t)v0.x | ((uint64_t)v0.y << 32), (uint64_t)v0.z | ((uint64_t)v0.w << 32),
                                (uint64_t)v1.x | ((uint64_t)v1.y << 32), (uint64_t)v1.z | ((uint64_t)v1.w << 32)};
                            store_row<4>(dst + op.slot * BK_SLOT, prow, x);
                            fence_proxy_async();
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&full_bar[op.slot]);
                        op.next();
                        if (reads && s + BK_AHEAD < n_stages) load(s + BK_AHEAD, ahead[p]);
                    }
                }
            } else {
                // ---- MMA issuer: an M = 128 MMA per A half and K step, sharing the B tile ----
                // The whole warp waits and one elected lane issues. Issued from a branch of one lane, with a loop's
                // waits and exits around them, the same MMAs came at a third of the rate (3,090 against 9,740 TFLOP/s
                // back to back), and this kernel took 0.83 us a stage.
                tc_fence_after();
                constexpr uint32_t desc0 = instr_desc<4>() & ~((uint32_t)0x3F << 17);
                const uint32_t id_lo = desc0 | ((uint32_t)(n_lo >> 3) << 17);
                const uint32_t id_hi = desc0 | ((uint32_t)(n_hi >> 3) << 17);
                for (int s = done; s < s_end; s++) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[op.slot], op.phase, abort_flag, first_wait_ns)))
                        break;
                    tc_fence_after();
                    // A half h: rows h TH .. of block ub; on a diagonal block pair, rows of the B tile.
                    const uint32_t b_addr = smem_u32(slots + op.slot * BK_SLOT) + BK_TILE;
                    const uint32_t a_lo = diag ? b_addr : b_addr - BK_TILE;
                    const uint32_t a_hi = a_lo + TH * 128;
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            mma_mxf4(tmem, smem_desc(a_lo + 32 * k), smem_desc(b_addr + 32 * k), id_lo,
                                     (s > 0 || k > 0) ? 1u : 0u, tmem + SF_COL);
                        if (two) {
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                mma_mxf4(tmem + T, smem_desc(a_hi + 32 * k), smem_desc(b_addr + 32 * k), id_hi,
                                         (s > 0 || k > 0) ? 1u : 0u, tmem + SF_COL);
                        }
                        mma_commit(&empty_bar[op.slot]);
                    }
                    __syncwarp();
                    op.next();
                }
                // A block pair without stages (an empty prefix) issues no MMA and commits nothing: its warps do not wait
                // for the accumulator, and acc_bar's phases stay one per run of stages, so a later pair's epilogue can
                // never take an earlier phase for its own.
                if (n_stages > 0 && elect_one()) mma_commit(&acc_bar);  // at the end, and at every check
                __syncwarp();
                if (s_end >= n_stages) next_item(cur);
            }
            // ---- epilogue: warp w reads lanes 32 (w % 4) .. of accumulator w / 8, columns 128 ((w / 4) % 2) .. ----
            // Every lane observes the accumulator barrier itself (its own acquire before its tcgen05
            // fence), and the warp takes one decision, as the tcgen05.ld below needs the whole warp.
            const bool ok =
                n_stages == 0 || __all_sync(0xffffffffu, mbar_wait(&acc_bar, acc_phase, abort_flag, WAIT_NS));
            const int accn = warp >> 3, lane_base = (warp & 3) * 32;
            const int jl = accn * TH + lane_base + lane;  // this lane's member of block ub
            const int c_end = min(n_i, accn == 0 && diag ? TH : T);
            if (s_end < n_stages) {
                // ---- check: can any of the pairs still reach min_count? ----
                // Member i of the first block has left_sh[i] rows yet to come, so (i, j) ends at its count so
                // far plus that at most. The pairs that can still get there say where they would stop if both
                // counts went on at their pace.
                tc_fence_after();
                if (ok && lane_base + 32 > TH && accn == (two ? 1 : 0)) {
                    const int32_t* tot = row_counts + grp_first[g] + i0;
                    for (int q = 0; q < 4; q++) {
                        const int col0 = ((warp >> 2) & 1) * 128 + q * 32;
                        if (col0 >= n_i) break;
                        uint32_t v[32];
                        tmem_ld32(v, tmem + ((uint32_t)lane_base << 16) + (uint32_t)(accn * T + col0));
                        if (lane == TH - lane_base) {
#pragma unroll
                            for (int c = 0; c < 32; c++)
                                if (col0 + c < n_i)
                                    left_sh[col0 + c] =
                                        tot[col0 + c] - __float2int_rn(__uint_as_float(v[c]) * Fmt<4>::SCALE);
                        }
                    }
                }
                __syncthreads();
                const bool lane_ok = (accn == 0 || two) && lane_base + lane < TH && jl < n_j;
                const float f = (float)s_end / (float)n_stages, mc = (float)min_count;
                const float inv_f = 1.f / f, inv_r = 1.f / (1.f - f);
                float want = 0.f;
                for (int q = 0; q < 4 && ok; q++) {
                    const int col0 = ((warp >> 2) & 1) * 128 + q * 32;
                    if (col0 >= c_end) break;  // warp-uniform
                    uint32_t v[32];
                    tmem_ld32(v, tmem + ((uint32_t)lane_base << 16) + (uint32_t)(accn * T + col0));
#pragma unroll
                    for (int c = 0; c < 32; c++) {
                        const int i = col0 + c;
                        if (!lane_ok || i >= c_end || i0 + i >= j0 + jl) continue;
                        const float so_far = __uint_as_float(v[c]) * Fmt<4>::SCALE, left = (float)left_sh[i];
                        if (so_far + left < mc) continue;
                        const float pace = so_far * inv_f, rest = left * inv_r;
                        want = fmaxf(want, pace >= mc ? 2.f : rest <= mc ? f : (rest - mc) / (rest - pace));
                    }
                }
                // At least one 65536th for a pair that is not decided.
                unsigned bits = want > 0.f ? max(1u, (unsigned)(fminf(want, 2.f) * 65536.f)) : 0u;
                bits = __reduce_max_sync(0xffffffffu, bits);
                if (lane == 0 && bits != 0u) atomicMax(&next_sh[n_checks & 1], bits);
            } else if (ok && (accn == 0 || two) && lane_base < TH) {
                tc_fence_after();
                const bool lane_ok = lane_base + lane < TH && jl < n_j;
                const int64_t j = j0 + jl;
                for (int q = 0; q < 4; q++) {
                    const int col0 = ((warp >> 2) & 1) * 128 + q * 32;
                    if (col0 >= c_end) break;  // warp-uniform
                    uint32_t v[32];
                    if (n_stages > 0) {
                        const uint32_t taddr = tmem + ((uint32_t)lane_base << 16) + (uint32_t)(accn * T + col0);
                        tmem_ld32(v, taddr);
                    } else {
#pragma unroll
                        for (int c = 0; c < 32; c++) v[c] = 0u;
                    }
                    // Slot of (i, j), i = i0 + col0 + c: row i starts (m - i - 2) after row i - 1's (j - 1) slot.
                    int64_t t = cb + tri_index(i0 + col0, j, m);
                    int64_t step = m - (i0 + col0) - 2;
#pragma unroll
                    for (int c = 0; c < 32; c++) {
                        const int64_t i = i0 + col0 + c;
                        bool on = lane_ok && i < j && col0 + c < c_end;
                        const int32_t cnt = __float2int_rn(__uint_as_float(v[c]) * Fmt<4>::SCALE);
                        if (on && cls != nullptr) on = cls[t] == ETM_CAND_COUNT;
                        if (it.split) {
                            if (on && cnt != 0) atomicAdd(out + t, cnt);
                        } else if (surv == nullptr) {
                            if (on) out[t] = cnt;
                        } else {
                            const bool keep = on && cnt >= min_count;
                            if (keep) out[t] = cnt;
                            const unsigned bits = __ballot_sync(0xffffffffu, keep);
                            if (bits != 0u && lane == 0) {
                                // Bits of slots t .. t + 31 (lane 0's slot first): at most two words of the
                                // bitmask. Lane 0's slot lies before the bitmask where i > j, so the shift
                                // starts at the first survivor.
                                const int b1 = __ffs(bits) - 1;
                                const int64_t t1 = t + b1;
                                const uint32_t sh = (uint32_t)(t1 & 31), mb = bits >> b1;
                                atomicOr(surv + (t1 >> 5), mb << sh);
                                if (sh != 0u && (mb >> (32u - sh)) != 0u)
                                    atomicOr(surv + (t1 >> 5) + 1, mb >> (32u - sh));
                            }
                        }
                        t += step;
                        step -= 1;
                    }
                }
            }
            tc_fence_before();
            if (n_stages > 0) acc_phase ^= 1u;  // one acc_bar phase per run of stages
            __syncthreads();
            if (*abort_flag || s_end >= n_stages) break;
            const unsigned next = next_sh[n_checks & 1];
            if (next == 0u) {  // no pair of the item can survive
                if (warp == BK_MMA_WARP) next_item(cur);
                __syncthreads();
                break;
            }
            check = next_check((float)next * (1.f / 65536.f), s_end, n_stages);
            done = s_end;
            n_checks += 1;
        }
        if (*abort_flag) break;
    }

    if (warp == BK_MMA_WARP) {
        if (*abort_flag && elect_one()) {
            // Wait (bounded) for every MMA this CTA issued before its tensor memory is freed.
            mma_commit(&drain_bar);
            const uint64_t t0 = now_ns();
            while (!mbar_test(&drain_bar, 0) && now_ns() - t0 < WAIT_NS) __nanosleep(256);
        }
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
    if (tid == 0 && *abort_flag) atomicExch(&g_tc_status, ETM_ETIMEOUT);
}

// Issue rate of the Gram's own MMA shape: one CTA per SM, one thread issuing `iters` back-to-back MMAs
// (M = 128, N = T, the format's K per instruction) on a zeroed shared-memory tile into one accumulator,
// then a bounded wait for their completion. The roofline's tensor peak for that operand format.
template <int FMT>
__global__ void __launch_bounds__(128, 1) mma_rate_kernel(int64_t iters, int* status) {
    extern __shared__ uint8_t dsmem[];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_sh;
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dsmem) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int i = tid; i < 3 * HALF_BYTES / 16; i += blockDim.x) reinterpret_cast<uint4*>(tiles)[i] = make_uint4(0, 0, 0, 0);
    if (tid == 0) {
        mbar_init(&done_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_proxy_async();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_sh;
    if constexpr (FMT == 4) {
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + SF_COL;
        const uint32_t u = 0x7F7F7F7Fu;
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
            "%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
            "r"(u)
            : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }
    if (tid == 0) {
        const uint32_t a = smem_u32(tiles), b = a + HALF_BYTES;
        for (int64_t it = 0; it < iters; it++) {
            const int k = (int)(it & 3);
            mma_ss<FMT>(tmem, smem_desc(a + 32 * k), smem_desc(b + 32 * k), it > 0 ? 1u : 0u, tmem + SF_COL);
        }
        mma_commit(&done_bar);
        const uint64_t t0 = now_ns();
        bool ok = true;
        while (!mbar_test(&done_bar, 0)) {
            if (now_ns() - t0 > WAIT_NS) {
                ok = false;
                break;
            }
            __nanosleep(128);
        }
        if (!ok) atomicExch(status, ETM_ETIMEOUT);
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

std::mutex g_cfg_lock;
// The MMA thread's wait for a filled stage: WAIT_NS unless a test set it (0 = give up at once).
uint64_t g_first_wait_ns = WAIT_NS;

struct GramArgs {
    const uint64_t* cbuf;
    const int64_t *cbase, *cwords, *cld;
    const int32_t* grp_size;
    const int64_t *cand_off, *work_groups, *work_off;
    const int64_t* parts;  // parts per block pair of each work entry (nullptr: one)
    int64_t n_work, n_tiles, chunk_base;
    const uint8_t* cls;
    int32_t min_count;
    int32_t* out;
    uint32_t* surv;
    int64_t* work_counter;
    bool blocked;
    cudaStream_t s;
    const int64_t* grp_first = nullptr;   // with row_counts: the groups' first rows in the level and
    const int32_t* row_counts = nullptr;  // the level's counts
};

// One CTA per SM over the work items, claimed from the counter when there is one.
int gram_launch_setup(const GramArgs& a, const void* kernel, int smem, bool* configured, uint64_t* first_wait,
                      int* grid) {
    {
        std::lock_guard<std::mutex> guard(g_cfg_lock);
        if (!*configured) {
            ETM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            *configured = true;
        }
        *first_wait = g_first_wait_ns;
    }
    const int64_t sms = max(1, sm_count());
    *grid = (int)max64(1, min64(sms, a.n_tiles > 0 ? a.n_tiles : sms));
    if (a.work_counter != nullptr) ETM_CUDA(cudaMemsetAsync(a.work_counter, 0, sizeof(int64_t), a.s));
    return ETM_OK;
}

template <int FMT>
int launch_gram(const GramArgs& a) {
    static bool configured = false;
    uint64_t first_wait;
    int grid;
    if (const int st = gram_launch_setup(a, (const void*)gram_kernel<FMT>, SMEM_BYTES, &configured, &first_wait, &grid))
        return st;
    gram_kernel<FMT><<<grid, THREADS, SMEM_BYTES, a.s>>>(
        a.cbuf, a.cbase, a.cwords, a.cld, a.grp_size, a.cand_off, a.work_groups, a.work_off, a.n_work, a.chunk_base,
        a.cls, a.min_count, a.out, a.surv, reinterpret_cast<unsigned long long*>(a.work_counter), first_wait, a.blocked);
    ETM_LAUNCHED("gram_tc");
    return ETM_OK;
}

int launch_gram_blocked(const GramArgs& a) {
    static bool configured = false;
    uint64_t first_wait;
    int grid;
    if (const int st = gram_launch_setup(a, (const void*)gram_blocked_kernel, BK_SMEM, &configured, &first_wait, &grid))
        return st;
    gram_blocked_kernel<<<grid, BK_THREADS, BK_SMEM, a.s>>>(
        a.cbuf, a.cbase, a.cwords, a.cld, a.grp_size, a.cand_off, a.work_groups, a.work_off, a.parts, a.n_work,
        a.chunk_base, a.cls, a.min_count, a.out, a.surv, a.grp_first, a.row_counts,
        reinterpret_cast<unsigned long long*>(a.work_counter), first_wait);
    ETM_LAUNCHED("gram_tc");
    return ETM_OK;
}

}  // namespace

namespace etm {

int gram_block_members(int32_t elem) {
    const int e = elem & ~(ETM_TC_WIDE | ETM_TC_BLOCKED);
    return e == ETM_TC_MXF4 ? Fmt<4>::T : e == 1 || e == 2 ? Fmt<1>::T : 0;
}

int gram_tc(const uint64_t* cbuf, const int64_t* cbase, const int64_t* cwords, const int64_t* cld,
            const int32_t* grp_size, const int64_t* cand_off, const int64_t* work_groups, const int64_t* work_off,
            int64_t n_work, int64_t n_tiles, int64_t chunk_base, const uint8_t* cls, int32_t elem, int32_t min_count,
            int32_t* out, uint32_t* surv, int64_t* work_counter, cudaStream_t s) {
    // elem: 1 = e4m3, 2 = f16, ETM_TC_MXF4 = packed e2m1; ETM_TC_WIDE is accepted and changes nothing;
    // + ETM_TC_BLOCKED: the member rows are in the projection's blocked layout with blocks of T members.
    const bool blocked = (elem & ETM_TC_BLOCKED) != 0;
    const int e = elem & ~(ETM_TC_WIDE | ETM_TC_BLOCKED);
    ETM_REQUIRE(e == 1 || e == 2 || e == ETM_TC_MXF4, ETM_EINVAL,
                "gram_tc: element code %d (1 = e4m3, 2 = f16, %d = e2m1 block-scaled)", elem, ETM_TC_MXF4);
    const GramArgs a{cbuf, cbase, cwords, cld, grp_size, cand_off, work_groups, work_off, nullptr, n_work, n_tiles,
                     chunk_base, cls, min_count, out, surv, work_counter, blocked, s};
    if (e == ETM_TC_MXF4) return blocked ? launch_gram_blocked(a) : launch_gram<4>(a);
    return e == 2 ? launch_gram<2>(a) : launch_gram<1>(a);
}

int count_tiles_tensor(const uint64_t*, int64_t, int64_t, const int32_t*, int32_t, const int64_t*, const int32_t*,
                       const int64_t*, const int64_t*, const int64_t*, int64_t, int64_t, const uint8_t*, int32_t*,
                       cudaStream_t) {
    set_error("etm_count_tiles: the tensor method counts projected groups; use etm_count_tiles_tc");
    return ETM_EINVAL;
}

}  // namespace etm

extern "C" int etm_count_tiles_tc(const uint64_t* cbuf, const int64_t* cbase, const int64_t* cwords,
                                  const int64_t* cld, const int32_t* grp_size, const int64_t* cand_off,
                                  const int64_t* work_groups, const int64_t* work_off, int64_t n_work,
                                  int64_t n_tiles, int64_t chunk_base, const uint8_t* cls, int32_t elem,
                                  int32_t* out_counts, int64_t* work_counter, void* stream) {
    ETM_REQUIRE((reinterpret_cast<uintptr_t>(cbuf) & 15) == 0, ETM_EINVAL, "etm_count_tiles_tc: cbuf must be 16-byte aligned");
    if (n_work <= 0) return ETM_OK;
    return etm::gram_tc(cbuf, cbase, cwords, cld, grp_size, cand_off, work_groups, work_off, n_work, n_tiles,
                        chunk_base, cls, elem, 0, out_counts, nullptr, work_counter, as_stream(stream));
}

extern "C" int etm_count_tiles_tc_sel(const uint64_t* cbuf, const int64_t* cbase, const int64_t* cwords,
                                      const int64_t* cld, const int32_t* grp_size, const int64_t* cand_off,
                                      const int64_t* work_groups, const int64_t* work_off, int64_t n_work,
                                      int64_t n_tiles, int64_t chunk_base, const uint8_t* cls, int32_t elem,
                                      int32_t min_count, int32_t* out_counts, uint32_t* surv_bits,
                                      int64_t* work_counter, void* stream) {
    ETM_REQUIRE((reinterpret_cast<uintptr_t>(cbuf) & 15) == 0, ETM_EINVAL,
                "etm_count_tiles_tc_sel: cbuf must be 16-byte aligned");
    ETM_REQUIRE(surv_bits != nullptr, ETM_EINVAL, "etm_count_tiles_tc_sel: surv_bits is required");
    if (n_work <= 0) return ETM_OK;
    return etm::gram_tc(cbuf, cbase, cwords, cld, grp_size, cand_off, work_groups, work_off, n_work, n_tiles,
                        chunk_base, cls, elem, min_count, out_counts, surv_bits, work_counter, as_stream(stream));
}

extern "C" int etm_count_tiles_tc_parts(const uint64_t* cbuf, const int64_t* cbase, const int64_t* cwords,
                                        const int64_t* cld, const int32_t* grp_size, const int64_t* cand_off,
                                        const int64_t* work_groups, const int64_t* work_off, const int64_t* parts,
                                        int64_t n_work, int64_t n_items, int64_t chunk_base, const uint8_t* cls,
                                        int32_t* out_counts, int64_t* work_counter, void* stream) {
    ETM_REQUIRE((reinterpret_cast<uintptr_t>(cbuf) & 15) == 0, ETM_EINVAL,
                "etm_count_tiles_tc_parts: cbuf must be 16-byte aligned");
    ETM_REQUIRE(parts != nullptr, ETM_EINVAL, "etm_count_tiles_tc_parts: parts is required");
    if (n_work <= 0) return ETM_OK;
    return launch_gram_blocked(GramArgs{cbuf, cbase, cwords, cld, grp_size, cand_off, work_groups, work_off, parts,
                                       n_work, n_items, chunk_base, cls, 0, out_counts, nullptr, work_counter, true,
                                       as_stream(stream)});
}

extern "C" int etm_count_tiles_tc_bound(const uint64_t* cbuf, const int64_t* cbase, const int64_t* cwords,
                                        const int64_t* cld, const int32_t* grp_size, const int64_t* cand_off,
                                        const int64_t* work_groups, const int64_t* work_off, int64_t n_work,
                                        int64_t n_tiles, int64_t chunk_base, const uint8_t* cls, int32_t min_count,
                                        int32_t* out_counts, uint32_t* surv_bits, const int64_t* grp_first,
                                        const int32_t* row_counts, int64_t* work_counter, void* stream) {
    ETM_REQUIRE((reinterpret_cast<uintptr_t>(cbuf) & 15) == 0, ETM_EINVAL,
                "etm_count_tiles_tc_bound: cbuf must be 16-byte aligned");
    ETM_REQUIRE(surv_bits != nullptr && grp_first != nullptr && row_counts != nullptr, ETM_EINVAL,
                "etm_count_tiles_tc_bound: surv_bits, grp_first and row_counts are required");
    if (n_work <= 0) return ETM_OK;
    GramArgs a{cbuf, cbase, cwords, cld, grp_size, cand_off, work_groups, work_off, nullptr, n_work, n_tiles,
               chunk_base, cls, min_count, out_counts, surv_bits, work_counter, true, as_stream(stream)};
    a.grp_first = grp_first;
    a.row_counts = row_counts;
    return launch_gram_blocked(a);
}

extern "C" int etm_gram_block_members(int32_t elem) { return etm::gram_block_members(elem); }

namespace {
template <int FMT>
int mma_rate(int64_t iters, int* status, cudaStream_t s) {
    constexpr int smem = 3 * HALF_BYTES + 1024;
    ETM_CUDA(cudaFuncSetAttribute(mma_rate_kernel<FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    mma_rate_kernel<FMT><<<max(1, sm_count()), 128, smem, s>>>(iters, status);
    ETM_LAUNCHED("mma_rate");
    return ETM_OK;
}
}  // namespace

extern "C" int etm_tc_mma_rate(int32_t elem, int64_t iters, double* out_tflops, void* stream) {
    // Times `iters` MMAs per SM of the Gram's shape for `elem` on every SM (CUDA events on `stream`, which is
    // synchronized) and returns the dense rate in TFLOP/s: 2 M N K per MMA.
    const int e = elem & ~ETM_TC_WIDE;
    ETM_REQUIRE(e == 1 || e == 2 || e == ETM_TC_MXF4, ETM_EINVAL, "etm_tc_mma_rate: element code %d", elem);
    ETM_REQUIRE(iters > 0 && iters < (1LL << 32) && out_tflops != nullptr, ETM_EINVAL, "etm_tc_mma_rate: bad iters");
    cudaStream_t s = as_stream(stream);
    int* status = nullptr;
    ETM_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&status), g_tc_status));
    cudaEvent_t e0, e1;
    ETM_CUDA(cudaEventCreate(&e0));
    ETM_CUDA(cudaEventCreate(&e1));
    int st = ETM_OK;
    auto run = [&]() { return e == ETM_TC_MXF4 ? mma_rate<4>(iters, status, s) : e == 2 ? mma_rate<2>(iters, status, s)
                                                                                         : mma_rate<1>(iters, status, s); };
    st = run();  // warm-up
    if (st == ETM_OK) {
        cudaEventRecord(e0, s);
        st = run();
        cudaEventRecord(e1, s);
    }
    float ms = 0.f;
    if (st == ETM_OK) {
        const cudaError_t err = cudaEventSynchronize(e1);
        if (err != cudaSuccess) {
            etm::set_error("etm_tc_mma_rate: %s", cudaGetErrorString(err));
            st = ETM_ECUDA;
        } else {
            cudaEventElapsedTime(&ms, e0, e1);
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st != ETM_OK) return st;
    const double k = e == ETM_TC_MXF4 ? 64.0 : e == 1 ? 32.0 : 16.0;
    const double n = e == ETM_TC_MXF4 ? Fmt<4>::T : Fmt<1>::T;
    const double flops = 2.0 * 128.0 * n * k * (double)iters * (double)max(1, sm_count());
    *out_tflops = ms > 0.f ? flops / (ms * 1e-3) / 1e12 : 0.0;
    return ETM_OK;
}

extern "C" int etm_set_wait_limits(int64_t gram_first_wait_ns, int64_t proj_first_wait_ns) {
    {
        std::lock_guard<std::mutex> guard(g_cfg_lock);
        g_first_wait_ns = gram_first_wait_ns < 0 ? WAIT_NS : (uint64_t)gram_first_wait_ns;
    }
    etm::proj_set_first_wait(proj_first_wait_ns);
    return ETM_OK;
}

extern "C" int etm_device_status(void* stream) {
    // Both status words are read and cleared on every call, so a stale word never outlives the call
    // that reports it.
    int v = 0;
    ETM_CUDA(cudaMemcpyFromSymbolAsync(&v, g_tc_status, sizeof(int), 0, cudaMemcpyDeviceToHost, as_stream(stream)));
    ETM_CUDA(cudaStreamSynchronize(as_stream(stream)));
    if (v != 0) {
        const int zero = 0;
        ETM_CUDA(cudaMemcpyToSymbolAsync(g_tc_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, as_stream(stream)));
        ETM_CUDA(cudaStreamSynchronize(as_stream(stream)));
    }
    int p = 0;
    const int st = etm::proj_status_take(as_stream(stream), &p);
    if (st != ETM_OK) return st;
    if (v != 0 && p != 0)
        etm::set_error("a tensor-core counting kernel (status %d) and the projection (status %d) gave up bounded waits",
                       v, p);
    else if (v != 0)
        etm::set_error("a tensor-core counting kernel gave up a bounded wait (status %d)", v);
    else if (p == ETM_EINVAL)
        etm::set_error("the row-major projection met a member column past its row-major copy (status %d)", p);
    else if (p != 0)
        etm::set_error("the projection gave up a bounded wait for its bulk copies (status %d)", p);
    return v != 0 ? v : p;
}
