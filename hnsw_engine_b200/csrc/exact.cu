// Exact brute-force k-NN on B200 tensor cores (the reference's oracle.exact_search,
// src/hnsw_engine/oracle.py:35-126, re-designed for sm_100a).
//
// Algorithm (the reference's filter-then-rerank, with this kernel's own error bound):
//  1. prep: rows -> BF16 operands. Integer data with |v| <= 256 is exact in BF16 (one term). Other
//     data is split v = hi + lo (hi = bf16(v), lo = bf16(v - hi)) and the operands are concatenated
//     along K as Q' = [q_hi, q_hi, q_lo], X' = [x_hi, x_lo, x_hi], so one GEMM yields
//     hi.hi + hi.lo + lo.hi (relative error about 2^-16). Norms are computed in float64.
//  2. filter GEMM (tcgen05.mma kind::f16, BF16 x BF16 -> FP32 in TMEM, TMA-fed, warp specialised):
//     approx distance a = |q|^2 + |x|^2 - 2 q.x (l2), -q.x (ip) or 1 - q.x (cosine, on float64-
//     normalised rows); every (query, row) with a <= tau_q + margin_q is appended to the query's
//     candidate list. margin_q = 2 e_q where e_q bounds |a - exact| for this arithmetic, so every true
//     top-k row survives whenever tau_q is at least the k-th smallest approximate distance.
//  3. tau_q: pass one runs the filter on a sample of the data's tiles with tau = +inf, and a radix
//     select takes a low rank of its approximate distances (sample_rank): all but surely at or above
//     the k-th smallest of all rows, which pass two checks. Pass two filters all rows; a second
//     select tightens tau to the k-th smallest candidate.
//  4. rerank: float64 distances (sequential over dimensions) of the surviving candidates, best k by
//     (distance, id) -- ties to the lower id, as np.lexsort((ids, exact)) in the reference.
// Waits on mbarriers are bounded by a wall-clock limit; on expiry the kernel records an error,
// drains what it issued and frees its TMEM.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "hnsw_b200.h"
#include "scratch.cuh"
#include "split.cuh"

namespace hb {
int fail(int code, const std::string &msg);  // search.cu: records the thread's last error
}

namespace hbx {

constexpr int BM = 128;  // queries per tile (TMEM lanes)
constexpr int BN = 256;  // data rows per tile (TMEM columns per accumulator)
constexpr int BK = 64;   // K elements per stage (128 bytes of BF16: one swizzle-128B row)
constexpr int MAX_STAGES = 6;
constexpr int A_BYTES = BM * BK * 2;
constexpr int B_BYTES = BN * BK * 2;
// Epilogue warps: EPI_PER_QUARTER per TMEM lane quarter; each takes the two CW-column chunks
// part and part + EPI_PER_QUARTER of a tile, so every warp has the same work in every tile.
constexpr int EPI_PER_QUARTER = 4;
constexpr int EPI_WARPS = 4 * EPI_PER_QUARTER;
constexpr int CW = 32;  // columns per TMEM load
static_assert(BN == 2 * CW * EPI_PER_QUARTER, "two chunks a warp and tile");
constexpr int FILTER_THREADS = 128 + 32 * EPI_WARPS;
constexpr int BAR_BYTES = 512;  // barriers and flags after the operand buffers and the |x|^2 ring
constexpr int XSLOTS = 4;       // |x|^2 ring slots (one tile's BN values each)
constexpr int SMEM_MAX = 227 * 1024;
// Rows of at least COOP_DIM dimensions are re-scored by the whole warp, one candidate at a time.
constexpr int COOP_DIM = 256;
// Byte rows: one result in VERIFY_EVERY of each query is re-scored in float64 as a check.
constexpr int VERIFY_EVERY = 16;
constexpr uint32_t TMEM_COLS = 512;  // two accumulators of BN columns
constexpr unsigned long long WAIT_LIMIT_NS = 4000000000ull;  // 4 s

// UMMA instruction descriptor: BF16 A and B (K-major), FP32 accumulator, M = 128, N = 256.
constexpr uint32_t IDESC = (1u << 4)            // c_format F32
                           | (1u << 7)          // a_format BF16
                           | (1u << 10)         // b_format BF16
                           | (uint32_t(BN >> 3) << 17) | (uint32_t(BM >> 4) << 24);
// The same for byte rows (kind::i8): unsigned 8-bit A and B (formats 0), S32 accumulator (c_format
// 2). Integer products and sums are exact, so the filter values are the exact distances.
constexpr uint32_t IDESC_I8 = (2u << 4) | (uint32_t(BN >> 3) << 17) | (uint32_t(BM >> 4) << 24);
// Byte rows: a K chunk of one stage is 128 elements (one 128-byte swizzle row), 32 per instruction.
constexpr int BK8 = 128;
// Largest |distance| whose float value is exact (integers below 2^24).
constexpr float EXACT_LIM = 16777216.f;
// Filter value of a padding column in the byte path: above every distance the path admits.
constexpr int32_t I8_PAD = 0x3fffffff;

struct FilterParams {
    int32_t nq;            // valid queries
    int32_t row_end;       // one past the last data row
    int32_t tiles;         // tiles of BN rows in this pass: 0, tile_stride, 2 tile_stride, ...
    int32_t tile_stride;
    int32_t kchunks;       // K' / BK
    int32_t stages;        // operand stages in flight
    int32_t a_resident;    // the query tile's operand is loaded once and stays (else with each stage)
    int32_t tiles_per_split;
    int32_t block_tiles;   // threshold pass: tiles of a block of rows (see the pass), or 0: a block is four rows
    int32_t metric;
    const float *qq;       // |q|^2 per query (l2)
    const float *xx;       // per row: |x|^2 (l2) or 0; +inf past the data rows
    const int32_t *qqi;    // byte rows: exact |q|^2 per query (l2)
    const int32_t *xxi;    // byte rows: exact |x|^2 (l2) or 0; I8_PAD past the data rows
    const float *thr;      // per query: tau + margin (NULL: +inf, the threshold pass)
    // Candidates in segments: every epilogue thread of the grid owns one segment of its query's
    // list (segment = row split x epilogue part), so appends need no atomics. Segment s of query q
    // starts at (q * nseg + s) * cap.
    float *cand_val;       // (nq, nseg, cap) approximate distances
    int32_t *cand_id;      // (nq, nseg, cap) row ids
    int32_t *cand_cnt;     // (nq, nseg) appended counts (may exceed cap: overflow)
    int32_t cap;           // entries per segment
    int32_t mul;           // -2 (l2) or -1 (see EpiThread)
    int32_t *err;          // nonzero: a bounded wait expired
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One bounded probe of a barrier phase. The thread may be suspended by the hardware for up to
// MBAR_SUSPEND_NS while the phase is incomplete (instead of spinning on issue slots).
constexpr uint32_t MBAR_SUSPEND_NS = 100000;  // 0.1 ms
__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(MBAR_SUSPEND_NS)
        : "memory");
    return ok != 0;
}

// Bounded wait: false if the wall-clock limit expired (the caller records the error).
// The abort flag and the clock are read every 64th probe: a waiting thread then issues little
// besides the probes, leaving the issue slots to the warps that work.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
    if (mbar_try(bar, parity)) return true;
    const unsigned long long t0 = now_ns();
    for (uint32_t i = 1;; i++) {
        if (mbar_try(bar, parity)) return true;
        if ((i & 63u) == 0u) {
            if (*abort_flag) return false;
            if (now_ns() - t0 > WAIT_LIMIT_NS) return false;
        }
    }
}

__device__ __forceinline__ void tma_load_2d(const CUtensorMap *map, uint64_t *bar, void *dst, int x,
                                            int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, "
        "%4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// Plain (untiled, non-multicast) bulk copy of `bytes` from this GPU's global memory into shared
// memory, completing on bar: both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: rows of 128 bytes, 8-row groups
// 1024 bytes apart (stride byte offset), leading byte offset 16 bytes, descriptor version 1.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= uint64_t((saddr >> 4) & 0x3FFF);
    d |= uint64_t(1) << 16;            // leading byte offset (16 B) >> 4
    d |= uint64_t(1024 >> 4) << 32;    // stride byte offset >> 4
    d |= uint64_t(1) << 46;            // version
    d |= uint64_t(2) << 61;            // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(IDESC), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_u8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(IDESC_I8), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

// Issue a load of 32 accumulator columns; tmem_wait makes the registers readable (they are its
// operands, so no use of them can be moved before the wait).
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[CW]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
        "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
        "%30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait(uint32_t (&r)[CW]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
                   "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                   "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27])
                 :
                 : "memory");
    asm volatile("" : "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]) : : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]) : : "memory");
}

__device__ __forceinline__ int32_t min3(int32_t a, int32_t b, int32_t c) { return __vimin3_s32(a, b, c); }
__device__ __forceinline__ float min3(float a, float b, float c) { return fminf(fminf(a, b), c); }
__device__ __forceinline__ int32_t min2(int32_t a, int32_t b) { return min(a, b); }
__device__ __forceinline__ float min2(float a, float b) { return fminf(a, b); }

// What one epilogue thread (one query of the tile) carries through its chunks. A row's filter value is
// a = v + add with v = |x|^2 - 2 q.x (l2) or -q.x.
template <bool I8>
struct EpiThread {
    using V = std::conditional_t<I8, int32_t, float>;
    V add;       // |q|^2 (l2), 0 (ip), 1 (cosine)
    V thr;       // a candidate has v <= thr (byte path) or fl(v + add) <= thr (BF16 path)
    V mul;       // -2 (l2) or -1, from a kernel argument: on bytes that keeps the multiply-add on the FMA
                 // pipe (of a constant the compiler makes shifts and adds, on the pipe of the minima)
    float *cv;
    int32_t *ci;
    int cnt, cap;

    // x: the row's term from the ring: |x|^2 (l2) or 0; above every threshold past the data rows
    __device__ __forceinline__ V value(uint32_t r, uint32_t x) const {
        if constexpr (I8) return int32_t(r) * mul + int32_t(x);
        else return fmaf(mul, __uint_as_float(r), __uint_as_float(x));
    }
    __device__ __forceinline__ bool pass(V v) const {
        if constexpr (I8) return v <= thr;
        else return v + add <= thr;
    }

    // Minima of the groups of four of a chunk of CW accumulators, and of the chunk. xs: the terms of the
    // chunk's rows in shared memory (the same addresses in every lane).
    __device__ __forceinline__ V minima(const uint32_t (&r)[CW], const unsigned char *xs,
                                        V (&mg)[CW / 4]) const {
#pragma unroll
        for (int g = 0; g < CW / 4; g++) {
            const uint4 x = reinterpret_cast<const uint4 *>(xs)[g];
            mg[g] = min2(min3(value(r[4 * g], x.x), value(r[4 * g + 1], x.y), value(r[4 * g + 2], x.z)),
                         value(r[4 * g + 3], x.w));
        }
        return min3(min3(min3(mg[0], mg[1], mg[2]), mg[3], mg[4]), min2(mg[5], mg[6]), mg[7]);
    }

    // Threshold pass: keeps the first `count` of the block minima m.
    __device__ __forceinline__ void keep(const V (&m)[CW / 4], int count) {
#pragma unroll
        for (int g = 0; g < CW / 4; g++)
            if (g < count && cnt + g < cap) cv[cnt + g] = float(m[g] + add);
        cnt += count;
    }

    // Appends the chunk's candidates: of the groups of four that hold one for some query of the warp,
    // read again from TMEM (a loop of little code: unrolled over the chunk's registers, 16 diverging
    // warps ran out of the instruction cache and the pass took twice the time). Every lane calls it.
    __device__ __forceinline__ void append(uint32_t taddr, const unsigned char *xs, int col0, int valid,
                                           const V (&mg)[CW / 4]) {
        uint32_t gm = 0;
#pragma unroll
        for (int g = 0; g < CW / 4; g++) gm |= pass(mg[g]) ? 1u << g : 0u;
        gm = __reduce_or_sync(0xffffffffu, gm);
#pragma unroll 1
        for (; gm; gm &= gm - 1) {
            const int g = __ffs(gm) - 1;
            uint32_t r[4];
            tmem_ld4(taddr + uint32_t(4 * g), r);
            const uint4 x = reinterpret_cast<const uint4 *>(xs)[g];
            const V v[4] = {value(r[0], x.x), value(r[1], x.y), value(r[2], x.z), value(r[3], x.w)};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (pass(v[j]) && 4 * g + j < valid) {
                    if (cnt < cap) {
                        cv[cnt] = float(v[j] + add);
                        ci[cnt] = col0 + 4 * g + j;
                    }
                    cnt++;
                }
            }
            // The lanes part above, and the TMEM instructions that follow (the next group's load, the
            // caller's wait) are .aligned: the whole warp has to execute them together.
            __syncwarp();
        }
    }
};

// The filter pass. What bounds it is the epilogue: a tile is 128 queries x 256 rows, its MMAs take 512
// cycles of the tensor pipe on bytes at d = 128, and its 32,768 values go through 16 epilogue warps
// in about 2,300 (1,024 queries x 1M rows under ncu: 489,000 cycles for 212 tiles an SM; issue slots 51% busy,
// tensor pipe 22%, 146 warp instructions a chunk of 32 columns). So a warp takes exactly two chunks of a tile and loads the second while it
// works on the first, a value costs one multiply-add (on the FMA pipe) and at most one minimum, rows past
// the data carry a term above every threshold instead of a test on each value, and candidates are looked
// for by groups of four in a small loop. The query tile's operand stays in shared memory over a
// CTA's tiles wherever three stages of rows fit beside it (up to seven 128-byte chunks of K), else it
// comes again with every tile. 10K queries x 1M x 128 bytes, both passes: 5.68 -> 2.60 ms; 1,000
// x 200K x 100 floats: 177 -> 145 us.
// I8: byte rows on kind::i8 (exact integer filter values); otherwise BF16 terms on kind::f16.
// BMIN: the threshold pass over the sample, which keeps block minima only.
template <bool I8, bool BMIN>
__global__ void __launch_bounds__(FILTER_THREADS, 1)
    knn_filter_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const FilterParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // 1024-byte aligned operand buffers (swizzle-128B atoms): the resident query operand, the stages;
    // then |x|^2 of a tile's BN rows (float or int32, 4 bytes each) in a ring of XSLOTS (the
    // producer fills slot lt % XSLOTS, the epilogue reads it and releases it); then the barriers.
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int nst = p.stages;
    const int a_bytes = p.a_resident ? p.kchunks * A_BYTES : 0;
    const int stage_bytes = p.a_resident ? B_BYTES : A_BYTES + B_BYTES;
    unsigned char *stages = smem + a_bytes;
    unsigned char *xring = stages + nst * stage_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(xring + XSLOTS * BN * 4);
    uint64_t *empty = full + MAX_STAGES;
    uint64_t *tfull = empty + MAX_STAGES;
    uint64_t *tempty = tfull + 2;
    uint64_t *xfull = tempty + 2;
    uint64_t *xempty = xfull + XSLOTS;
    uint64_t *afull = xempty + XSLOTS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(afull + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int qt = blockIdx.x;
    const int t0 = blockIdx.y * p.tiles_per_split;
    const int t1 = min(p.tiles, t0 + p.tiles_per_split);
    const int ntiles = max(0, t1 - t0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < nst; s++) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(tfull + b, 1);
            mbar_init(tempty + b, EPI_WARPS);
        }
        for (int x = 0; x < XSLOTS; x++) {
            mbar_init(xfull + x, 1);
            mbar_init(xempty + x, EPI_WARPS);
        }
        mbar_init(afull, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0 && lane == 0) {
        // ---------------------------------------------------------------- TMA producer
        int it = 0, xs = 0;  // stages and |x|^2 slots issued
        bool ok = true;
        const bool a_once = p.a_resident && ntiles > 0;
        if (a_once) {
            mbar_expect_tx(afull, uint32_t(p.kchunks) * A_BYTES);
            for (int kc = 0; kc < p.kchunks; kc++)
                tma_load_2d(&tmA, afull, smem + kc * A_BYTES, kc * (I8 ? BK8 : BK), qt * BM);
        }
        int s = 0;
        uint32_t par = 1;  // of the stage's release
        for (int lt = 0; lt < ntiles && ok; lt++) {
            const int row0 = (t0 + lt) * p.tile_stride * BN;
            {  // the tile's |x|^2 (rows row0 .. row0 + BN - 1 < n_pad) into its ring slot
                const int x = lt % XSLOTS;
                if (!mbar_wait(xempty + x, ((lt / XSLOTS) & 1) ^ 1, abort_flag)) {
                    ok = false;
                    break;
                }
                mbar_expect_tx(xfull + x, BN * 4);
                const void *src = I8 ? static_cast<const void *>(p.xxi + row0)
                                     : static_cast<const void *>(p.xx + row0);
                bulk_load(xring + x * BN * 4, src, BN * 4, xfull + x);
                xs++;
            }
            for (int kc = 0; kc < p.kchunks; kc++, it++) {
                if (!mbar_wait(empty + s, par, abort_flag)) {
                    ok = false;
                    break;
                }
                unsigned char *b = stages + s * stage_bytes;
                mbar_expect_tx(full + s, uint32_t(stage_bytes));
                tma_load_2d(&tmB, full + s, b, kc * (I8 ? BK8 : BK), row0);
                if (!p.a_resident)
                    tma_load_2d(&tmA, full + s, b + B_BYTES, kc * (I8 ? BK8 : BK), qt * BM);
                if (++s == nst) {
                    s = 0;
                    par ^= 1;
                }
            }
        }
        if (!ok) {
            atomicExch(p.err, 1);
            *abort_flag = 1;
        }
        // Drain: everything issued must land before the CTA may exit.
        auto drain = [&](uint64_t *bar, uint32_t parity) {
            const unsigned long long t = now_ns();
            while (!mbar_try(bar, parity) && now_ns() - t < WAIT_LIMIT_NS) {
            }
        };
        for (int j = max(0, it - nst); j < it; j++) drain(full + j % nst, (j / nst) & 1);
        for (int j = max(0, xs - XSLOTS); j < xs; j++) drain(xfull + j % XSLOTS, (j / XSLOTS) & 1);
        if (a_once) drain(afull, 0);
    } else if (warp == 1 && lane == 0) {
        // ---------------------------------------------------------------- MMA issuer
        int it = 0;
        bool ok = true;
        if (p.a_resident && ntiles > 0) ok = mbar_wait(afull, 0, abort_flag);
        int s = 0, last = 0;
        uint32_t par = 0, last_par = 0;
        for (int lt = 0; lt < ntiles && ok; lt++) {
            const int b = lt & 1;
            if (!mbar_wait(tempty + b, ((lt >> 1) & 1) ^ 1, abort_flag)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tmem_d = tmem_base + uint32_t(b * BN);
            for (int kc = 0; kc < p.kchunks; kc++, it++) {
                if (!mbar_wait(full + s, par, abort_flag)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t b_addr = smem_u32(stages + s * stage_bytes);
                const uint32_t a_addr = p.a_resident ? smem_u32(smem + kc * A_BYTES) : b_addr + B_BYTES;
#pragma unroll
                for (int j = 0; j < 4; j++) {  // 32 bytes of K per instruction (16 BF16 or 32 bytes)
                    if constexpr (I8)
                        umma_u8(tmem_d, sw128_desc(a_addr + j * 32), sw128_desc(b_addr + j * 32),
                                (kc | j) != 0);
                    else
                        umma_bf16(tmem_d, sw128_desc(a_addr + j * 32), sw128_desc(b_addr + j * 32),
                                  (kc | j) != 0);
                }
                umma_commit(empty + s);
                last = s;
                last_par = par;
                if (++s == nst) {
                    s = 0;
                    par ^= 1;
                }
            }
            if (ok) umma_commit(tfull + b);
        }
        if (!ok) {
            atomicExch(p.err, 1);
            *abort_flag = 1;
        }
        // Every MMA issued must finish before TMEM is released: wait for the last stage's commit
        // (tcgen05.commit tracks all prior MMAs of this thread).
        if (it > 0) {
            const unsigned long long t = now_ns();
            while (!mbar_try(empty + last, last_par) && now_ns() - t < WAIT_LIMIT_NS) {
            }
        }
    } else if (warp >= 4) {
        // ---------------------------------------------------------------- epilogue
        // Warp w reads TMEM lanes 32 (w % 4) .. +31 (its hardware lane quarter: one query per
        // thread) and the chunks part and part + EPI_PER_QUARTER of each accumulator.
        const int quarter = warp & 3;
        const int part = (warp - 4) >> 2;  // 0 .. EPI_PER_QUARTER - 1
        const int row = quarter * 32 + lane;  // TMEM lane = query row of the tile
        const int q = qt * BM + row;
        const int nseg = int(gridDim.y) * EPI_PER_QUARTER;
        EpiThread<I8> E;
        const bool qvalid = q < p.nq, l2 = p.metric == HNSW_B200_L2;
        const float thr = !qvalid ? -INFINITY : p.thr ? p.thr[q] : INFINITY;
        if constexpr (I8) {
            E.add = qvalid && l2 ? p.qqi[q] : 0;
            E.mul = p.mul;
            // Largest v whose float distance fl(v + add) may be <= thr: exact below 2^24; above it a
            // float is the rounding of integers up to 64 away, so the bound is widened (a few rows
            // beyond the threshold then join the candidates). No value for -inf or NaN.
            const double t = double(thr);
            const double w = floor(fmin(fmax(t, -2147483648.0), 2147483647.0)) - double(E.add) +
                             (fabs(t) >= 16777216.0 ? 128.0 : 0.0);
            E.thr = !(t > -INFINITY) ? INT32_MIN
                                     : int32_t(fmax(fmin(w, double(I8_PAD - 1)), -2147483647.0));
        } else {
            E.add = !qvalid ? 0.f : l2 ? p.qq[q] : (p.metric == HNSW_B200_COSINE ? 1.f : 0.f);
            E.mul = float(p.mul);
            E.thr = thr;
        }
        const int64_t seg = int64_t(qvalid ? q : 0) * nseg + int64_t(blockIdx.y) * EPI_PER_QUARTER + part;
        E.cv = p.cand_val + seg * p.cap;
        E.ci = p.cand_id + seg * p.cap;
        E.cap = p.cap;
        E.cnt = 0;  // this thread's appends (its own segment: no atomics)
        const int c0 = part * CW, c1 = c0 + CW * EPI_PER_QUARTER;
        typename EpiThread<I8>::V bm[CW / 4];  // threshold pass: the current blocks' minima
        for (int lt = 0; lt < ntiles; lt++) {
            const int b = lt & 1;
            const int row0 = (t0 + lt) * p.tile_stride * BN;
            const bool ok = mbar_wait(xfull + lt % XSLOTS, (lt / XSLOTS) & 1, abort_flag) &&
                            mbar_wait(tfull + b, (lt >> 1) & 1, abort_flag);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) {
                    atomicExch(p.err, 1);
                    *abort_flag = 1;
                }
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // TMEM columns of this warp's lane quarter in accumulator b; the tile's |x|^2 in its slot
            const uint32_t tbase = tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(b * BN);
            const unsigned char *xslot = xring + (lt % XSLOTS) * BN * 4;
            const int valid0 = p.row_end - row0 - c0, valid1 = p.row_end - row0 - c1;
            uint32_t r0[CW], r1[CW];
            typename EpiThread<I8>::V mg[CW / 4];
            tmem_ld(tbase + uint32_t(c0), r0);
            tmem_wait(r0);
            tmem_ld(tbase + uint32_t(c1), r1);  // in flight while the first chunk is worked on
            const auto m0 = E.minima(r0, xslot + c0 * 4, mg);
            if constexpr (BMIN) {
                if (p.block_tiles == 0) {
                    if (qvalid) E.keep(mg, CW / 4);
                } else if ((lt & (p.block_tiles - 1)) == 0) {
#pragma unroll
                    for (int g = 0; g < CW / 4; g++) bm[g] = mg[g];
                } else {
#pragma unroll
                    for (int g = 0; g < CW / 4; g++) bm[g] = min2(bm[g], mg[g]);
                }
            }
            if (!BMIN && __any_sync(0xffffffffu, E.pass(m0)))
                E.append(tbase + uint32_t(c0), xslot + c0 * 4, row0 + c0, valid0, mg);
            tmem_wait(r1);
            const auto m1 = E.minima(r1, xslot + c1 * 4, mg);
            if (!BMIN && __any_sync(0xffffffffu, E.pass(m1)))
                E.append(tbase + uint32_t(c1), xslot + c1 * 4, row0 + c1, valid1, mg);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(tempty + b);
                mbar_arrive(xempty + lt % XSLOTS);
            }
            // Threshold pass: one value per block, its minimum. A block is the g-th groups of four columns of
            // this thread's chunks of block_tiles tiles: of rows in any order as good as one of neighbouring
            // rows, and where near rows are neighbours (rows stored by cluster or by time) they are in many
            // blocks and not in one (10K queries x 1M x 128 bytes in runs of 1,000 similar rows, k = 100: 10.8 ->
            // 7.6 ms; 500K x 64 in tight ones, inner product, 1,000 queries, k = 10: 1.54 -> 1.03). The r-th smallest of the blocks' minima is at least the r-th smallest of all
            // the values (a subset's r-th is never below the set's), and nearly as tight where there are at
            // least twice as many blocks (see the host). Values only: the pass needs no row ids.
            if constexpr (BMIN) {
                if (p.block_tiles == 0) {
                    if (qvalid) E.keep(mg, CW / 4);
                } else {
#pragma unroll
                    for (int g = 0; g < CW / 4; g++) bm[g] = min2(bm[g], mg[g]);
                    const int in = lt & (p.block_tiles - 1);
                    if (in == p.block_tiles - 1 || lt + 1 == ntiles) {
                        // Fewer tiles than block_tiles (the CTA's last ones): as many fewer blocks.
                        int count = CW / 4;
                        if (2 * (in + 1) <= p.block_tiles) {
                            count = 4;
#pragma unroll
                            for (int g = 0; g < 4; g++) bm[g] = min2(bm[g], bm[g + 4]);
                        }
                        if (4 * (in + 1) <= p.block_tiles) {
                            count = 2;
                            bm[0] = min2(bm[0], bm[2]);
                            bm[1] = min2(bm[1], bm[3]);
                        }
                        if (8 * (in + 1) <= p.block_tiles) {
                            count = 1;
                            bm[0] = min2(bm[0], bm[1]);
                        }
                        if (qvalid) E.keep(bm, count);
                    }
                }
            }
        }
        if (qvalid) p.cand_cnt[seg] = E.cnt;
    }
    __syncthreads();
    if (warp == 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(TMEM_COLS));
    }
}

// ------------------------------------------------------------------------------------- prep
// Four values of a byte row from element i, as bytes of a word (zero past dim). vec: the row starts on a
// boundary of four elements and dim is a multiple of 4, so one load fetches them.
__device__ __forceinline__ uint32_t byte_word(const uint8_t *x, int i, int dim, bool vec) {
    if (vec) return i < dim ? __ldg(reinterpret_cast<const uint32_t *>(x + i)) : 0u;
    uint32_t word = 0;
#pragma unroll
    for (int t = 0; t < 4; t++) word |= (i + t < dim ? uint32_t(x[i + t]) : 0u) << (8 * t);
    return word;
}
__device__ __forceinline__ uint32_t byte_word(const float *x, int i, int dim, bool vec) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (vec && i < dim) {
        const float4 f = __ldg(reinterpret_cast<const float4 *>(x + i));
        v[0] = f.x;
        v[1] = f.y;
        v[2] = f.z;
        v[3] = f.w;
    } else if (!vec) {
#pragma unroll
        for (int t = 0; t < 4; t++)
            if (i + t < dim) v[t] = x[i + t];
    }
    uint32_t word = 0;
#pragma unroll
    for (int t = 0; t < 4; t++) word |= uint32_t(int32_t(v[t]) & 255) << (8 * t);
    return word;
}

// Byte rows (values checked to be integers in [0, 255]): a warp writes the u8 operand rows of width
// kpad (a multiple of 128, zero past dim), four bytes a lane, and sq: the exact |x|^2 (norms; else 0; `past` beyond the rows), four rows at a time
// so that their loads overlap (bound by memory: 1M x 128 bytes 112 -> 71 us, a row and a byte at a time before).
template <typename T>
__global__ void prep_rows_u8(const T *src, int64_t rows, int dim, int64_t rows_pad, int kpad,
                             uint8_t *dst, int32_t *sq, bool vec, bool norms, int32_t past) {
    constexpr int R = 4;
    const int lane = threadIdx.x & 31;
    const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
    for (int64_t r = (int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * R; r < rows_pad;
         r += warps * R) {
        uint32_t ss[R] = {0u, 0u, 0u, 0u};
        for (int i = lane * 4; i < kpad; i += 128) {
            uint32_t w[R];
#pragma unroll
            for (int t = 0; t < R; t++) w[t] = r + t < rows ? byte_word(src + (r + t) * dim, i, dim, vec) : 0u;
#pragma unroll
            for (int t = 0; t < R; t++) {
                ss[t] = __dp4a(w[t], w[t], ss[t]);
                if (r + t < rows_pad) *reinterpret_cast<uint32_t *>(dst + (r + t) * kpad + i) = w[t];
            }
        }
#pragma unroll
        for (int t = 0; t < R; t++) {
            const uint32_t sum = __reduce_add_sync(0xffffffffu, ss[t]);
            if (lane == 0 && r + t < rows_pad) sq[r + t] = r + t >= rows ? past : norms ? int32_t(sum) : 0;
        }
    }
}

// One warp per row: float64 norm, cosine normalisation, BF16 operand row(s) of width kpad, and sq32:
// |x|^2 (norms; else 0; `past` beyond the rows). terms == 1: [v]; terms == 3: A-side [hi, hi, lo]
// (queries) or B-side [hi, lo, hi] (data). A lane keeps up to PREP_REGS values of its row in registers, so
// that a value is read once (bound by memory and the row's latency; 200K x 100 floats: 86 -> 65 us, and
// 105 us with four rows a warp).
constexpr int PREP_REGS = 4;
template <typename T>
__global__ void prep_rows(const T *src, int64_t rows, int dim, int64_t rows_pad, int kpad,
                          int terms, int a_side, int cosine, __nv_bfloat16 *dst, double *norm64,
                          float *sq32, bool norms, float past) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    const int seg = kpad / terms;  // padded dim per term
    for (int64_t r = warp; r < rows_pad; r += nwarps) {
        const T *xr = src + r * dim;
        auto value = [&](int i) { return r < rows && i < dim ? float(xr[i]) : 0.f; };
        float x[PREP_REGS];
#pragma unroll
        for (int t = 0; t < PREP_REGS; t++) x[t] = value(lane + 32 * t);
        double ss = 0.0;
#pragma unroll
        for (int t = 0; t < PREP_REGS; t++) ss += double(x[t]) * double(x[t]);
        for (int i = lane + 32 * PREP_REGS; i < dim; i += 32) {
            const double v = double(value(i));
            ss += v * v;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const double nrm = sqrt(ss);
        const double scale = cosine ? (nrm > 0 ? 1.0 / nrm : 0.0) : 1.0;
        __nv_bfloat16 *out = dst + r * kpad;
        auto put = [&](int i, float raw) {
            const double v = double(raw) * scale;
            const __nv_bfloat16 hi = __float2bfloat16_rn(float(v));
            out[i] = hi;
            if (terms != 1) {
                const __nv_bfloat16 lo = __float2bfloat16_rn(float(v - double(__bfloat162float(hi))));
                out[seg + i] = a_side ? hi : lo;
                out[2 * seg + i] = a_side ? lo : hi;
            }
        };
#pragma unroll
        for (int t = 0; t < PREP_REGS; t++)
            if (lane + 32 * t < seg) put(lane + 32 * t, x[t]);
        for (int i = lane + 32 * PREP_REGS; i < seg; i += 32) put(i, value(i));
        if (lane == 0) {
            norm64[r] = nrm;  // cosine rerank re-normalises with it; margins use 1 for cosine
            sq32[r] = r >= rows ? past : norms ? float(ss) : 0.f;
        }
    }
}

// ------------------------------------------------------------------------------ radix select
// Order-preserving key of a float (ascending floats -> ascending unsigned keys).
__device__ __forceinline__ uint32_t fkey(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float funkey(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Moves one query's candidates (segments of `cap` entries, counts in cnt) to the front of its
// region, in segment order, by one warp; returns how many there are. In place: an entry's new index
// (its rank in segment order) is never above its old one, and the warp moves the entries in rank
// order, 32 at a time, reading a batch before writing it, so no entry is overwritten before it has
// moved. A lane finds its entry's segment by a binary search over the 32 segment offsets of the
// group (shuffles).
__device__ __forceinline__ int compact_list(float *v, int32_t *id, const int32_t *cnt, int32_t cap,
                                            int32_t nseg, int lane) {
    int base = 0;
    for (int s0 = 0; s0 < nseg; s0 += 32) {
        const int sg = s0 + lane;
        const int n_sg = sg < nseg ? min(cnt[sg], cap) : 0;
        int incl = n_sg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const int excl = incl - n_sg;
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        for (int b = 0; b < total; b += 32) {
            const int r = b + lane;  // rank within the group
            int lo = 0;  // last segment of the group whose offset is <= r (every lane searches)
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int e = __shfl_sync(0xffffffffu, excl, min(lo + step, 31));
                if (lo + step < 32 && e <= r) lo += step;
            }
            const int off = __shfl_sync(0xffffffffu, excl, lo);
            float val = 0.f;
            int32_t ident = 0;
            if (r < total) {
                const int64_t src = int64_t(s0 + lo) * cap + (r - off);
                val = v[src];
                if (id) ident = id[src];
            }
            __syncwarp();
            if (r < total) {
                v[base + r] = val;
                if (id) id[base + r] = ident;
            }
            __syncwarp();
        }
        base += total;
    }
    return base;
}

// One warp per query, 8 per block: tau[q] = k-th smallest of the candidate values (or +inf if
// fewer than k), then out_thr[q] = tau + margin[q]. A 4-pass radix select, 8 bits a pass, over the
// query's segments; the bin of the rank-th key comes from each lane's 8 bins and a warp scan.
constexpr int SELECT_WARPS = 8;
// The query's list is first compacted in place (compact_list) and its length stored in
// cand_m[q], so the radix passes and the re-rank read one dense run of entries.
// step SELECT_FIRST: the list is pass one's. SELECT_TIGHTEN: it is what pass two could keep before segments
// overflowed; the threshold becomes the k-th smallest of that where it is lower (a subset's k-th is never below
// the set's). SELECT_FINAL: the list is pass two's, out_tau holds the threshold it was collected with (without the
// margin), and *short_lists is set when that threshold turns out too low: fewer than k entries, or
// a k-th smallest above it. stat_max: largest |value| the error bound is stated for (byte rows: the
// finite final thresholds; else the margins), as float bits. longest (final step): the longest segment count;
// where lists overflowed they are collected again, and nothing here is worth doing.
enum SelectStep : int { SELECT_FIRST, SELECT_FINAL, SELECT_TIGHTEN };
__global__ void select_kth(float *cand_val, int32_t *cand_id, const int32_t *cand_cnt, int32_t cap,
                           int32_t nseg, int32_t nq, int32_t k, const float *margin, float *out_thr,
                           float *out_tau, int32_t *cand_m, SelectStep step, int bytes,
                           int32_t *short_lists, unsigned int *stat_max, const unsigned long long *longest) {
    __shared__ uint32_t hist_all[SELECT_WARPS][256];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * SELECT_WARPS + wid;
    if (q >= nq || (longest && *longest > static_cast<unsigned long long>(cap))) return;  // no block-wide barrier below
    uint32_t *hist = hist_all[wid];
    float *v = cand_val + int64_t(q) * nseg * cap;
    const int m = compact_list(v, cand_id ? cand_id + int64_t(q) * nseg * cap : nullptr,
                               cand_cnt + int64_t(q) * nseg, cap, nseg, lane);
    if (lane == 0) cand_m[q] = m;
    if (m < k) {
        if (lane == 0 && step != SELECT_TIGHTEN) {
            if (step == SELECT_FINAL) atomicOr(short_lists, 1);
            out_tau[q] = INFINITY;
            out_thr[q] = INFINITY;
        }
        return;
    }
    uint32_t prefix = 0, rank = uint32_t(k);  // rank: 1-based position within the current bucket
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int i = lane; i < 256; i += 32) hist[i] = 0;
        __syncwarp();
        const uint32_t hmask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
        for (int i = lane; i < m; i += 32) {
            const uint32_t key = fkey(v[i]);
            if ((key & hmask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
        }
        __syncwarp();
        uint32_t c[8], sum = 0;
#pragma unroll
        for (int b = 0; b < 8; b++) {
            c[b] = hist[lane * 8 + b];
            sum += c[b];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        uint32_t run = incl - sum, bucket = 0, nrank = 0;
        const bool mine = run < rank && rank <= incl;  // exactly one lane
        if (mine) {
#pragma unroll
            for (int b = 0; b < 8; b++) {
                if (nrank == 0 && run + c[b] >= rank) {
                    bucket = uint32_t(lane * 8 + b);
                    nrank = rank - run;
                }
                run += c[b];
            }
        }
        const int src = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
        bucket = __shfl_sync(0xffffffffu, bucket, src);
        nrank = __shfl_sync(0xffffffffu, nrank, src);
        prefix |= bucket << shift;
        rank = nrank;
        __syncwarp();
    }
    if (lane == 0) {
        const float tau = funkey(prefix), mg = margin[q];
        if (step == SELECT_TIGHTEN && !(tau < out_tau[q])) return;
        if (step == SELECT_FINAL) {
            if (!(tau <= out_tau[q])) atomicOr(short_lists, 1);
            const float b = bytes ? fabsf(tau + mg) : mg;
            const unsigned int bits = isfinite(b) || !bytes ? __float_as_uint(b) : 0u;
            if (bits > *static_cast<volatile unsigned int *>(stat_max)) atomicMax(stat_max, bits);
        }
        out_tau[q] = tau;
        out_thr[q] = tau + mg;
    }
}

// ------------------------------------------------------------------------------------ rerank
// (distance, id) order of numbers.
__device__ __forceinline__ bool below(double da, int32_t ia, double db, int32_t ib) {
    return da < db || (da == db && ia < ib);
}
// The same with NaN distances last, by id among themselves (a zero row or query under cosine divides by
// zero): a total order, as placing a result by counting the ones below it needs.
__device__ __forceinline__ bool pair_lt(double da, int32_t ia, double db, int32_t ib) {
    return isnan(db) ? !isnan(da) || ia < ib : below(da, ia, db, ib);
}

// Float64 distance of row x to the query qv by one lane, the sums in dimension order.
template <typename T>
__device__ __forceinline__ double dist_f64_lane(const T *x, const T *qv, int dim, int metric,
                                                double xn, double qn) {
    double acc = 0.0;
    if (metric == HNSW_B200_L2) {
        for (int j = 0; j < dim; j++) {
            const double df = __dsub_rn(double(x[j]), double(qv[j]));
            acc = __dadd_rn(acc, __dmul_rn(df, df));
        }
        return acc;
    }
    if (metric == HNSW_B200_IP) {
        for (int j = 0; j < dim; j++) acc = __dadd_rn(acc, __dmul_rn(double(x[j]), double(qv[j])));
        return -acc;
    }
    for (int j = 0; j < dim; j++)
        acc = __dadd_rn(acc, __dmul_rn(__ddiv_rn(double(x[j]), xn), __ddiv_rn(double(qv[j]), qn)));
    return __dsub_rn(1.0, acc);
}

// The same by the whole warp (long rows): lane l sums dimensions l, l + 32, ..., then a fixed
// shuffle tree adds the lanes (the same value on every run; on integer data every order gives the
// same exact sum), so the float64 chains are 32 times shorter. The result is on every lane.
template <typename T>
__device__ __forceinline__ double dist_f64_warp(const T *x, const T *qv, int dim, int metric,
                                                double xn, double qn, int lane) {
    double acc = 0.0;
    if (metric == HNSW_B200_L2) {
        for (int i = lane; i < dim; i += 32) {
            const double df = __dsub_rn(double(x[i]), double(qv[i]));
            acc = __dadd_rn(acc, __dmul_rn(df, df));
        }
    } else if (metric == HNSW_B200_IP) {
        for (int i = lane; i < dim; i += 32) acc = __dadd_rn(acc, __dmul_rn(double(x[i]), double(qv[i])));
    } else {
        for (int i = lane; i < dim; i += 32)
            acc = __dadd_rn(acc, __dmul_rn(__ddiv_rn(double(x[i]), xn), __ddiv_rn(double(qv[i]), qn)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = __dadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    return metric == HNSW_B200_L2 ? acc : (metric == HNSW_B200_IP ? -acc : __dsub_rn(1.0, acc));
}

// Survivors (candidates within the final threshold) of a query that rerank_topk gathers in shared
// memory and sorts there; a query with more (many exact ties) inserts them one by one.
__host__ __device__ constexpr int survivor_slots(int k) { return k + k / 4 + 64; }
// Shared memory of one warp of rerank_topk: distances and ids of the results and of the survivors, and a
// queue of 64 survivors for the insertion.
__host__ __device__ inline size_t rerank_smem(int k, bool gather) {
    return (size_t(k + 1 + (gather ? survivor_slots(k) : 0)) * 12 + 64 * 8 + 15) & ~size_t(15);
}

// One warp per query: exact float64 distances of the candidates within the final threshold,
// best k by (distance, id), written as int64 / float64.
// gather: the survivors are first collected in shared memory (most candidates fail the final threshold:
// scored in batches of candidates, a float64 chain ran for one or two of 32 lanes), scored 32 at a
// time and placed by counting the ones below each: about k^2 / 32 steps, against k insertions of about 80
// instructions. 10K queries x 1M x 128 bytes, k = 100: 332 -> 102 us. Where the slots would leave too few warps
// (the host's choice) or with more survivors than slots (ties), sorted insertion.
// exact_lim > 0 (byte rows, integer filter): a candidate whose filter value is below exact_lim in
// magnitude already holds its exact distance and is not re-scored; one result in VERIFY_EVERY of
// every query (positions q, q + VERIFY_EVERY, ... mod VERIFY_EVERY, so a batch covers every
// position) is re-scored in float64 at the end instead, and any difference sets *mismatch. (Re-scoring every query's results cost 0.55 ms of 8.6 on the 1M x 128 mixture and
// 0.63 of 2.6 on the 60K x 784 set, 10K queries each; integer products and sums are exact, so
// the check is there to catch a wrong operand layout or descriptor, which a sample shows.)
// longest, short_lists (NULL: not looked at): as for select_kth; lists that overflowed or came from too low a
// threshold are collected again, and their results would be thrown away. 10K queries x 1M x 128 bytes in runs of
// 1,000 similar rows, k = 100: 12.9 -> 12.4 ms; 2,000 x 60K x 784 floats in runs of 600: 3.77 -> 2.84 ms.
template <typename T>
__global__ void rerank_topk(const T *data, const T *queries, int dim, int32_t nq, int32_t k,
                            int32_t metric, const double *xnorm, const double *qnorm,
                            const float *cand_val, const int32_t *cand_id, const int32_t *cand_m,
                            int32_t cap, int32_t nseg, const float *thr, int64_t *out_ids,
                            double *out_d, unsigned long long *err_max, float exact_lim,
                            int32_t *mismatch, int gather, const unsigned long long *longest,
                            const int32_t *short_lists) {
    extern __shared__ __align__(16) unsigned char sm[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * (blockDim.x >> 5) + w;
    if (q >= nq || *longest > static_cast<unsigned long long>(cap) || (short_lists && *short_lists))
        return;  // no block-wide barrier below
    const int slots = gather ? survivor_slots(k) : 0;
    unsigned char *base = sm + size_t(w) * rerank_smem(k, gather);
    double *Ad = reinterpret_cast<double *>(base);       // results
    double *Sd = Ad + k + 1;                             // survivors
    int32_t *Ai = reinterpret_cast<int32_t *>(Sd + slots);
    int32_t *Si = Ai + k + 1;
    float *Wv = reinterpret_cast<float *>(Si + slots);   // the queue
    int32_t *Wi = reinterpret_cast<int32_t *>(Wv + 64);
    const float t = thr[q];
    const T *qv = queries + int64_t(q) * dim;
    const bool cos = metric == HNSW_B200_COSINE;
    const double qn = cos ? qnorm[q] : 1.0;
    int a = 0;
    double err = 0.0;  // largest |filter value - exact distance| over this lane's re-scored survivors
    // The query's candidates, compacted by select_kth to the front of its region: batches of 32,
    // one per lane.
    const int m = cand_m[q];
    const int64_t region = int64_t(q) * nseg * cap;
    int ns = -1;  // survivors gathered (-1: insert one by one)
    if (gather) {
        ns = 0;
        for (int b0 = 0; b0 < m; b0 += 32) {
            const bool in = b0 + lane < m;
            const float approx = in ? cand_val[region + b0 + lane] : INFINITY;
            const bool has = in && approx <= t;
            const uint32_t hm = __ballot_sync(0xffffffffu, has);
            const int at = ns + __popc(hm & ((1u << lane) - 1u));
            if (has && at < slots) {
                Sd[at] = double(approx);
                Si[at] = cand_id[region + b0 + lane];
            }
            ns += __popc(hm);
            if (ns > slots) break;  // uniform
        }
        if (ns > slots) ns = -1;
        __syncwarp();
    }
    if (ns >= 0) {
        for (int b0 = 0; b0 < ns; b0 += 32) {
            const int s = b0 + lane;
            const double approx = s < ns ? Sd[s] : 0.0;
            const bool need = s < ns && !(fabs(approx) < double(exact_lim));
            const uint32_t nm = __ballot_sync(0xffffffffu, need);
            if (!nm) continue;  // uniform
            double d = approx;
            if (dim >= COOP_DIM) {
                for (uint32_t hm = nm; hm; hm &= hm - 1) {
                    const int j = __ffs(hm) - 1;
                    const int32_t idj = Si[b0 + j];
                    const double dd = dist_f64_warp(data + int64_t(idj) * dim, qv, dim, metric,
                                                    cos ? xnorm[idj] : 1.0, qn, lane);
                    if (lane == j) d = dd;
                }
            } else if (need) {
                d = dist_f64_lane(data + int64_t(Si[s]) * dim, qv, dim, metric, cos ? xnorm[Si[s]] : 1.0, qn);
            }
            if (need) {
                err = fmax(err, fabs(approx - d));
                Sd[s] = d;
            }
        }
        __syncwarp();
        for (int s = lane; s < ns; s += 32) {
            const double d = Sd[s];
            const int32_t id = Si[s];
            int pos = 0;
            for (int j = 0; j < ns; j++) pos += below(Sd[j], Si[j], d, id);
            if (isnan(d)) {  // apart: a test in the loop above cost 40 us of the 10K x 1M byte case
                pos = 0;
                for (int j = 0; j < ns; j++) pos += pair_lt(Sd[j], Si[j], d, id);
            }
            if (pos < k) {
                Ad[pos] = d;
                Ai[pos] = id;
            }
        }
        a = min(ns, k);
        __syncwarp();
    } else {
        // Survivors wait in a queue until there are 32: scored as they come, a float64 chain would run for the
        // few of a batch of candidates (1,000 queries x 2,000 x 64 floats, cosine, k = 400: 937 -> 647 us).
        int held = 0;
        for (int b0 = 0; b0 < m || held > 0; b0 += 32) {
            const bool in = b0 + lane < m;
            const float value = in ? cand_val[region + b0 + lane] : INFINITY;
            const uint32_t hm = __ballot_sync(0xffffffffu, in && value <= t);
            if ((hm >> lane) & 1u) {
                const int at = held + __popc(hm & ((1u << lane) - 1u));
                Wv[at] = value;
                Wi[at] = cand_id[region + b0 + lane];
            }
            held += __popc(hm);
            if (held < 32 && b0 + 32 < m) continue;  // uniform
            __syncwarp();
            const bool has = lane < held;
            const float approx = has ? Wv[lane] : INFINITY;
            const int32_t id = has ? Wi[lane] : -1;
            const bool more = 32 + lane < held;
            const float next_v = more ? Wv[32 + lane] : 0.f;
            const int32_t next_i = more ? Wi[32 + lane] : 0;
            __syncwarp();
            if (more) {
                Wv[lane] = next_v;
                Wi[lane] = next_i;
            }
            held = max(held - 32, 0);
            const bool known = has && fabsf(approx) < exact_lim;  // exact already (byte rows)
            const bool need = has && !known;
            double d = known ? double(approx) : INFINITY;
            if (dim >= COOP_DIM) {
                for (uint32_t hm = __ballot_sync(0xffffffffu, need); hm; hm &= hm - 1) {
                    const int j = __ffs(hm) - 1;
                    const int32_t idj = __shfl_sync(0xffffffffu, id, j);
                    const double dd = dist_f64_warp(data + int64_t(idj) * dim, qv, dim, metric,
                                                    cos ? xnorm[idj] : 1.0, qn, lane);
                    if (lane == j) d = dd;
                }
            } else if (need) {
                d = dist_f64_lane(data + int64_t(id) * dim, qv, dim, metric, cos ? xnorm[id] : 1.0, qn);
            }
            if (need) err = fmax(err, fabs(double(approx) - d));
            // Once there are k results, only candidates below the last go on, told by their lanes together; the
            // last only comes nearer, so each is tested again at its turn.
            uint32_t am = __ballot_sync(0xffffffffu, has && (a < k || pair_lt(d, id, Ad[k - 1], Ai[k - 1])));
            while (am) {
                const int j = __ffs(am) - 1;
                am &= am - 1;
                const double xd = __shfl_sync(0xffffffffu, d, j);
                const int32_t xi = __shfl_sync(0xffffffffu, id, j);
                if (a == k && !pair_lt(xd, xi, Ad[k - 1], Ai[k - 1])) continue;
                int c = 0;
                if (!isnan(xd)) {
                    for (int r = lane; r < a; r += 32) c += below(Ad[r], Ai[r], xd, xi);
                } else {
                    for (int r = lane; r < a; r += 32) c += pair_lt(Ad[r], Ai[r], xd, xi);
                }
                const int pos = __reduce_add_sync(0xffffffffu, c);
                for (int top = a - 1; top >= pos; top -= 32) {
                    const int r = top - lane;
                    double dv = 0;
                    int32_t iv = 0;
                    if (r >= pos) {
                        dv = Ad[r];
                        iv = Ai[r];
                    }
                    __syncwarp();
                    if (r >= pos) {
                        Ad[r + 1] = dv;
                        Ai[r + 1] = iv;
                    }
                    __syncwarp();
                }
                if (lane == 0) {
                    Ad[pos] = xd;
                    Ai[pos] = xi;
                }
                __syncwarp();
                a = min(a + 1, k);
            }
        }
    }
    if (exact_lim > 0.f) {  // results r = q, q + VERIFY_EVERY, ... (mod VERIFY_EVERY) in float64
        bool bad = false;
        const int r0 = q % VERIFY_EVERY;
        if (dim >= COOP_DIM) {
            for (int r = r0; r < a; r += VERIFY_EVERY) {
                const double dd = dist_f64_warp(data + int64_t(Ai[r]) * dim, qv, dim, metric, 1.0, qn, lane);
                bad |= dd != Ad[r];
            }
        } else {
            for (int r = r0 + lane * VERIFY_EVERY; r < a; r += 32 * VERIFY_EVERY)
                bad |= dist_f64_lane(data + int64_t(Ai[r]) * dim, qv, dim, metric, 1.0, qn) != Ad[r];
        }
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(mismatch, 1);
    }
    for (int r = lane; r < k; r += 32) {
        out_ids[int64_t(q) * k + r] = r < a ? int64_t(Ai[r]) : -1;
        out_d[int64_t(q) * k + r] = r < a ? Ad[r] : INFINITY;
    }
    // Non-negative doubles order as their bit patterns: an integer maximum over the warp, then
    // one atomic per query.
    unsigned long long eb = static_cast<unsigned long long>(__double_as_longlong(err));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) eb = max(eb, __shfl_xor_sync(0xffffffffu, eb, o));
    if (lane == 0 && eb) atomicMax(err_max, eb);
}

// Value classes of a float array: *flag gets bit 1 when a value is not an integer with |v| <= 256
// (exact in BF16), bit 2 when one is not an integer in [0, 255] (a byte). Written with explicit
// branches and an integer OR across the warp: a form that combined two boolean warp votes set the
// wrong bits on the GPU (every non-integer and 300 read as bytes), this one was checked against
// those values there.
__device__ __forceinline__ int value_class(float v) {
    int f = 0;
    const float r = rintf(v);
    if (r != v || !(fabsf(v) <= 256.f)) f |= 1;
    if (r != v || !(v >= 0.f) || !(v <= 255.f)) f |= 2;
    return f;
}

__global__ void check_small_int(const float *x, int64_t count, int32_t *flag) {
    int f = 0;
    const int64_t at = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, step = int64_t(gridDim.x) * blockDim.x;
    const int64_t n4 = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? count >> 2 : 0;  // 16-byte pieces
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
#pragma unroll 4
    for (int64_t i = at; i < n4; i += step) {
        const float4 v = __ldg(x4 + i);
        f |= value_class(v.x) | value_class(v.y) | value_class(v.z) | value_class(v.w);
    }
    for (int64_t i = 4 * n4 + at; i < count; i += step) f |= value_class(x[i]);
    f = int(__reduce_or_sync(0xffffffffu, uint32_t(f)));
    if (f && (threadIdx.x & 31) == 0) atomicOr(flag, f);
}

// Largest and total of the segment counts (overflow check and the candidate total).
__global__ void count_stats(const int32_t *cnt, int64_t len, unsigned long long *out) {
    unsigned long long mx = 0, sum = 0;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < len;
         i += int64_t(gridDim.x) * blockDim.x) {
        const unsigned long long c = static_cast<unsigned long long>(cnt[i]);
        mx = max(mx, c);
        sum += c;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out, mx);
        atomicAdd(out + 1, sum);
    }
}

// Error bound of the filter arithmetic and the per-query margins (2 e_q).
// Largest of n non-negative doubles: their bit patterns order as unsigned integers.
__global__ void max_norm_kernel(const double *xn, int64_t n, unsigned long long *out) {
    unsigned long long m = 0;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x)
        m = max(m, static_cast<unsigned long long>(__double_as_longlong(xn[i])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void margins_kernel(const double *qnorm, int32_t nq, double xmax, int kp, int terms,
                               int metric, float *margin) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nq) return;
    const double qn = metric == HNSW_B200_COSINE ? 1.0 : qnorm[q];
    const double xm = metric == HNSW_B200_COSINE ? 1.0 : xmax;
    const double rep = terms == 1 ? 0.0 : ldexp(1.0, -15);          // dropped lo.lo and rounding
    const double acc = double(kp + 8) * ldexp(1.0, -22);             // FP32 accumulation (2u per add)
    const double e_dot = (rep + acc) * 1.25 * qn * xm;
    double e = e_dot;
    if (metric == HNSW_B200_L2) e = 2.0 * e_dot + ldexp(1.0, -20) * (qn + xm) * (qn + xm);
    else e = e_dot + ldexp(1.0, -22);
    margin[q] = float(2.0 * e * 1.0001);
}

// ============================================================================== host
using hb::fail;

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        cudaDriverEntryPointQueryResult q;
        void *p = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// Tiled map of a row-major operand of kpad elements a row: boxes of one 128-byte swizzle row (BK
// BF16 or BK8 bytes) by box_rows rows.
int make_map(CUtensorMap *map, const void *base, int64_t rows, int kpad, int box_rows, bool u8 = false) {
    auto fn = encode_fn();
    if (!fn) return fail(HNSW_B200_ECUDA, "cuTensorMapEncodeTiled unavailable");
    cuuint64_t dims[2] = {cuuint64_t(kpad), cuuint64_t(rows)};
    cuuint64_t strides[1] = {cuuint64_t(kpad) * (u8 ? 1 : 2)};
    cuuint32_t box[2] = {cuuint32_t(u8 ? BK8 : BK), cuuint32_t(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, u8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                    const_cast<void *>(base), dims, strides,
                    box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(HNSW_B200_ECUDA, "cuTensorMapEncodeTiled failed: " + std::to_string(int(r)));
    return 0;
}

struct CudaMem {
    static bool device(int *d) { return cudaGetDevice(d) == cudaSuccess; }
    static bool alloc(void **p, size_t bytes) {
        if (cudaMalloc(p, bytes) == cudaSuccess) return true;
        cudaGetLastError();
        return false;
    }
    static void release(int d, void *p) {
        int now = d;
        cudaGetDevice(&now);
        if (now != d) cudaSetDevice(d);
        cudaFree(p);
        if (now != d) cudaSetDevice(now);
    }
};
using Scratch = DeviceScratch<CudaMem>;

#define XT(expr)                                                                               \
    do {                                                                                       \
        cudaError_t e_ = (expr);                                                               \
        if (e_ != cudaSuccess) return fail(HNSW_B200_ECUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
    } while (0)

size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Candidate lists take at most CAND_BYTES of scratch: (query, segment) pairs x cap x 8 bytes.
constexpr int64_t CAND_BYTES = int64_t(4) << 30;
// and this much, whatever candidates are expected, or twice as much where segments are then as long as the columns
// that they cover (a list just too short for its rows costs most): rows
// stored by cluster or by time fill few segments, and an overflow runs the call again. 1,000 queries x 1M x 128
// bytes in runs of 1,000 similar rows, k = 10, 2.26 -> 1.27 ms; 1,000 x 200K x 100 floats in runs of 2,000, cosine, k =
// 10, 1.28 -> 0.79 ms; rows in no order take the same time.
constexpr int64_t CAND_ROOM = int64_t(1) << 30;
constexpr int64_t MAX_CHUNK = 16384;  // queries of a batch filtered together
// A segment of pass two is sized for SEGMENT_FACTOR times its even share of the candidates expected, for
// thresholds looser than expected and uneven shares, and for SEGMENT_SLACK entries more: the columns it has
// in two tiles, for rows stored by cluster or by time, whose near rows lie in one or two tiles of one
// segment. With half a tile's columns of slack (32) such rows overflowed and the call ran twice: 10K
// queries x 1M x 128 bytes in 10,000 runs of similar rows, k = 100, 8.36 -> 4.20 ms; 2,000 x 200K x 64 floats
// in 10,000 runs, k = 10, 936 -> 480 us; rows in no order take the same time with either (3.21 ms,
// 430 us).
constexpr int64_t SEGMENT_FACTOR = 6;
constexpr int64_t SEGMENT_SLACK = 4 * CW;
// Byte rows use the integer filter (1) or the BF16 one (0).
#ifndef HB_EXACT_I8
#define HB_EXACT_I8 1
#endif
// Longest byte row of the integer filter: 2 dim 255^2 stays below 2^31.
constexpr int MAX_DIM_I8 = 8192;
// Pass one filters a sample: every tile_stride-th tile of the data, about sqrt(SAMPLE_BALANCE k n)
// rows (a longer sample costs filter time, a shorter one gives a looser threshold and pass two more
// candidates to append, select from and re-rank). Both passes with their selects and the re-rank, 10K
// queries x 1M x 128 bytes, k = 100: 2.91 ms at 25, 2.81 at 60, 2.82 at 150, 2.91 at 300.
constexpr double SAMPLE_BALANCE = 75.0;

// Which of a sample's smallest values is the threshold. A sample of a share f of the rows holds about
// k f of the k nearest, with a deviation of at most sqrt(k f), so its (k f + 6 sqrt(k f) + 8)-th
// smallest lies beyond the k-th nearest of all rows but for about one query in 10^9, while only about
// (k f + 6 sqrt(k f) + 8) / f rows pass it (at k = 100, f = 1/8: 330; the sample's k-th
// smallest, which is never too low, let 830 pass). Pass two counts: where a threshold was too low after
// all (rows stored by cluster or by time, a query's near ones in a sampled tile) the chunk runs again with
// the k-th smallest.
int sample_rank(int64_t k, int64_t sample_tiles, int64_t tiles) {
    if (sample_tiles >= tiles) return int(k);
    const double mean = double(k) * double(sample_tiles) / double(tiles);
    return int(std::min<double>(double(k), std::ceil(mean + 6.0 * std::sqrt(mean) + 8.0)));
}

// What the kernels report to the host, read once per chunk.
struct Stats {
    // of the current chunk
    int32_t err;         // a bounded wait expired
    int32_t mismatch;    // an integer filter distance differs from its float64 re-score
    int32_t short_lists; // a sampled threshold was too low
    int32_t pad;
    unsigned long long longest, total;  // candidate segments
    // of the call
    unsigned long long filter_err;  // largest |filter value - distance|, as bits of the double
    unsigned int bound;             // largest value the error bound is stated for, as bits of the float
    unsigned int pad2;
};

// One attempt at the whole batch with candidate lists of at least cap_min entries. Returns
// HNSW_B200_ERETRY with *cap_needed set when a query's candidates outgrew its list (many rows
// within the margin of the k-th distance, e.g. exact ties); the caller retries with that size.
template <typename T>
int exact_knn_typed(const hnsw_b200_exact_args_t *a, cudaStream_t s, int64_t cap_min,
                    int64_t *cap_needed) {
    const int64_t n = a->n, nq_all = a->nq;
    const int dim = a->dim, k = a->k, metric = a->metric;
    int integer = a->integer_valued;
    // Byte rows (every value an integer in [0, 255], L2 or inner product, int32-safe sums) take the
    // integer tensor-core filter, whose values are the exact distances.
    const bool bytes_ok = HB_EXACT_I8 && metric != HNSW_B200_COSINE && dim <= MAX_DIM_I8;
    bool bytes = false;
    if constexpr (std::is_same_v<T, uint8_t>) {
        integer = 1;
        bytes = bytes_ok;
    } else if (integer != 0) {  // find out on the device, one pass over each array
        static thread_local Scratch flag_buf;
        int32_t *flag = static_cast<int32_t *>(flag_buf.get(16));
        if (!flag) return fail(HNSW_B200_ENOMEM, "exact knn scratch allocation failed");
        XT(cudaMemsetAsync(flag, 0, 4, s));
        check_small_int<<<1024, 256, 0, s>>>(static_cast<const float *>(a->data), n * dim, flag);
        check_small_int<<<256, 256, 0, s>>>(static_cast<const float *>(a->queries), nq_all * dim, flag);
        XT(cudaGetLastError());
        int32_t hflag = 0;
        XT(cudaMemcpyAsync(&hflag, flag, 4, cudaMemcpyDeviceToHost, s));
        XT(cudaStreamSynchronize(s));
        if (integer < 0) integer = (hflag & 1) ? 0 : 1;
        bytes = bytes_ok && (hflag & 3) == 0;
    }
    const int terms = integer && metric != HNSW_B200_COSINE ? 1 : 3;
    const int seg = (dim + BK - 1) / BK * BK;
    // K of a row: BF16 elements (terms segments), or bytes in 128-byte chunks
    const int kp = bytes ? (dim + BK8 - 1) / BK8 * BK8 : seg * terms;
    const int64_t n_pad = (n + BN - 1) / BN * BN;
    int sms = 148;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);

    // Split of a pass over `tiles` tiles for a chunk of nqc queries.
    auto geo = [&](int64_t nqc, int tiles) { return split_tiles(int((nqc + BM - 1) / BM), tiles, sms); };
    // Pass one keeps the minimum of every block of rows (block_tiles), or every row where the sample has fewer than
    // 4 k; pass two keeps the rows within tau + margin. Each epilogue thread appends to its own segment of the query's list: in pass one at most one entry per block
    // or its 2 CW columns of a tile; pass two's segments get SEGMENT_FACTOR times their even share of the
    // expected candidates and SEGMENT_SLACK more, and never more than the columns that they cover (an
    // overflow re-runs the call with longer segments).
    const int tiles = int((n + BN - 1) / BN);
    const int64_t sample_rows = std::min<int64_t>(
        n, std::max<int64_t>(int64_t(64) * k, int64_t(std::sqrt(SAMPLE_BALANCE * double(k) * double(n)))));
    const int stride = std::max<int>(1, int(tiles / ((sample_rows + BN - 1) / BN)));
    const int sample = (tiles + stride - 1) / stride;  // tiles 0, stride, 2 stride, ... of pass one
    const int64_t pad = int64_t(sample - 1) * stride == tiles - 1 ? n_pad - n : 0;  // of the last sampled tile
    const int64_t whole = sample - (pad > 0), sampled = int64_t(sample) * BN - pad;
    // The largest blocks of which the sample surely has 2 k: k ln 4 rows of it lie below the k-th smallest of 2 k
    // minima, and fewer blocks make a looser threshold (1,000 rows' k-th of k minima is their largest) while every
    // row kept makes pass one append, which takes ten times as long (200 queries x 700 rows, k = 10: 68 us of a
    // call's 225).
    constexpr int GROUPS = CW / 4 * EPI_PER_QUARTER;  // blocks of a query in block_tiles tiles
    int block_tiles = 16;
    while (block_tiles > 0 && whole / block_tiles * GROUPS < 2 * int64_t(k)) block_tiles /= 2;
    const bool block_min = block_tiles > 0 || sampled / 4 >= k;
    const int rank = sample_rank(k, sample, tiles);
    const int64_t expect2 = int64_t(rank) * tiles / sample + int64_t(k) / 2;  // candidates of a query
    int64_t QB = std::min<int64_t>(nq_all, MAX_CHUNK);  // queries per chunk
    int64_t cap = 0, slots = 0;                           // entries per segment; (query, segment) pairs
    int64_t most = 0;  // columns of a segment of pass two
    for (;;) {
        cap = slots = most = 0;
        const int64_t last = nq_all % QB ? nq_all % QB : QB;
        for (int64_t nqc : {QB, last}) {
            const Split g1 = geo(nqc, sample), g2 = geo(nqc, tiles);
            const int64_t nseg2 = int64_t(g2.splits) * EPI_PER_QUARTER, columns = int64_t(2 * CW) * g2.tps;
            const int64_t share = (SEGMENT_FACTOR * expect2 + nseg2 - 1) / nseg2 + SEGMENT_SLACK;
            cap = std::max<int64_t>(cap, !block_min ? int64_t(2 * CW) * g1.tps
                                         : block_tiles ? CW / 4 * int64_t((g1.tps + block_tiles - 1) / block_tiles) : int64_t(2 * CW / 4) * g1.tps);
            cap = std::max<int64_t>(cap, std::min(std::max(cap_min, share), columns));
            most = std::max(most, columns);
            slots = std::max<int64_t>(slots, nqc * std::max(g1.splits, g2.splits) * EPI_PER_QUARTER);
        }
        if (slots * cap * 8 <= CAND_BYTES || QB <= BM) break;
        QB = std::max<int64_t>(BM, QB / 2 / BM * BM);  // longer lists: fewer queries per chunk
    }
    const int64_t q_pad = (QB + BM - 1) / BM * BM;
    static thread_local Scratch buf;
    size_t off = 0;
    auto carve = [&](size_t bytes) {
        size_t o = off;
        off += al256(bytes);
        return o;
    };
    const size_t esz = bytes ? 1 : 2;  // operand element bytes
    const size_t o_xb = carve(size_t(n_pad) * kp * esz);
    const size_t o_qb = carve(size_t(q_pad) * kp * esz);
    const size_t o_xn = carve(size_t(n_pad) * 8);
    const size_t o_qn = carve(size_t(q_pad) * 8);
    const size_t o_xx = carve(size_t(n_pad) * 4);
    const size_t o_qq = carve(size_t(q_pad) * 4);
    const size_t o_mg = carve(size_t(QB) * 4);
    const size_t o_th = carve(size_t(QB) * 4);
    const size_t o_tau = carve(size_t(QB) * 4);
    const size_t o_cnt = carve(size_t(slots) * 4);
    const size_t o_cm = carve(size_t(QB) * 4);
    const size_t o_st = carve(sizeof(Stats));
    const size_t o_mx = carve(16);
    // The lists last: longer where memory allows (CAND_ROOM), else as long as they have to be.
    const int64_t roomy = std::max(cap, most <= CAND_ROOM / (4 * slots) ? most : CAND_ROOM / (8 * slots));
    const size_t o_cv = off;
    auto list_bytes = [&](int64_t entries) { return al256(size_t(slots) * entries * 4); };
    char *B = static_cast<char *>(buf.get(off + 2 * list_bytes(roomy)));
    if (B) cap = roomy;
    else B = static_cast<char *>(buf.get(off + 2 * list_bytes(cap)));
    const size_t o_ci = o_cv + list_bytes(cap);
    if (!B) return fail(HNSW_B200_ENOMEM, "exact knn scratch allocation failed");
    auto *xb = reinterpret_cast<__nv_bfloat16 *>(B + o_xb);
    auto *qb = reinterpret_cast<__nv_bfloat16 *>(B + o_qb);
    auto *xn = reinterpret_cast<double *>(B + o_xn);
    auto *qn = reinterpret_cast<double *>(B + o_qn);
    auto *xx = reinterpret_cast<float *>(B + o_xx);
    auto *qq = reinterpret_cast<float *>(B + o_qq);
    auto *xb8 = reinterpret_cast<uint8_t *>(B + o_xb);  // byte path: the same buffers as u8 / int32
    auto *qb8 = reinterpret_cast<uint8_t *>(B + o_qb);
    auto *xxi = reinterpret_cast<int32_t *>(B + o_xx);
    auto *qqi = reinterpret_cast<int32_t *>(B + o_qq);
    auto *mg = reinterpret_cast<float *>(B + o_mg);
    auto *th = reinterpret_cast<float *>(B + o_th);
    auto *tau = reinterpret_cast<float *>(B + o_tau);
    auto *cnt = reinterpret_cast<int32_t *>(B + o_cnt);
    auto *cm = reinterpret_cast<int32_t *>(B + o_cm);  // per query: candidates after compaction
    auto *cv = reinterpret_cast<float *>(B + o_cv);
    auto *ci = reinterpret_cast<int32_t *>(B + o_ci);
    auto *st = reinterpret_cast<Stats *>(B + o_st);
    const T *X = static_cast<const T *>(a->data);
    const int cos = metric == HNSW_B200_COSINE;
    const bool l2 = metric == HNSW_B200_L2;
    int64_t launches = 0;

    // rows that can be read four elements a load
    auto vec = [&](const T *p) { return (dim & 3) == 0 && reinterpret_cast<uintptr_t>(p) % (4 * sizeof(T)) == 0; };
    if (bytes)
        prep_rows_u8<T><<<int(std::min<int64_t>(4096, (n_pad + 31) / 32)), 256, 0, s>>>(
            X, n, dim, n_pad, kp, xb8, xxi, vec(X), l2, I8_PAD);
    else
        prep_rows<T><<<int(std::min<int64_t>(8192, (n_pad + 7) / 8)), 256, 0, s>>>(
            X, n, dim, n_pad, kp, terms, 0, cos, xb, xn, xx, l2, INFINITY);
    XT(cudaGetLastError());
    launches++;
    double xmax = 1.0;  // largest data norm (margins): a device reduction, one 8-byte copy
    if (!cos && !bytes) {
        auto *mx = reinterpret_cast<unsigned long long *>(B + o_mx);
        XT(cudaMemsetAsync(mx, 0, 8, s));
        max_norm_kernel<<<int(std::min<int64_t>(1024, (n + 255) / 256)), 256, 0, s>>>(xn, n, mx);
        XT(cudaGetLastError());
        unsigned long long bits = 0;
        XT(cudaMemcpyAsync(&bits, mx, 8, cudaMemcpyDeviceToHost, s));
        XT(cudaStreamSynchronize(s));
        std::memcpy(&xmax, &bits, 8);
        launches++;
    }
    CUtensorMap tmA, tmB;
    if (int rc = make_map(&tmA, B + o_qb, q_pad, kp, BM, bytes)) return rc;
    if (int rc = make_map(&tmB, B + o_xb, n_pad, kp, BN, bytes)) return rc;
    // Operand buffers: the query tile's operand resident beside at least three stages of rows where
    // that fits, else loaded with every stage.
    const int kchunks = kp / (bytes ? BK8 : BK);
    const size_t room = SMEM_MAX - 1024 - XSLOTS * BN * 4 - BAR_BYTES;
    const bool resident = size_t(kchunks) * A_BYTES + 3 * size_t(B_BYTES) <= room;
    const size_t a_bytes = resident ? size_t(kchunks) * A_BYTES : 0;
    const size_t stage_bytes = resident ? B_BYTES : A_BYTES + B_BYTES;
    const int nstages = int(std::min<size_t>(MAX_STAGES, (room - a_bytes) / stage_bytes));
    const size_t smem = a_bytes + nstages * stage_bytes + XSLOTS * BN * 4 + 1024 + BAR_BYTES;
    const int wpb = 4;
    if (size_t(wpb) * (k + 1) * 12 > 200 * 1024) return fail(HNSW_B200_EINVAL, "k too large for the rerank kernel");
    // Survivors are gathered where that leaves an SM two blocks of four queries (k up to about 1,000), under cosine
    // eight (k up to about 220): a lane's divisions want many warps, which the insertion's smaller memory lets
    // in. Time of a search with them gathered over inserted (before the insertion's queue), 20K to 100K rows of 32 to 400 values, 100 to 10K
    // queries: l2 and ip 0.67 to 1.14 up to k = 1,000 and 0.74 to 1.53 above, bytes 0.63 to 1.05 and 0.71 to
    // 1.31, cosine 0.58 to 0.99 up to k = 200 and 0.69 to 1.77 above. (With the products of a batch's rows laid out in
    // shared memory as well, cosine at k = 10 took the same time, and from k = 1,000 on up to 1.5 times the time
    // without.)
    const bool gather = wpb * rerank_smem(k, true) * (cos ? 8 : 2) <= size_t(SMEM_MAX);
    const size_t rsm = wpb * rerank_smem(k, gather);
    XT(cudaFuncSetAttribute(rerank_topk<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(rsm)));
    XT(cudaMemsetAsync(st, 0, sizeof(Stats), s));
    Stats hst;
    int64_t total_cand = 0;

    for (int64_t q0 = 0; q0 < nq_all; q0 += QB) {
        const int64_t nq = std::min<int64_t>(QB, nq_all - q0);
        const T *Q = static_cast<const T *>(a->queries) + q0 * dim;
        if (bytes) {  // exact filter values: no margin
            prep_rows_u8<T><<<int(std::min<int64_t>(4096, (q_pad + 31) / 32)), 256, 0, s>>>(
                Q, nq, dim, q_pad, kp, qb8, qqi, vec(Q), l2, 0);
            XT(cudaMemsetAsync(mg, 0, size_t(nq) * 4, s));
        } else {
            prep_rows<T><<<int(std::min<int64_t>(4096, (q_pad + 7) / 8)), 256, 0, s>>>(
                Q, nq, dim, q_pad, kp, terms, 1, cos, qb, qn, qq, l2, 0.f);
            margins_kernel<<<int((nq + 255) / 256), 256, 0, s>>>(qn, int32_t(nq), xmax, kp, terms, metric, mg);
        }
        XT(cudaGetLastError());
        launches += 2;
        // Query tiles of this chunk only (the last chunk may be short), rows split to fill the GPU.
        const int qt_chunk = int((nq + BM - 1) / BM);
        int nseg = 0;  // segments per query of the last pass run
        auto run_filter = [&](int pass_tiles, int pass_stride, const float *pass_thr, bool bmin) -> int {
            const Split gg = geo(nq, pass_tiles);
            nseg = gg.splits * EPI_PER_QUARTER;
            FilterParams fp;
            fp.nq = int32_t(nq);
            fp.row_end = int32_t(n);
            fp.tiles = pass_tiles;
            fp.tile_stride = pass_stride;
            fp.kchunks = kchunks;
            fp.stages = nstages;
            fp.a_resident = resident ? 1 : 0;
            fp.tiles_per_split = gg.tps;
            fp.block_tiles = block_tiles;
            fp.metric = metric;
            fp.qq = qq;
            fp.xx = xx;
            fp.qqi = qqi;
            fp.xxi = xxi;
            fp.thr = pass_thr;
            fp.cand_val = cv;
            fp.cand_id = ci;
            fp.cand_cnt = cnt;
            fp.cap = int32_t(cap);
            fp.mul = metric == HNSW_B200_L2 ? -2 : -1;
            fp.err = &st->err;
            auto launch = [&](auto kern) -> int {
                XT(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
                kern<<<dim3(qt_chunk, gg.splits), FILTER_THREADS, smem, s>>>(tmA, tmB, fp);
                XT(cudaGetLastError());
                return 0;
            };
            const int rc = bytes ? (bmin ? launch(knn_filter_kernel<true, true>) : launch(knn_filter_kernel<true, false>))
                                 : (bmin ? launch(knn_filter_kernel<false, true>) : launch(knn_filter_kernel<false, false>));
            if (rc) return rc;
            launches++;
            return 0;
        };
        const int sel_blocks = int((nq + SELECT_WARPS - 1) / SELECT_WARPS);
        auto select = [&](SelectStep step, int32_t *ids, int sel_rank) {
            const bool last = step == SELECT_FINAL;
            select_kth<<<sel_blocks, 32 * SELECT_WARPS, 0, s>>>(
                cv, ids, cnt, int32_t(cap), int32_t(nseg), int32_t(nq), sel_rank, mg, th, tau, cm, step, bytes,
                last ? &st->short_lists : nullptr, last ? &st->bound : nullptr, last ? &st->longest : nullptr);
            launches++;
        };
        for (int pass_rank = rank;; pass_rank = k) {
            // Pass one: the sampled tiles give tau, the threshold of pass two.
            if (int rc = run_filter(sample, stride, nullptr, block_min)) return rc;
            select(SELECT_FIRST, nullptr, pass_rank);
            // Pass two: every row against tau + margin; the k-th smallest candidate is the global
            // k-th approximate distance, the final threshold. Where segments overflow, what they kept gives a
            // lower tau, and the pass runs again, twice at most: a loose threshold (rows stored by cluster or by time)
            // costs a pass and not a call with longer lists, which is left for exact ties and the like. 10K queries x
            // 1M x 128 bytes in runs of similar rows (with blocks of neighbouring rows): 10,000 rows each, k = 10, 32.4 ->
            // 15.2 ms; 1,000, k = 100, 12.5 -> 10.8 ms; but 1,000, k = 1,000, 28.8 -> 37.7 ms, where the passes do not
            // suffice. (A second one only where the first halved the longest segment: 35, 17.0, 37.6 ms.)
            for (int again = 0;; again++) {
                if (int rc = run_filter(tiles, 1, th, false)) return rc;
                count_stats<<<int(std::min<int64_t>(1024, (nq * nseg + 255) / 256)), 256, 0, s>>>(
                    cnt, nq * nseg, &st->longest);
                select(SELECT_FINAL, ci, k);
                rerank_topk<T><<<int((nq + wpb - 1) / wpb), wpb * 32, rsm, s>>>(
                    X, Q, dim, int32_t(nq), k, metric, xn, qn, cv, ci, cm, int32_t(cap), int32_t(nseg), th,
                    a->out_ids + q0 * k, a->out_dists + q0 * k, &st->filter_err, bytes ? EXACT_LIM : 0.f,
                    &st->mismatch, gather, &st->longest, pass_rank == k ? nullptr : &st->short_lists);
                XT(cudaGetLastError());
                launches += 2;
                XT(cudaMemcpyAsync(&hst, st, sizeof(Stats), cudaMemcpyDeviceToHost, s));
                XT(cudaMemsetAsync(st, 0, offsetof(Stats, filter_err), s));
                XT(cudaStreamSynchronize(s));
                if (hst.err) return fail(HNSW_B200_ECUDA, "exact knn: a bounded wait expired in the filter kernel");
                if (int64_t(hst.longest) <= cap || again == 2) break;
                select(SELECT_TIGHTEN, nullptr, k);
            }
            if (int64_t(hst.longest) > cap) {
                *cap_needed = int64_t(hst.longest);
                return fail(HNSW_B200_ERETRY, "exact knn: candidate buffer overflow (" +
                                                  std::to_string(hst.longest) + " > " + std::to_string(cap) + ")");
            }
            if (!hst.short_lists || pass_rank == k) break;
        }
        if (bytes && hst.mismatch)  // the integer results against their float64 re-scores
            return fail(HNSW_B200_ECUDA, "exact knn: an integer filter distance differs from its float64 re-score");
        total_cand += int64_t(hst.total);
    }
    if (a->out_filter_error_bound) {
        // BF16 filter: half the largest margin. Byte rows: the integer distances are exact and
        // only their float copies of 2^24 or more round, by at most half a float ulp of the
        // final threshold (counted here as a margin of a whole ulp).
        float v;
        std::memcpy(&v, &hst.bound, 4);
        // inner product: candidates reach below the threshold, down to -dim 255^2
        if (bytes && metric == HNSW_B200_IP) v = float(dim) * 65025.f;
        double max_margin = 0.0;
        if (!bytes) {
            max_margin = double(v);
        } else if (v >= EXACT_LIM) {
            int e = 0;
            std::frexp(double(v), &e);  // v in [2^(e-1), 2^e)
            max_margin = std::ldexp(1.0, e - 24);
        }
        *a->out_filter_error_bound = max_margin / 2.0;
    }
    if (a->out_filter_max_error) std::memcpy(a->out_filter_max_error, &hst.filter_err, 8);
    if (a->out_candidates) *a->out_candidates = total_cand;
    if (a->out_launches) *a->out_launches = launches;
    return 0;
}

}  // namespace hbx

extern "C" int hnsw_b200_exact_knn(const hnsw_b200_exact_args_t *a, void *stream) {
    using namespace hbx;
    if (!a || !a->data || !a->queries || !a->out_ids || !a->out_dists)
        return fail(HNSW_B200_EINVAL, "null argument");
    if (a->n < 1 || a->n > 0x7ffffff0 || a->dim < 1 || a->k < 1 || a->k > a->n || a->nq < 0)
        return fail(HNSW_B200_EINVAL, "need n >= 1, dim >= 1, 1 <= k <= n");
    if (a->metric < 0 || a->metric > 2) return fail(HNSW_B200_EINVAL, "unknown metric");
    if (a->nq == 0) return 0;
    if (a->dtype != HNSW_B200_F32 && a->dtype != HNSW_B200_U8)
        return fail(HNSW_B200_EINVAL, "unsupported dtype");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // A candidate overflow re-runs the batch with lists long enough for the largest count seen
    // (plus a quarter); a segment as long as the columns it covers cannot overflow, so this ends.
    int64_t cap_min = 0;
    for (int attempt = 0; attempt < 4; attempt++) {
        int64_t need = 0;
        const int rc = a->dtype == HNSW_B200_F32 ? exact_knn_typed<float>(a, s, cap_min, &need)
                                                 : exact_knn_typed<uint8_t>(a, s, cap_min, &need);
        if (rc != HNSW_B200_ERETRY || need <= 0) return rc;
        cap_min = std::max(cap_min, need + need / 4 + 64);
    }
    return fail(HNSW_B200_ERETRY, "exact knn: candidate lists still overflowed after retries");
}
