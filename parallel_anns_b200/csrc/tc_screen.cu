// Distance screens on the 5th-generation tensor cores.
//
// A screen computes s(x, y) = ||y||^2 - 2 x.y for blocks of 128 rows x against
// tiles of 128 columns y (the squared distance less ||x||^2) and hands on the
// few pairs that can matter; whoever called it ranks those exactly in float64.
// Two forms share the kernel:
//   k-NN    per row, every column that can be among its k nearest: a running
//           threshold t + 2 e, where t is the (k + 1)-th smallest s seen so far
//           (the row itself included) and e bounds the error of s. No true
//           neighbour is ever dropped; a row whose list overflows (many exact
//           ties) or holds non-finite values is reported instead.
//   range   per query, every column with s below a fixed threshold + e.
//
// Precision. The rows of both sides are shifted to the base's mean and multiplied
// by a power of two (exact) that brings the base's spread to about 1; s, the
// thresholds and the bounds below are all in these units. Each float32 operand is
// split in two BF16 parts, x = x1 + x2 + r with |r| <= 2^-18 |x|, and x.y is taken
// as x1.y1 + x1.y2 + x2.y1 in float32 accumulators, ||y||^2 riding in the
// contraction as three BF16 parts against ones. Left out of s: 2 * 3 * 2^-18
// |x||y|. The accumulation takes ceil((d + 3) / 16) + 2 ceil(d / 16) <= 49 steps,
// each within 2^-22 of the sum of the terms' sizes, 2 |x||y| + |y|^2. Together
// 2^-14.4 |x||y| + 2^-16.4 |y|^2. The float32 shift moves a squared distance by
// at most 2^-23 (|x| + |y|)^2, and a threshold's own roundings add 2^-23 (|x|^2 +
// |y|^2). Parts below BF16's or float32's normal range (2^-126) are off
// absolutely: by 2^-122 (|x| + |y|), which the terms above cover unless it is
// below 1e-60, and by 2^-117 in sums. e = 2^-14 |x| max|y| + 2^-16 max|y|^2 +
// 2^-21 |x|^2 + 1e-30 is larger than all of it for squared norms below 1e36
// (kTcLarge); a screen that meets a larger finite one says so (the spread is taken
// from a sample), a row with an infinity or a NaN is reported.
// Against a single TF32 product (the form before) the split costs 1.5 times the
// tensor time for 2^-16 instead of 2^-10, which makes the lists both short
// (about k + 3 entries instead of k + 32) and safe.
//
// Skipping. Rows and columns are processed in a locality order; every tile has
// a centre and a radius, and a tile whose ball is further from the row block's
// ball than any threshold of the block is not computed. On clustered bases
// that leaves a few percent of the tiles (250,000 x 96, 64 clusters: 2 %); on
// unclustered ones it costs a lookup per tile.
//
// One persistent CTA per SM takes (row block, split) items from a counter:
//   warp 4   producer: picks the tiles, tells the other warps through a ring of
//            entries, and loads the row block's operand (once per item) and
//            the column tiles' 64-wide slices (a ring of stages) by TMA;
//   warp 5   one thread issues the MMAs (M = 128, N = 128, K = 16) into one of
//            two TMEM accumulators of 128 columns;
//   warps 0-3 epilogue: thread t of warp w owns row 32 w + t (TMEM lane),
//            reads its accumulators 32 at a time and appends the columns under
//            its threshold to the row's list in global memory (L2). When a list
//            of the k-NN form runs full, the warp finds its (k + 1)-th smallest
//            by bisection, lowers the threshold and repacks it.
// Operands are K-major with the 128-byte swizzle: a slice is one TMA box of 128
// rows x 64 BF16, an MMA's K step advances the descriptor by 32 bytes.
// Every wait on an mbarrier is bounded: on expiry the kernel records an error,
// every role stops, the producer waits for its copies in flight, and the CTA
// still releases its tensor memory. No multicast anywhere.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/panns_b200.h"
#include "dev_scratch.h"
#include "learned.h"
#include "tc_screen.h"

namespace panns {

namespace cg = cooperative_groups;
namespace {

constexpr uint32_t kTcSliceW = 64;     // BF16 per TMA box row (128 bytes)
constexpr uint32_t kTcBox = kTcM * 128;  // bytes of one box
constexpr uint32_t kTcThreads = 192;   // 4 epilogue warps, producer, MMA issuer
constexpr uint32_t kTcTmemCols = 256;  // two accumulators of 128 columns
constexpr uint32_t kTcMaxWait = 1u << 24;
constexpr uint32_t kTcRing = 16;       // entries between the producer and the other roles
constexpr uint32_t kTcMaxStages = 8;
constexpr uint32_t kTcCap = 384;       // list entries per row of the k-NN form
constexpr uint32_t kTcEnd = 0xffffffffu, kTcExit = 0xfffffffeu, kTcTighten = 0xfffffffdu;
constexpr uint32_t kTcFirst = 0x80000000u;
constexpr float kTcBig = 1e38f;        // threshold of a list that is not full yet
constexpr float kTcLarge = 1e36f;      // squared norms the error bound holds up to
constexpr uint32_t kTcKnnBlocks = 32768;  // row blocks whose operand is held at a time (2 GB at d = 96)
constexpr uint32_t kNone = 0xffffffffu;

enum : uint32_t { TC_ERR_TIMEOUT = 1u };
enum : uint32_t { TC_NORM_BAD = 1u, TC_NORM_LARGE = 2u };  // a norm not below kTcLarge; one of finite values
enum { TC_KNN = 0, TC_RANGE = 1 };

struct TcArgs {
    uint32_t rows;        // rows of the row operand (positions < rows may hold a row)
    uint32_t rb0, items;  // first row block of this launch, (row block, split) items
    uint32_t splits;
    uint32_t tiles;       // column tiles
    uint32_t slices, stages;
    uint32_t k_hh, k_x;   // MMA K steps of the hi * hi product and of each cross product
    const float *lb2;     // squared lower bound of (row block - rb0, tile), or null
    const float *xn;      // ||x||^2 by row position
    const uint32_t *ymax; // float bits of the largest ||y||^2
    uint2 *lists;
    uint32_t cap;
    uint32_t *counter, *error;
    // k-NN form
    uint32_t k, C;
    const uint32_t *perm;  // position -> row (~0: none), null = identity
    uint32_t *cand, *fail_rows, *fail_count;
    const uint32_t *blk_cell, *cell_tile0, *near, *avail;  // cell-restricted screen, or null
    uint32_t P;
    // range form
    const float *tau;  // squared radius by query (rounded up)
    uint32_t *cnt;     // entries per (split, query)
    uint32_t id0;      // added to column positions (column chunks)
};

struct TcSmem {  // offsets into the dynamic shared memory (bytes)
    uint32_t a, b, bar, total;
};

__host__ __device__ inline TcSmem tc_layout(uint32_t slices, uint32_t stages) {
    TcSmem s;
    s.a = 0;                                   // slices x (hi, lo)
    s.b = s.a + slices * 2 * kTcBox;           // stages x (hi, lo)
    s.bar = s.b + stages * 2 * kTcBox;         // mbarriers, ring, thresholds, TMEM address
    s.total = s.bar + 8 * (2 + 2 * kTcMaxStages + 4 + 2 * kTcRing + 1) + kTcRing * 8 + 4 * 4 * 4 + 16;
    return s;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t) __cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Wait for the phase of parity `parity` to complete; false after kTcMaxWait
// tries, or when another role has given up (the caller stops).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t i = 0; i < kTcMaxWait; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
        if ((i & 255u) == 255u && *abort_flag) return false;
    }
    return false;
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int32_t x, int32_t y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"((uint64_t) map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart, Blackwell descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    uint64_t desc = 0;
    desc |= (uint64_t) ((saddr & 0x3FFFFu) >> 4);   // start address
    desc |= (uint64_t) 1 << 16;                     // leading byte offset (unused with this swizzle)
    desc |= (uint64_t) (1024 >> 4) << 32;           // stride byte offset
    desc |= (uint64_t) 1 << 46;                     // version
    desc |= (uint64_t) 2 << 61;                     // SWIZZLE_128B
    return desc;
}

// Instruction descriptor: D float32, A and B BF16, both K-major, N = M = 128.
constexpr uint32_t kTcIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kTcM >> 3) << 17) | ((kTcM >> 4) << 24);

__device__ __forceinline__ void umma_bf16(uint32_t tmem, uint64_t da, uint64_t db, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %3, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %4, p;\n\t}"
        ::"r"(tmem), "l"(da), "l"(db), "r"(accumulate), "r"(kTcIdesc)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 32 columns of this warp's 32 TMEM lanes; the values may be used after tmem_wait.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]),
                   "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]),
                   "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]),
                   "+r"(v[29]), "+r"(v[30]), "+r"(v[31])::"memory");
}

// The warp repacks up to four rows' lists at once (n[j] <= kTcCap entries each,
// 0 = none; four, because one row's loads and reductions are a chain of
// latencies that four rows share): per row, an upper bound t of its `want`-th
// smallest value with at most `slack` more entries at or below it (fewer only
// where equal values allow), by bisection between the smallest and the largest;
// then the entries <= t + margin are kept, in order. kept[j] = how many,
// bound[j] = t + margin, the same on every lane.
constexpr int kTcRows = 4;
__device__ __forceinline__ void tc_repack(uint2 *const (&list)[kTcRows], const uint32_t (&n)[kTcRows], uint32_t want,
                                          uint32_t slack, const float (&margin)[kTcRows], uint32_t (&kept)[kTcRows],
                                          float (&bound)[kTcRows], int lane) {
    constexpr int kPer = kTcCap / 32;
    const float kInf = __int_as_float(0x7f800000);
    float v[kTcRows][kPer];
    uint32_t id[kTcRows][kPer];
    float lo[kTcRows], hi[kTcRows];
#pragma unroll
    for (int j = 0; j < kTcRows; ++j) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const uint32_t p = i * 32 + lane;
            uint2 e = make_uint2(__float_as_uint(kInf), 0u);
            if (p < n[j]) e = __ldcg(list[j] + p);
            v[j][i] = __uint_as_float(e.x);
            id[j][i] = e.y;
        }
    }
#pragma unroll
    for (int j = 0; j < kTcRows; ++j) {
        lo[j] = kInf;
        hi[j] = -kInf;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            lo[j] = fminf(lo[j], v[j][i]);
            if (v[j][i] < kInf) hi[j] = fmaxf(hi[j], v[j][i]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < kTcRows; ++j) {
            lo[j] = fminf(lo[j], __shfl_xor_sync(0xffffffffu, lo[j], o));
            hi[j] = fmaxf(hi[j], __shfl_xor_sync(0xffffffffu, hi[j], o));
        }
    // count(<= hi) >= want throughout; count(<= lo) < want once lo has moved.
    bool done[kTcRows];
#pragma unroll
    for (int j = 0; j < kTcRows; ++j) {
        done[j] = n[j] <= want + slack;  // the largest will do
        lo[j] = lo[j] - (fabsf(lo[j]) * 1e-6f + 1e-30f);
    }
    for (int step = 0; step < 64; ++step) {
        float mid[kTcRows];
        uint32_t c[kTcRows];
        bool all = true;
#pragma unroll
        for (int j = 0; j < kTcRows; ++j) {
            mid[j] = 0.5f * lo[j] + 0.5f * hi[j];
            if (!(mid[j] > lo[j] && mid[j] < hi[j])) done[j] = true;
            all = all && done[j];
            c[j] = 0;
#pragma unroll
            for (int i = 0; i < kPer; ++i) c[j] += v[j][i] <= mid[j] ? 1u : 0u;
        }
        if (all) break;  // warp-uniform
#pragma unroll
        for (int j = 0; j < kTcRows; ++j) c[j] = __reduce_add_sync(0xffffffffu, c[j]);
#pragma unroll
        for (int j = 0; j < kTcRows; ++j) {
            if (done[j]) continue;
            if (c[j] >= want) {
                hi[j] = mid[j];
                done[j] = c[j] <= want + slack;
            } else {
                lo[j] = mid[j];
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kTcRows; ++j) {
        bound[j] = hi[j] + margin[j];
        kept[j] = 0;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const bool keep = i * 32 + (uint32_t) lane < n[j] && v[j][i] <= bound[j];
            const uint32_t bm = __ballot_sync(0xffffffffu, keep);
            if (keep)
                __stcg(list[j] + kept[j] + __popc(bm & ((1u << lane) - 1u)), make_uint2(__float_as_uint(v[j][i]), id[j][i]));
            kept[j] += __popc(bm);
        }
    }
    __syncwarp();
}

template <int FORM>
__global__ void __launch_bounds__(kTcThreads, 1)
    tc_screen_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     TcArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t) 1023);
    const TcSmem L = tc_layout(a.slices, a.stages);
    uint8_t *sa = smem + L.a;
    uint8_t *sb = smem + L.b;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bar);
    uint64_t *a_full = bars, *a_empty = bars + 1;
    uint64_t *b_full = bars + 2, *b_empty = b_full + kTcMaxStages;
    uint64_t *t_full = b_empty + kTcMaxStages, *t_empty = t_full + 2;
    uint64_t *r_full = t_empty + 2, *r_empty = r_full + kTcRing;
    uint64_t *tight = r_empty + kTcRing;
    volatile uint2 *ring = reinterpret_cast<volatile uint2 *>(tight + 1);
    // wmax[item & 3][w]: the largest squared distance a row of epilogue warp w can still use
    volatile float *wmax = reinterpret_cast<volatile float *>(const_cast<uint2 *>(ring) + kTcRing);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(const_cast<float *>(wmax) + 16);
    volatile uint32_t *abort_flag = tmem_slot + 1;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float kInf = __int_as_float(0x7f800000);

    if (threadIdx.x == 0) {
        mbar_init(a_full, 1);
        mbar_init(a_empty, 1);
        for (uint32_t s = 0; s < a.stages; ++s) {
            mbar_init(b_full + s, 1);
            mbar_init(b_empty + s, 1);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(t_full + t, 1);
            mbar_init(t_empty + t, 4);
        }
        for (uint32_t s = 0; s < kTcRing; ++s) {
            mbar_init(r_full + s, 1);
            mbar_init(r_empty + s, 5);
        }
        mbar_init(tight, 4);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTcTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    auto fail = [&]() {
        atomicOr(a.error, TC_ERR_TIMEOUT);
        *abort_flag = 1;
    };

    if (warp == 4) {
        // ---- producer ----
        uint32_t g = 0, bs = 0, na = 0, seq = 0, nt_ = 0;  // ring entries, stages filled, row operands loaded, items, tightenings
        bool ok = true;
        auto push = [&](uint32_t item, uint32_t what) {
            if (lane == 0) {
                const uint32_t s = g % kTcRing;
                ok = mbar_wait(r_empty + s, ((g / kTcRing) & 1) ^ 1, abort_flag);
                if (ok) {
                    ring[s].x = item;
                    ring[s].y = what;
                    mbar_arrive(r_full + s);
                }
            }
            ++g;
            ok = __shfl_sync(0xffffffffu, ok, 0);
        };
        while (ok) {
            uint32_t item = 0;
            if (lane == 0) item = atomicAdd(a.counter, 1u);
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= a.items) {
                push(0, kTcExit);
                break;
            }
            const uint32_t rbl = item / a.splits, sp = item % a.splits, rb = a.rb0 + rbl;
            // The item's bound slot starts open. KNN: four items later at the
            // earliest is it used again, and the ring and the row operand's
            // barrier keep the producer less than two items ahead.
            if (FORM == TC_KNN && lane < 4) wmax[(seq & 3) * 4 + lane] = kInf;
            __syncwarp();
            const float *lb = a.lb2 ? a.lb2 + (size_t) rbl * a.tiles : nullptr;
            bool first = true;
            auto issue = [&](uint32_t t) {  // tile t of this item, by lane 0 (warp-uniform call)
                push(item, t | (first ? kTcFirst : 0u));
                if (ok && lane == 0) {
                    if (first) {
                        ok = mbar_wait(a_empty, (na & 1) ^ 1, abort_flag);
                        if (ok) {
                            mbar_expect_tx(a_full, a.slices * 2 * kTcBox);
                            for (uint32_t sl = 0; sl < a.slices; ++sl)
                                for (uint32_t h = 0; h < 2; ++h)
                                    tma_load_2d(sa + (sl * 2 + h) * kTcBox, &map_a, a_full,
                                                (int32_t) ((h * a.slices + sl) * kTcSliceW), (int32_t) (rbl * kTcM));
                        }
                    }
                    for (uint32_t sl = 0; ok && sl < a.slices; ++sl, ++bs) {
                        const uint32_t s = bs % a.stages;
                        ok = mbar_wait(b_empty + s, ((bs / a.stages) & 1) ^ 1, abort_flag);
                        if (!ok) break;
                        mbar_expect_tx(b_full + s, 2 * kTcBox);
                        for (uint32_t h = 0; h < 2; ++h)
                            tma_load_2d(sb + (s * 2 + h) * kTcBox, &map_b, b_full + s,
                                        (int32_t) ((h * a.slices + sl) * kTcSliceW), (int32_t) (t * kTcM));
                    }
                }
                if (first) ++na;
                first = false;
                bs = __shfl_sync(0xffffffffu, bs, 0);
                ok = __shfl_sync(0xffffffffu, ok, 0);
            };
            if (FORM == TC_KNN && a.blk_cell) {
                // the tiles of the block's cell, then of its near cells
                const uint32_t cell = a.blk_cell[rb];
                for (uint32_t sgi = 0; ok && sgi <= a.P; ++sgi) {
                    const uint32_t c = sgi == 0 ? cell : a.near[(size_t) cell * a.P + sgi - 1];
                    if (c == kNone) continue;
                    for (uint32_t t = a.cell_tile0[c]; ok && t < a.cell_tile0[c + 1]; ++t) issue(t);
                }
            } else {
                // Every tile of the split, 32 bounds at a time. The k-NN form
                // takes the tiles whose balls meet the block's first, from
                // the block's own tile outwards, so that its thresholds are
                // low before the far tiles come up.
                const int rounds = FORM == TC_KNN && lb ? 2 : 1;
                const uint32_t t_lo = (uint32_t) ((uint64_t) a.tiles * sp / a.splits);
                const uint32_t t_hi = (uint32_t) ((uint64_t) a.tiles * (sp + 1) / a.splits);
                const uint32_t nt = t_hi - t_lo;
                for (int round = 0; ok && round < rounds; ++round) {
                    if (round == 1 && !first) {
                        // The far tiles are looked at once every row's threshold
                        // is as low as the near ones make it.
                        push(item, kTcTighten);
                        if (ok && lane == 0) ok = mbar_wait(tight, nt_ & 1, abort_flag);
                        ++nt_;
                        ok = __shfl_sync(0xffffffffu, ok, 0);
                    }
                    for (uint32_t i0 = 0; ok && i0 < nt; i0 += 32) {
                        const uint32_t i = i0 + lane;
                        uint32_t t = t_lo + i;
                        if (FORM == TC_KNN) {  // one split: rb, rb + 1, rb - 1, rb + 2, ... (mod tiles)
                            const uint32_t h = (i + 1) >> 1;
                            t = (i & 1) ? rb + h : rb + a.tiles - h;
                            t = t >= a.tiles ? t - a.tiles : t;
                        }
                        float v = kInf;
                        if (i < nt) v = lb ? __ldg(lb + t) : 0.f;
                        auto now = [&]() {
                            if (FORM == TC_RANGE) return 0.f;  // lb2 holds 0 (needed) or +inf
                            volatile float *w = wmax + (seq & 3) * 4;
                            return fmaxf(fmaxf(w[0], w[1]), fmaxf(w[2], w[3]));
                        };
                        // not above the bound (a NaN is not), and of this round
                        const bool mine = i < nt && (rounds == 1 || (v > 0.f) == (round == 1));
                        uint32_t want = __ballot_sync(0xffffffffu, mine && !(v > now()));
                        while (want && ok) {
                            const int src = __ffs(want) - 1;
                            want &= want - 1;
                            const uint32_t ts = __shfl_sync(0xffffffffu, t, src);
                            const float vs = __shfl_sync(0xffffffffu, v, src);
                            const bool still = FORM == TC_RANGE || !(vs > __shfl_sync(0xffffffffu, now(), 0));
                            if (still) issue(ts);
                        }
                    }
                }
            }
            if (ok) push(item, kTcEnd);
            ++seq;
        }
        if (!ok && lane == 0) {
            fail();
            // copies in flight land before the CTA's memory goes
            for (uint32_t s = 0; s < a.stages; ++s) {
                const uint32_t used = bs > s ? (bs - 1 - s) / a.stages + 1 : 0;  // times stage s was filled
                if (used)
                    for (uint32_t i = 0; i < kTcMaxWait; ++i) {
                        uint32_t done;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                            "selp.u32 %0, 1, 0, p;\n\t}"
                            : "=r"(done)
                            : "r"(smem_u32(b_full + s)), "r"((used - 1) & 1)
                            : "memory");
                        if (done) break;
                    }
            }
            if (na)
                for (uint32_t i = 0; i < kTcMaxWait; ++i) {
                    uint32_t done;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                        "selp.u32 %0, 1, 0, p;\n\t}"
                        : "=r"(done)
                        : "r"(smem_u32(a_full)), "r"((na - 1) & 1)
                        : "memory");
                    if (done) break;
                }
        }
    } else if (warp == 5) {
        // ---- MMA issuer ----
        if (lane == 0) {
            uint32_t g = 0, bs = 0, na = 0, tg = 0;
            bool ok = true, open = false;
            while (ok) {
                const uint32_t s = g % kTcRing;
                ok = mbar_wait(r_full + s, (g / kTcRing) & 1, abort_flag);
                if (!ok) break;
                const uint32_t what = ring[s].y;
                mbar_arrive(r_empty + s);
                ++g;
                if (what == kTcExit) break;
                if (what == kTcTighten) continue;
                if (what == kTcEnd) {
                    if (open) umma_commit(a_empty);
                    open = false;
                    continue;
                }
                if (what & kTcFirst) {
                    ok = mbar_wait(a_full, na & 1, abort_flag);
                    ++na;
                    open = true;
                }
                const uint32_t t = tg & 1, tph = (tg >> 1) & 1;
                ok = ok && mbar_wait(t_empty + t, tph ^ 1, abort_flag);
                ++tg;
                const uint32_t d = tmem + t * kTcM;
                uint32_t acc = 0;
                for (uint32_t sl = 0; ok && sl < a.slices; ++sl, ++bs) {
                    const uint32_t st = bs % a.stages;
                    ok = mbar_wait(b_full + st, (bs / a.stages) & 1, abort_flag);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t ah = smem_u32(sa + sl * 2 * kTcBox), al = ah + kTcBox;
                    const uint32_t bh = smem_u32(sb + st * 2 * kTcBox), bl = bh + kTcBox;
                    for (uint32_t ks = 0; ks < 4; ++ks) {
                        const uint32_t kk = sl * 4 + ks;
                        if (kk < a.k_hh) {
                            umma_bf16(d, umma_desc(ah + ks * 32), umma_desc(bh + ks * 32), acc);
                            acc = 1;
                        }
                        if (kk < a.k_x) {
                            umma_bf16(d, umma_desc(ah + ks * 32), umma_desc(bl + ks * 32), 1);
                            umma_bf16(d, umma_desc(al + ks * 32), umma_desc(bh + ks * 32), 1);
                        }
                    }
                    umma_commit(b_empty + st);
                }
                if (ok) umma_commit(t_full + t);
            }
            if (!ok) fail();
        }
    } else {
        // ---- epilogue: warps 0-3, thread r = 32 w + lane owns row r of the block ----
        const uint32_t r = warp * 32 + lane;
        uint32_t g = 0, tg = 0, seq = 0;
        uint32_t row = kNone, cnt = 0;       // this thread's row (position) and list length
        float thr = -kInf, eps = 0.f, xn = 0.f;
        uint2 *list = nullptr;
        bool live = false, open = false, ok = true;
        const float ymax2 = __uint_as_float(*a.ymax);
        uint2 *my_lists = a.lists + (size_t) blockIdx.x * kTcM * kTcCap;  // KNN: this CTA's lists
        // Repack the lists of the rows in `which`, lower their thresholds, and
        // publish the largest squared distance any row of the warp can still use.
        auto lower = [&](uint32_t which, uint32_t want, uint32_t slack) {
            while (which) {
                uint2 *ls[kTcRows];
                uint32_t n[kTcRows], kept[kTcRows];
                int src[kTcRows];
                float e2[kTcRows], bound[kTcRows];
#pragma unroll
                for (int j = 0; j < kTcRows; ++j) {
                    src[j] = which ? __ffs(which) - 1 : -1;
                    which &= which - 1;
                    const int sj = src[j] < 0 ? 0 : src[j];
                    n[j] = __shfl_sync(0xffffffffu, cnt, sj);
                    e2[j] = 2.f * __shfl_sync(0xffffffffu, eps, sj);
                    if (src[j] < 0) n[j] = 0;
                    ls[j] = my_lists + (size_t) (warp * 32 + sj) * kTcCap;
                }
                tc_repack(ls, n, want, slack, e2, kept, bound, lane);
#pragma unroll
                for (int j = 0; j < kTcRows; ++j) {
                    if ((int) lane == src[j]) {
                        cnt = kept[j];
                        thr = fminf(thr, bound[j]);
                        if (cnt > kTcCap - kTcM) {  // too many within the error bound: the row is reported
                            cnt = 0;
                            thr = -kInf;
                        }
                    }
                }
            }
            // A dead or reported row asks for nothing; an open one for every tile.
            float m = thr >= kTcBig ? kInf : thr > -kInf ? (thr + xn) + 1e-5f * (fabsf(thr) + xn) : -kInf;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane == 0) wmax[(seq & 3) * 4 + warp] = m;
        };
        while (true) {
            const uint32_t s = g % kTcRing;
            ok = mbar_wait(r_full + s, (g / kTcRing) & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint32_t item = ring[s].x, what = ring[s].y;
            __syncwarp();
            if (lane == 0) mbar_arrive(r_empty + s);
            ++g;
            if (what == kTcExit) break;
            if (FORM == TC_KNN && what == kTcTighten) {
                lower(__ballot_sync(0xffffffffu, cnt > a.k + 9 && thr > -kInf), a.k + 1, 4);
                __syncwarp();
                if (lane == 0) mbar_arrive(tight);
                continue;
            }
            if (what == kTcEnd) {
                if (FORM == TC_RANGE) {
                    if (open && live) a.cnt[(size_t) (item % a.splits) * a.rows + row] = cnt;
                } else {
                    // Every list down to what cand holds, then the candidates
                    // out (all there are, where the cells hold fewer rows).
                    uint32_t want = a.k + 1;
                    if (a.blk_cell) want = min(want, a.avail[a.blk_cell[a.rb0 + item]]);
                    lower(__ballot_sync(0xffffffffu, live && cnt >= want && cnt > a.C + 1 && thr > -kInf), want,
                          min(8u, (a.C - a.k) / 4));
                    const bool good = live && cnt >= want && cnt <= a.C + 1 && thr > -kInf;
                    const uint32_t self = live ? (a.perm ? a.perm[row] : row) : kNone;
                    if (live && !good) a.fail_rows[atomicAdd(a.fail_count, 1u)] = self;
                    for (uint32_t todo = __ballot_sync(0xffffffffu, good); todo;) {
                        uint32_t n[kTcRows], sf[kTcRows], out[kTcRows], most = 0;
                        const uint2 *ls[kTcRows];
#pragma unroll
                        for (int j = 0; j < kTcRows; ++j) {
                            const int src = todo ? __ffs(todo) - 1 : -1;
                            todo &= todo - 1;
                            const int sj = src < 0 ? 0 : src;
                            n[j] = __shfl_sync(0xffffffffu, cnt, sj);
                            sf[j] = __shfl_sync(0xffffffffu, self, sj);
                            if (src < 0) n[j] = 0;
                            ls[j] = my_lists + (size_t) (warp * 32 + sj) * kTcCap;
                            out[j] = 0;
                            most = max(most, n[j]);
                        }
                        for (uint32_t i0 = 0; i0 < most; i0 += 32) {
                            uint32_t id[kTcRows];
#pragma unroll
                            for (int j = 0; j < kTcRows; ++j)
                                id[j] = i0 + lane < n[j] ? __ldcg(&ls[j][i0 + lane].y) : kNone;
                            if (a.perm) {
#pragma unroll
                                for (int j = 0; j < kTcRows; ++j) id[j] = id[j] != kNone ? a.perm[id[j]] : kNone;
                            }
#pragma unroll
                            for (int j = 0; j < kTcRows; ++j) {
                                const bool keep = id[j] != kNone && id[j] != sf[j];
                                const uint32_t bm = __ballot_sync(0xffffffffu, keep);
                                const uint32_t at = out[j] + __popc(bm & ((1u << lane) - 1u));
                                if (keep && at < a.C) a.cand[(size_t) sf[j] * a.C + at] = id[j];
                                out[j] += __popc(bm);
                            }
                        }
#pragma unroll
                        for (int j = 0; j < kTcRows; ++j)
                            if (n[j])
                                for (uint32_t i = out[j] + lane; i < a.C; i += 32)
                                    a.cand[(size_t) sf[j] * a.C + i] = kNone;
                    }
                }
                open = false;
                ++seq;
                continue;
            }
            if (what & kTcFirst) {
                const uint32_t rb = a.rb0 + item / a.splits, sp = item % a.splits;
                row = rb * kTcM + r;
                live = row < a.rows && (FORM == TC_RANGE || !a.perm || a.perm[row] != kNone);
                open = true;
                cnt = 0;
                thr = -kInf;
                if (live) {
                    xn = a.xn[row];
                    eps = 0x1p-14f * sqrtf(xn) * sqrtf(ymax2) + 0x1p-16f * ymax2 + 0x1p-21f * xn + 1e-30f;
                    if (FORM == TC_RANGE) {
                        cnt = a.cnt[(size_t) sp * a.rows + row];
                        thr = a.tau[row] - xn + eps;
                        list = a.lists + ((size_t) sp * a.rows + row) * a.cap;
                    } else {
                        thr = xn < kTcLarge ? kTcBig : -kInf;  // (a NaN is not): reported
                        list = my_lists + (size_t) r * kTcCap;
                    }
                }
            }
            const uint32_t c0 = (what & ~kTcFirst) * kTcM + (FORM == TC_RANGE ? a.id0 : 0u);
            const uint32_t t = tg & 1, tph = (tg >> 1) & 1;
            ++tg;
            ok = mbar_wait(t_full + t, tph, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem + ((warp * 32) << 16) + t * kTcM;
            uint32_t v[2][32];
            tmem_ld32(taddr, v[0]);
            tmem_wait(v[0]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q < 3) tmem_ld32(taddr + 32 * (q + 1), v[(q + 1) & 1]);
#pragma unroll
                for (int o = 0; o < 32; o += 8) {
                    float m = __uint_as_float(v[q & 1][o]);
#pragma unroll
                    for (int j = 1; j < 8; ++j) m = fminf(m, __uint_as_float(v[q & 1][o + j]));
                    if (m <= thr) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const uint32_t b = v[q & 1][o + j];
                            if (__uint_as_float(b) <= thr) {
                                // KNN: cnt + 128 <= kTcCap at the start of a tile
                                if (FORM == TC_KNN || cnt < a.cap)
                                    __stcg(list + cnt, make_uint2(b, c0 + 32 * q + o + j));
                                ++cnt;
                            }
                        }
                    }
                }
                __syncwarp();
                if (q < 3) tmem_wait(v[(q + 1) & 1]);
                if (q == 2) {  // everything is in registers
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(t_empty + t);
                }
            }
            __syncwarp();
            if (FORM == TC_KNN) {
                const uint32_t full = __ballot_sync(0xffffffffu, cnt > kTcCap - kTcM);
                if (full) lower(full, a.k + 1, 8);
            }
        }
        if (!ok && lane == 0) fail();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcTmemCols));
    }
}

// ---- operands, balls, bounds -------------------------------------------------

// shift = the mean of up to 4,096 rows at a fixed stride (one block per
// dimension), spread = the largest finite distance of one of their values to it
// (float bits, zeroed beforehand). Distances do not change under a shift, and the
// error bound follows the norms, so data far from the origin loses nothing.
__global__ void __launch_bounds__(256) tc_shift_kernel(const float *__restrict__ x, uint32_t n, uint32_t d,
                                                       float *__restrict__ shift, uint32_t *__restrict__ spread) {
    constexpr uint32_t kRows = 4096, kPer = kRows / 256;
    __shared__ float red[8];
    __shared__ float mean;
    const uint32_t j = blockIdx.x, m = min(n, kRows);
    float v[kPer], s = 0.f;
#pragma unroll
    for (uint32_t t = 0; t < kPer; ++t) {
        const uint32_t i = threadIdx.x + 256 * t;
        v[t] = i < m ? x[((uint64_t) i * n / m) * d + j] : 0.f;
        s += v[t];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i) s += red[i];
        s /= (float) m;
        mean = shift[j] = fabsf(s) < 1e30f ? s : 0.f;
    }
    __syncthreads();
    float far = 0.f;
#pragma unroll
    for (uint32_t t = 0; t < kPer; ++t) {
        const float u = fabsf(v[t] - mean);
        if (threadIdx.x + 256 * t < m && u < 3e38f) far = fmaxf(far, u);
    }
    const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(far));
    if ((threadIdx.x & 31) == 0) atomicMax(spread, most);
}

// The d shifts in scaled units, in place, and the scale after them: element j of a
// row goes into the screen as x_j * frame[d] - frame[j]. The scale is the power of
// two (exact to multiply by) that brings the spread to [0.5, 1), or as near as
// float32's exponents allow; 1 for a spread of 0. One block.
__global__ void __launch_bounds__(256) tc_frame_kernel(float *__restrict__ frame, const uint32_t *__restrict__ spread,
                                                       uint32_t d) {
    const uint32_t bits = *spread, e = bits >> 23;  // biased exponent; 0 below the normal range
    const float scale = bits ? __uint_as_float(max(1, 253 - (int) e) << 23) : 1.f;
    for (uint32_t j = threadIdx.x; j < d; j += 256) frame[j] *= scale;
    if (threadIdx.x == 0) frame[d] = scale;
}

// One block per tile of kTcM positions from p0: its rows (row perm[p] of x, p
// itself without perm; no row from `valid` on or where perm says ~0) go through
// shared memory once and leave as
//   operand rows less the shift and scaled, [hi (W) | lo (W)] BF16: A (row side)
//   holds x's parts and three ones after the high one; B (column side) the parts
//   of -2 x and ||x||^2 (float64 sum) in three parts, a position without a row a
//   norm no threshold reaches;
//   xn = ||x||^2, the maximum of the norms (float bits), both of the scaled rows;
//   *large |= TC_NORM_BAD where one is not below kTcLarge, TC_NORM_LARGE too where
//   the row is finite;
//   the tile's centre (mean of its rows) and radius (rounded up; a tile without
//   rows gets one that puts it out of every reach), scaled, not shifted.
// Null outputs are skipped. Bound by issue: a lane keeps its column pairs in
// registers from the norm to the two operands. 1M x 96 as columns: 0.72 ms with
// 440 instructions a row, 0.50 ms so, 0.54 ms with the scale.
constexpr int kPrepSteps = 5;  // 64-wide steps of an operand row: W <= 320

__global__ void __launch_bounds__(256) tc_prepare_kernel(const float *__restrict__ x, uint32_t n, uint32_t d,
                                                         const uint32_t *__restrict__ perm, uint32_t p0,
                                                         uint32_t valid, uint32_t W, const float *__restrict__ frame,
                                                         __nv_bfloat16 *__restrict__ A, __nv_bfloat16 *__restrict__ B,
                                                         float *__restrict__ xn, uint32_t *__restrict__ ymax,
                                                         uint32_t *__restrict__ large, float *__restrict__ centre,
                                                         float *__restrict__ radius) {
    extern __shared__ __align__(16) float tile[];  // kTcM x d
    __shared__ uint32_t rows[kTcM];
    __shared__ float c[256], sh[256];
    __shared__ float rmax[8], nmax[8];
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, t0 = blockIdx.x * kTcM;
    bool filled = false;
    if (tid < kTcM) {
        const uint32_t p = p0 + t0 + tid;
        const uint32_t row = p < valid ? (perm ? perm[p] : p) : kNone;
        filled = row < n;
        rows[tid] = filled ? row : kNone;
    }
    const float scale = frame[d];
    if (tid < d) sh[tid] = frame[tid];
    const uint32_t count = (uint32_t) __syncthreads_count(filled);
    if (d % 4 == 0) {
        const uint32_t d4 = d / 4, di = 256 / d4, dq = 256 - di * d4;
        float4 *t4 = reinterpret_cast<float4 *>(tile);
        uint32_t i = tid / d4, q = tid - i * d4;
#pragma unroll 4
        for (uint32_t e = tid; e < kTcM * d4; e += 256) {
            t4[e] = rows[i] != kNone ? __ldg(reinterpret_cast<const float4 *>(x + (size_t) rows[i] * d) + q)
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
            i += di;
            q += dq;
            if (q >= d4) {
                q -= d4;
                ++i;
            }
        }
    } else {
        for (uint32_t e = tid; e < kTcM * d; e += 256) {
            const uint32_t i = e / d;
            tile[e] = rows[i] != kNone ? x[(size_t) rows[i] * d + (e - i * d)] : 0.f;
        }
    }
    __syncthreads();
    float nm = 0.f;
    uint32_t bad = 0;
    const bool even = d % 2 == 0;
    for (uint32_t i = w; i < kTcM; i += 8) {
        const bool have = rows[i] != kNone;
        const float *xr = tile + (size_t) i * d;
        // The lane's column pairs 2 lane + 64 t, shifted and scaled.
        float2 v[kPrepSteps];
        double s = 0.0;
#pragma unroll
        for (int t = 0; t < kPrepSteps; ++t) {
            const uint32_t e = 2 * lane + 64 * t;
            v[t] = make_float2(0.f, 0.f);
            if (64u * t >= d) continue;
            if (have && e + 1 < d) {
                float2 y = even ? *reinterpret_cast<const float2 *>(xr + e) : make_float2(xr[e], xr[e + 1]);
                v[t] = make_float2(fmaf(y.x, scale, -sh[e]), fmaf(y.y, scale, -sh[e + 1]));
            } else if (have && e < d) {
                v[t].x = fmaf(xr[e], scale, -sh[e]);
            }
            s = fma((double) v[t].x, (double) v[t].x, s);
            s = fma((double) v[t].y, (double) v[t].y, s);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float nf = (float) s;
        if (lane == 0 && xn) xn[t0 + i] = nf;
        if (have && nf < kTcLarge) {
            nm = fmaxf(nm, nf);
        } else if (have) {  // the warp agrees: the same sum on every lane
            bool finite = true;
            for (uint32_t e = lane; e < d; e += 32) finite = finite && fabsf(xr[e]) < __int_as_float(0x7f800000);
            bad |= __all_sync(0xffffffffu, finite) ? TC_NORM_BAD | TC_NORM_LARGE : TC_NORM_BAD;
        }
        const __nv_bfloat16 n1 = __float2bfloat16_rn(have ? nf : 3e38f);
        const float r1 = have ? nf - __bfloat162float(n1) : 0.f;
        const __nv_bfloat16 n2 = __float2bfloat16_rn(r1);
        const __nv_bfloat16 n3 = __float2bfloat16_rn(r1 - __bfloat162float(n2));
#pragma unroll
        for (int t = 0; t < kPrepSteps; ++t) {
            const uint32_t e = 2 * lane + 64 * t;
            if (64u * t >= W) break;
            __nv_bfloat162 hi = __floats2bfloat162_rn(v[t].x, v[t].y);
            const float2 hf = __bfloat1622float2(hi);
            const __nv_bfloat162 lo = __floats2bfloat162_rn(v[t].x - hf.x, v[t].y - hf.y);
            const size_t at = (size_t) (t0 + i) * 2 * W + e;
            const __nv_bfloat16 one = __float2bfloat16_rn(1.f);
            const uint32_t k0 = e - d, k1 = e + 1 - d;  // 0, 1, 2: the norm's parts
            if (A) {
                __nv_bfloat162 a = hi;
                if (e + 1 >= d) {
                    if (k0 < 3u) a.x = one;
                    if (k1 < 3u) a.y = one;
                }
                *reinterpret_cast<__nv_bfloat162 *>(A + at) = a;
                *reinterpret_cast<__nv_bfloat162 *>(A + at + W) = lo;
            }
            if (B) {
                const float2 lf = __bfloat1622float2(lo);
                __nv_bfloat162 b = __floats2bfloat162_rn(-2.f * hf.x, -2.f * hf.y);
                if (e + 1 >= d) {
                    if (k0 < 3u) b.x = k0 == 0 ? n1 : k0 == 1 ? n2 : n3;
                    if (k1 < 3u) b.y = k1 == 0 ? n1 : k1 == 1 ? n2 : n3;
                }
                *reinterpret_cast<__nv_bfloat162 *>(B + at) = b;
                *reinterpret_cast<__nv_bfloat162 *>(B + at + W) = __floats2bfloat162_rn(-2.f * lf.x, -2.f * lf.y);
            }
        }
    }
    if (lane == 0) nmax[w] = nm;
    if (large && lane == 0 && bad) atomicOr(large, bad);
    __syncthreads();
    if (ymax && tid == 0) {
        for (int i = 1; i < 8; ++i) nm = fmaxf(nm, nmax[i]);
        atomicMax(ymax, __float_as_uint(nm));
    }
    if (!centre) return;
    if (tid < d) {  // positions without a row hold zeros
        float s = 0.f;
#pragma unroll 16
        for (uint32_t i = 0; i < kTcM; ++i) s = fmaf(tile[(size_t) i * d + tid], scale, s);
        c[tid] = count ? s / (float) count : 0.f;
        centre[(size_t) blockIdx.x * d + tid] = c[tid];
    }
    __syncthreads();
    float m = 0.f;
    for (uint32_t i = w; i < kTcM; i += 8) {
        if (rows[i] == kNone) continue;
        float t = 0.f;
        for (uint32_t e = lane; e < d; e += 32) {
            const float u = fmaf(tile[(size_t) i * d + e], scale, -c[e]);
            t = fmaf(u, u, t);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        m = t > m || t != t ? t : m;  // a NaN stays
    }
    if (lane == 0) rmax[w] = m;
    __syncthreads();
    if (tid == 0) {
        float q = 0.f;
        for (int i = 0; i < 8; ++i) q = rmax[i] > q || rmax[i] != rmax[i] ? rmax[i] : q;
        radius[blockIdx.x] = count ? sqrtf(q) * 1.00002f + 1e-18f : -1e30f;
    }
}

// need[i][t] = 0 when some query of row block i can have a vertex of tile t
// within its radius, else +inf: max(0, |q - c_t| - r_t)^2 <= tau_q for one of
// its 128 queries (scaled here as the balls and radii are), each part rounded to
// the safe side. Per query rather than
// ball against ball: a block's queries may lie in several clusters. One block
// per (row block, 64 tiles), 8 x 4 distances per thread.
//
// Bound by the float32 distances (two operations an element; 10,000 queries x
// 7,813 tiles x 96: 0.42 ms of them). Slices of 16 dimensions are fetched into
// registers while the slice before is worked on and go to the other half of
// shared memory, one barrier a slice: 0.97 ms with loads between two barriers,
// 0.76 ms so.
__global__ void __launch_bounds__(256) tc_need_kernel(const float *__restrict__ q, const uint32_t *__restrict__ qperm,
                                                      uint32_t nq, const float *__restrict__ tau,
                                                      const float *__restrict__ scale_at, const float *__restrict__ cb, const float *__restrict__ rb,
                                                      uint32_t nb, uint32_t d, float *__restrict__ need) {
    __shared__ __align__(16) float sa[2][16][kTcM + 4];
    __shared__ __align__(16) float sb[2][16][68];
    __shared__ float st[kTcM];
    __shared__ uint32_t any[64];
    const uint32_t i0 = blockIdx.y * kTcM, t0 = blockIdx.x * 64, tid = threadIdx.x;
    const uint32_t ty = tid / 16, tx = tid % 16;
    // Thread tid brings 8 values of query tid / 2 and 4 of tile tid / 4 a slice.
    const uint32_t ra = tid / 2, ka = tid % 2 * 8, rc = tid / 4, kc = tid % 4 * 4;
    const float *qr = i0 + ra < nq ? q + (size_t) qperm[i0 + ra] * d : nullptr;
    const float *cr = t0 + rc < nb ? cb + (size_t) (t0 + rc) * d : nullptr;
    if (tid < kTcM) st[tid] = i0 + tid < nq ? tau[i0 + tid] : -1.f;
    if (tid < 64) any[tid] = 0;
    float va[8], vc[4];
    const float scale = *scale_at;
    const bool quads = d % 4 == 0;
    auto fetch4 = [&](const float *r, uint32_t k, float *v) {
        if (quads && r && k < d) {
            const float4 f = __ldg(reinterpret_cast<const float4 *>(r + k));
            v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = !quads && r && k + e < d ? __ldg(r + k + e) : 0.f;
        }
    };
    auto fetch = [&](uint32_t k0) {
        fetch4(qr, k0 + ka, va);
        fetch4(qr, k0 + ka + 4, va + 4);
        fetch4(cr, k0 + kc, vc);
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int e = 0; e < 8; ++e) sa[buf][ka + e][ra] = va[e] * scale;
#pragma unroll
        for (int e = 0; e < 4; ++e) sb[buf][kc + e][rc] = vc[e];
    };
    float acc[8][4] = {};
    fetch(0);
    store(0);
    __syncthreads();
    int buf = 0;
    for (uint32_t k0 = 0; k0 < d; k0 += 16, buf ^= 1) {
        const bool more = k0 + 16 < d;
        if (more) fetch(k0 + 16);
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            float av[8];
            const float4 a0 = *reinterpret_cast<const float4 *>(&sa[buf][kk][ty * 8]);
            const float4 a1 = *reinterpret_cast<const float4 *>(&sa[buf][kk][ty * 8 + 4]);
            const float4 b0 = *reinterpret_cast<const float4 *>(&sb[buf][kk][tx * 4]);
            av[0] = a0.x; av[1] = a0.y; av[2] = a0.z; av[3] = a0.w;
            av[4] = a1.x; av[5] = a1.y; av[6] = a1.z; av[7] = a1.w;
            const float bv[4] = {b0.x, b0.y, b0.z, b0.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float u = av[i] - bv[j];
                    acc[i][j] = fmaf(u, u, acc[i][j]);
                }
        }
        if (more) {
            store(buf ^ 1);
            __syncthreads();
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t tt = t0 + tx * 4 + j;
        if (tt >= nb) continue;
        const float r = rb[tt] * 1.00001f;
        bool hit = false;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float g = sqrtf(acc[i][j]) * 0.99997f - r;
            const float lb = g > 0.f ? g * g * 0.99999f : 0.f;
            hit = hit || (st[ty * 8 + i] >= 0.f && !(lb > st[ty * 8 + i]));
        }
        if (hit) any[tx * 4 + j] = 1u;
    }
    __syncthreads();
    if (tid < 64 && t0 + tid < nb)
        need[(size_t) blockIdx.y * nb + t0 + tid] = any[tid] ? 0.f : __int_as_float(0x7f800000);
}

// lb2[i][t] = a lower bound of the squared distance between any row of ball i
// (rows) and any of ball t (columns): (|c_i - c_t| - r_i - r_t)^2, each part
// rounded to the safe side; 0 when the balls meet. 64 x 64 tiles, 4 x 4 per
// thread.
__global__ void __launch_bounds__(256) tc_bound_kernel(const float *__restrict__ ca, const float *__restrict__ ra,
                                                       uint32_t na, const float *__restrict__ cb,
                                                       const float *__restrict__ rb, uint32_t nb, uint32_t d,
                                                       float *__restrict__ lb2) {
    __shared__ float sa[16][68], sb[16][68];
    const uint32_t i0 = blockIdx.y * 64, t0 = blockIdx.x * 64, tid = threadIdx.x;
    const uint32_t ty = tid / 16, tx = tid % 16;
    float acc[4][4] = {};
    for (uint32_t k0 = 0; k0 < d; k0 += 16) {
        for (uint32_t e = tid; e < 64 * 16; e += 256) {
            const uint32_t rr = e / 16, kk = e % 16;
            sa[kk][rr] = i0 + rr < na && k0 + kk < d ? ca[(size_t) (i0 + rr) * d + k0 + kk] : 0.f;
            sb[kk][rr] = t0 + rr < nb && k0 + kk < d ? cb[(size_t) (t0 + rr) * d + k0 + kk] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            float av[4], bv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                av[j] = sa[kk][ty * 4 + j];
                bv[j] = sb[kk][tx * 4 + j];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float u = av[i] - bv[j];
                    acc[i][j] = fmaf(u, u, acc[i][j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t ii = i0 + ty * 4 + i, tt = t0 + tx * 4 + j;
            if (ii >= na || tt >= nb) continue;
            const float g = sqrtf(acc[i][j]) * 0.99997f - (ra[ii] + rb[tt]) * 1.00001f;
            lb2[(size_t) ii * nb + tt] = g > 0.f ? g * g * 0.99999f : 0.f;
        }
}

// `cells` pivots by farthest-point seeding (Gonzalez, 1985) over S rows at a
// fixed stride, held as BF16 values in the shared memory of one cluster of 8
// CTAs, 128 rows each, four threads a row. Far-apart clusters each get a pivot
// before any gets two, which rows taken at a stride only give with many times
// more of them. BF16 distances only decide which rows are taken.
//
// Bound by the latency of a round: each CTA's farthest row goes to all eight
// (distributed shared memory), one cluster barrier, then every CTA fetches the
// winner's row from its owner. One CTA of 1,024 threads, bound by issue, took
// 3.6 us a round (256 rounds, d = 96); this takes 1.4 us.
constexpr int kPivCtas = 8, kPivRows = 128;

// Words per row: h rounded up to 4 mod 8, so that a warp's 8 rows x 4 words lie in 32 banks.
__host__ __device__ constexpr uint32_t piv_stride(uint32_t h) { return (h + 3) / 8 * 8 + 4; }

__global__ void __cluster_dims__(kPivCtas, 1, 1) __launch_bounds__(4 * kPivRows)
    tc_pivot_kernel(const float *__restrict__ x, uint32_t n, uint32_t d, uint32_t S, uint32_t cells,
                    uint32_t *__restrict__ pivots) {
    extern __shared__ __align__(16) __nv_bfloat162 srow[];  // [kPivRows][piv_stride(h)]
    __shared__ float2 prow[128];                             // the newest pivot's row
    __shared__ unsigned long long wkey[16], keys[2][kPivCtas];
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, h = (d + 1) / 2, hp = piv_stride(h);
    const uint32_t rank = cluster.block_rank(), row = tid / 4, sub = tid % 4, slot = rank * kPivRows + row;
    for (uint32_t e = tid; e < kPivRows * h; e += 4 * kPivRows) {
        const uint32_t i = e / h, q = 2 * (e - i * h), g = rank * kPivRows + i;
        if (g >= S) break;
        const float *r = x + ((uint64_t) g * n / S) * d;
        srow[(size_t) i * hp + q / 2] = __floats2bfloat162_rn(r[q], q + 1 < d ? r[q + 1] : 0.f);
    }
    float mind = 3e38f;
    uint32_t cur = 0;
    cluster.sync();
    for (uint32_t c = 0;; ++c) {
        if (rank == 0 && tid == 0) pivots[c] = (uint32_t) ((uint64_t) cur * n / S);
        if (c + 1 == cells) break;
        if (tid < h) {
            const __nv_bfloat162 *owner = cluster.map_shared_rank(srow, cur / kPivRows);
            prow[tid] = __bfloat1622float2(owner[(size_t) (cur % kPivRows) * hp + tid]);
        }
        __syncthreads();
        float s = 0.f;
        for (uint32_t q = sub; q < h; q += 4) {
            const float2 a = __bfloat1622float2(srow[(size_t) row * hp + q]), b = prow[q];
            const float u = a.x - b.x, v = a.y - b.y;
            s = fmaf(u, u, s);
            s = fmaf(v, v, s);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        mind = fminf(mind, s);
        // (distance, ~slot): the farthest row, ties to the lower slot.
        unsigned long long key = slot < S ? (unsigned long long) __float_as_uint(mind) << 32 | ~slot : 0ull;
#pragma unroll
        for (int o = 4; o < 32; o *= 2) {
            const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, key, o);
            key = k2 > key ? k2 : key;
        }
        if (lane == 0) wkey[w] = key;
        __syncthreads();
        if (w == 0) {
            key = wkey[lane % 16];
#pragma unroll
            for (int o = 1; o < 16; o *= 2) {
                const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, key, o);
                key = k2 > key ? k2 : key;
            }
            if (lane < kPivCtas) *cluster.map_shared_rank(&keys[c & 1][rank], lane) = key;
        }
        // Keys of the next round go to the other half, so one barrier a round is enough.
        cluster.sync();
        key = keys[c & 1][0];
#pragma unroll
        for (int i = 1; i < kPivCtas; ++i) key = keys[c & 1][i] > key ? keys[c & 1][i] : key;
        cur = ~(uint32_t) key;
    }
    cluster.sync();  // no CTA leaves while another may read its rows
}

// Counting sort of the rows by cell: the order within a cell is the order the
// atomics land in, which no result depends on.
__global__ void tc_hist_kernel(const uint32_t *__restrict__ cell, uint32_t n, uint32_t *__restrict__ count) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) atomicAdd(count + cell[i], 1u);
}

__global__ void tc_scatter_kernel(const uint32_t *__restrict__ cell, uint32_t n, uint32_t *__restrict__ start,
                                  uint32_t *__restrict__ perm) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) perm[atomicAdd(start + cell[i], 1u)] = i;
}

// Squared radii in scaled units, rounded up.
__global__ void tc_tau_kernel(const double *__restrict__ tau, uint32_t nq, const float *__restrict__ scale_at,
                              float *__restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const double scale = (double) *scale_at;
    if (i < nq) out[i] = __double2float_ru(tau[i] * (scale * scale));
}

int make_map(CUtensorMap *map, const __nv_bfloat16 *x, uint64_t rows, uint32_t width) {
    cudaDriverEntryPointQueryResult q;
    void *fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
        return set_error(PANNS_ECUDA, "tc screen: cuTensorMapEncodeTiled is not available");
    const auto encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    const cuuint64_t dims[2] = {width, rows};
    const cuuint64_t strides[1] = {(cuuint64_t) width * 2};
    const cuuint32_t box[2] = {kTcSliceW, kTcM};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16 *>(x), dims, strides,
                              box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return set_error(PANNS_ECUDA, "tc screen: cuTensorMapEncodeTiled failed (" + std::to_string((int) r) + ")");
    return PANNS_OK;
}

#define TCU(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return set_error(PANNS_ECUDA, std::string("tc screen: " #call ": ") + cudaGetErrorString(e_)); \
    } while (0)

template <typename T>
using TBuf = Scratch<T>;

struct TcShape {
    uint32_t W, slices, stages, k_hh, k_x;
    size_t smem;
};

TcShape tc_shape(uint32_t d) {
    TcShape s;
    s.W = (d + 3 + kTcSliceW - 1) / kTcSliceW * kTcSliceW;
    s.slices = s.W / kTcSliceW;
    s.k_hh = (d + 3 + 15) / 16;
    s.k_x = (d + 15) / 16;
    s.stages = 4;
    while (s.stages > 2 && tc_layout(s.slices, s.stages).total + 1024 > 227u * 1024u) --s.stages;
    s.smem = tc_layout(s.slices, s.stages).total + 1024;
    return s;
}

template <int FORM>
int tc_launch(const CUtensorMap &ma, const CUtensorMap &mb, const TcArgs &a, size_t smem, int num_sms, cudaStream_t s) {
    TCU(allow_shared((const void *) tc_screen_kernel<FORM>));
    TCU(cudaMemsetAsync(a.counter, 0, 4, s));
    tc_screen_kernel<FORM><<<std::min<uint32_t>(a.items, (uint32_t) num_sms), kTcThreads, smem, s>>>(ma, mb, a);
    TCU(cudaGetLastError());
    return PANNS_OK;
}

int tc_check(const uint32_t *error, cudaStream_t s) {
    uint32_t herr = 0;
    TCU(cudaMemcpyAsync(&herr, error, 4, cudaMemcpyDeviceToHost, s));
    TCU(cudaStreamSynchronize(s));
    if (herr) return set_error(PANNS_EDEVICE, "tc screen: an mbarrier wait expired");
    return PANNS_OK;
}

}  // namespace

bool tc_screen_supported(uint32_t n, uint32_t d, uint32_t C) {
    return d % 32 == 0 && d >= 32 && d <= 128 && C >= 1 && C <= 128 && C < n && n >= kTcM;
}

// 32 rows a pivot (two tiles' worth where cells are padded) up to 256 pivots: they
// are chosen one after the other (256 take 0.37 ms), and on a base of 64 clusters
// 64 are enough.
static uint32_t tc_pivots(uint32_t n, bool padded) {
    return std::max(1u, std::min(256u, n / (padded ? 2 * kTcM : 32)));
}

uint32_t tc_order_slots(uint32_t n, bool padded) { return padded ? n + tc_pivots(n, true) * (kTcM - 1) : n; }

int tc_locality_order(const float *x, uint32_t n, uint32_t d, bool padded, uint32_t *perm, uint32_t *slots,
                      cudaStream_t s) {
    if (d == 0 || d > 256) return set_error(PANNS_EINVAL, "tc screen: unsupported shape");
    const uint32_t cells = tc_pivots(n, padded);
    const uint32_t h = (d + 1) / 2, S = std::min(n, (uint32_t) (kPivCtas * kPivRows));
    const uint32_t psmem = kPivRows * piv_stride(h) * 4;
    std::vector<uint32_t> count(cells);
    TBuf<uint32_t> dpiv, cell, start;
    TCU(dpiv.alloc(cells, s));
    TCU(cell.alloc(n, s));
    TCU(start.alloc(cells, s));
    TCU(allow_shared((const void *) tc_pivot_kernel));
    tc_pivot_kernel<<<kPivCtas, 4 * kPivRows, psmem, s>>>(x, n, d, S, cells, dpiv.p);
    TCU(cudaGetLastError());
    const int rc = nearest_center(x, n, d, dpiv.p, cells, cell.p, s);
    if (rc) return rc;
    TCU(cudaMemsetAsync(start.p, 0, cells * 4ull, s));
    tc_hist_kernel<<<(n + 255) / 256, 256, 0, s>>>(cell.p, n, start.p);
    TCU(cudaGetLastError());
    TCU(cudaMemcpyAsync(count.data(), start.p, cells * 4ull, cudaMemcpyDeviceToHost, s));
    TCU(cudaStreamSynchronize(s));
    uint32_t at = 0;
    for (uint32_t c = 0; c < cells; ++c) {
        const uint32_t m = count[c];
        count[c] = at;
        at += padded ? (m + kTcM - 1) / kTcM * kTcM : m;
    }
    *slots = at;
    TCU(cudaMemcpyAsync(start.p, count.data(), cells * 4ull, cudaMemcpyHostToDevice, s));
    TCU(cudaMemsetAsync(perm, 0xff, (size_t) at * 4, s));
    tc_scatter_kernel<<<(n + 255) / 256, 256, 0, s>>>(cell.p, n, start.p, perm);
    TCU(cudaGetLastError());
    TCU(cudaStreamSynchronize(s));
    return PANNS_OK;
}

int tc_screen_knn(const float *x, uint32_t n, uint32_t d, uint32_t k, uint32_t C, const uint32_t *perm, uint32_t slots,
                  const TcCells *cells, uint32_t *cand, uint32_t *fail_rows, uint32_t *fail_count, bool *safe,
                  int num_sms, cudaStream_t s) {
    if (d == 0 || d > 256 || k == 0 || k + 1 > kTcCap - kTcM || C < k || n < 2)
        return set_error(PANNS_EINVAL, "tc screen: unsupported shape");
    const TcShape sh = tc_shape(d);
    const uint32_t tiles = (slots + kTcM - 1) / kTcM, pad = tiles * kTcM;
    TBuf<__nv_bfloat16> A, B;
    TBuf<float> xn, centre, radius, lb2, frame;
    TBuf<uint2> lists;
    TBuf<uint32_t> ctl;  // counter, error, ymax, large, spread
    // Row operands and bounds between tiles for a limited number of row blocks at a time.
    const bool skip = !cells && tiles > 32;
    uint32_t per = std::min(tiles, kTcKnnBlocks);
    if (skip) {
        per = std::min<uint32_t>(per, std::max<uint32_t>(4u * num_sms, (1u << 28) / tiles));
        TCU(centre.alloc((size_t) tiles * d, s));
        TCU(radius.alloc(tiles, s));
        TCU(lb2.alloc((size_t) per * tiles, s));
    }
    TCU(A.alloc((size_t) per * kTcM * 2 * sh.W, s));
    TCU(B.alloc((size_t) pad * 2 * sh.W, s));
    TCU(xn.alloc(pad, s));
    TCU(ctl.alloc(5, s));
    TCU(cudaMemsetAsync(ctl.p, 0, 20, s));
    TCU(cudaMemsetAsync(fail_count, 0, 4, s));
    TCU(frame.alloc(d + 1, s));
    tc_shift_kernel<<<d, 256, 0, s>>>(x, n, d, frame.p, ctl.p + 4);
    tc_frame_kernel<<<1, 256, 0, s>>>(frame.p, ctl.p + 4, d);
    TCU(allow_shared((const void *) tc_prepare_kernel));
    tc_prepare_kernel<<<tiles, 256, kTcM * d * 4, s>>>(x, n, d, perm, 0, slots, sh.W, frame.p,
                                                       per == tiles ? A.p : nullptr, B.p, xn.p, ctl.p + 2, ctl.p + 3,
                                                       centre.p, radius.p);
    TCU(cudaGetLastError());
    TCU(lists.alloc((size_t) std::min<uint32_t>(per, (uint32_t) num_sms) * kTcM * kTcCap, s));
    CUtensorMap ma, mb;
    int rc = make_map(&ma, A.p, (uint64_t) per * kTcM, 2 * sh.W);
    if (!rc) rc = make_map(&mb, B.p, pad, 2 * sh.W);
    if (rc) return rc;
    for (uint32_t rb0 = 0; rb0 < tiles; rb0 += per) {
        const uint32_t m = std::min(per, tiles - rb0);
        if (per != tiles) {
            tc_prepare_kernel<<<m, 256, kTcM * d * 4, s>>>(x, n, d, perm, rb0 * kTcM, slots, sh.W, frame.p, A.p,
                                                           nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
            TCU(cudaGetLastError());
        }
        if (skip) {
            tc_bound_kernel<<<dim3((tiles + 63) / 64, (m + 63) / 64), 256, 0, s>>>(
                centre.p + (size_t) rb0 * d, radius.p + rb0, m, centre.p, radius.p, tiles, d, lb2.p);
            TCU(cudaGetLastError());
        }
        TcArgs a{};
        a.rows = slots;
        a.rb0 = rb0;
        a.items = m;
        a.splits = 1;
        a.tiles = tiles;
        a.slices = sh.slices;
        a.stages = sh.stages;
        a.k_hh = sh.k_hh;
        a.k_x = sh.k_x;
        a.lb2 = skip ? lb2.p : nullptr;
        a.xn = xn.p;
        a.ymax = ctl.p + 2;
        a.lists = lists.p;
        a.cap = kTcCap;
        a.counter = ctl.p;
        a.error = ctl.p + 1;
        a.k = k;
        a.C = C;
        a.perm = perm;
        a.cand = cand;
        a.fail_rows = fail_rows;
        a.fail_count = fail_count;
        if (cells) {
            a.blk_cell = cells->blk_cell;
            a.cell_tile0 = cells->tile0;
            a.near = cells->near;
            a.avail = cells->avail;
            a.P = cells->P;
        }
        rc = tc_launch<TC_KNN>(ma, mb, a, sh.smem, num_sms, s);
        if (rc) return rc;
    }
    uint32_t large = 0;
    TCU(cudaMemcpyAsync(&large, ctl.p + 3, 4, cudaMemcpyDeviceToHost, s));
    rc = tc_check(ctl.p + 1, s);
    *safe = !(large & TC_NORM_LARGE);
    return rc;
}

size_t tc_knn_bytes(uint64_t slots, uint32_t d) {
    const size_t row = (size_t) tc_shape(d).W * 4;
    return (size_t) (slots + kTcM) * (row + 4) + std::min<size_t>(slots + kTcM, (size_t) kTcKnnBlocks * kTcM) * row +
           (64u << 20);
}

uint32_t tc_range_splits(uint32_t nq, int num_sms) {
    const uint32_t rb = (nq + kTcM - 1) / kTcM;
    return std::max(1u, std::min(kTcMaxSplits, (2u * (uint32_t) num_sms + rb - 1) / std::max(rb, 1u)));
}

int tc_screen_range(const float *x, uint32_t n, uint32_t d, const uint32_t *perm, uint32_t slots,
                    const float *queries, const uint32_t *qperm, uint32_t nq, const double *tau, uint32_t splits,
                    uint2 *lists, uint32_t cap, uint32_t *cnt, bool *safe, int num_sms, cudaStream_t s) {
    if (d == 0 || d > 256 || nq == 0 || splits == 0) return set_error(PANNS_EINVAL, "tc screen: unsupported shape");
    const TcShape sh = tc_shape(d);
    const uint32_t rb = (nq + kTcM - 1) / kTcM, qpad = rb * kTcM;
    // Columns in chunks, so that the operand copy stays below about 2 GB and
    // the tile lists below 1 GB at any base size.
    const uint64_t by_rows = (1ull << 31) / (4ull * sh.W), by_need = (1ull << 28) / rb * kTcM;
    const uint32_t chunk =
        (uint32_t) std::min<uint64_t>((slots + kTcM - 1) / kTcM * (uint64_t) kTcM,
                                      std::max<uint64_t>(kTcM, std::min(by_rows, by_need) / kTcM * kTcM));
    const uint32_t ct = chunk / kTcM;
    TBuf<__nv_bfloat16> A, B;
    TBuf<float> xn, cb, rad, need, ft, frame;
    TBuf<uint32_t> ctl;  // counter, error, ymax, large, spread
    TCU(A.alloc((size_t) qpad * 2 * sh.W, s));
    TCU(B.alloc((size_t) chunk * 2 * sh.W, s));
    TCU(xn.alloc(qpad, s));
    TCU(cb.alloc((size_t) ct * d, s));
    TCU(rad.alloc(ct, s));
    TCU(need.alloc((size_t) rb * ct, s));
    TCU(ft.alloc(nq, s));
    TCU(frame.alloc(d + 1, s));
    TCU(ctl.alloc(5, s));
    TCU(cudaMemsetAsync(ctl.p, 0, 20, s));
    TCU(cudaMemsetAsync(cnt, 0, (size_t) splits * nq * 4, s));
    tc_shift_kernel<<<d, 256, 0, s>>>(x, n, d, frame.p, ctl.p + 4);
    tc_frame_kernel<<<1, 256, 0, s>>>(frame.p, ctl.p + 4, d);
    tc_tau_kernel<<<(nq + 255) / 256, 256, 0, s>>>(tau, nq, frame.p + d, ft.p);
    TCU(allow_shared((const void *) tc_prepare_kernel));
    tc_prepare_kernel<<<rb, 256, kTcM * d * 4, s>>>(queries, kNone, d, qperm, 0, nq, sh.W, frame.p, A.p, nullptr,
                                                    xn.p, nullptr, ctl.p + 3, nullptr, nullptr);
    TCU(cudaGetLastError());
    CUtensorMap ma, mb;
    int rc = make_map(&ma, A.p, qpad, 2 * sh.W);
    if (!rc) rc = make_map(&mb, B.p, chunk, 2 * sh.W);
    if (rc) return rc;
    for (uint64_t c0 = 0; c0 < slots; c0 += chunk) {
        const uint32_t m = (uint32_t) std::min<uint64_t>(chunk, slots - c0), mt = (m + kTcM - 1) / kTcM;
        TCU(cudaMemsetAsync(ctl.p + 2, 0, 4, s));
        tc_prepare_kernel<<<mt, 256, kTcM * d * 4, s>>>(x, n, d, perm, (uint32_t) c0, slots, sh.W, frame.p, nullptr,
                                                        B.p, nullptr, ctl.p + 2, ctl.p + 3, cb.p, rad.p);
        tc_need_kernel<<<dim3((mt + 63) / 64, rb), 256, 0, s>>>(queries, qperm, nq, ft.p, frame.p + d, cb.p, rad.p,
                                                                mt, d, need.p);
        TCU(cudaGetLastError());
        TcArgs a{};
        a.rows = nq;
        a.rb0 = 0;
        a.items = rb * splits;
        a.splits = splits;
        a.tiles = mt;
        a.slices = sh.slices;
        a.stages = sh.stages;
        a.k_hh = sh.k_hh;
        a.k_x = sh.k_x;
        a.lb2 = need.p;
        a.xn = xn.p;
        a.ymax = ctl.p + 2;
        a.lists = lists;
        a.cap = cap;
        a.counter = ctl.p;
        a.error = ctl.p + 1;
        a.perm = perm;
        a.tau = ft.p;
        a.cnt = cnt;
        a.id0 = (uint32_t) c0;
        rc = tc_launch<TC_RANGE>(ma, mb, a, sh.smem, num_sms, s);
        if (rc) return rc;
    }
    uint32_t large = 0;
    TCU(cudaMemcpyAsync(&large, ctl.p + 3, 4, cudaMemcpyDeviceToHost, s));
    rc = tc_check(ctl.p + 1, s);
    *safe = !large;
    return rc;
}

}  // namespace panns
