// Several warps per query: the same search as search_kernel (PANNS order; the
// float32 rows, or a BF16 / FP8 copy with the exact float32 re-rank of the
// final L), for small batches where one warp per query leaves the GPU idle and
// every query pays the whole serial latency, and for long queues.
//
// One block of W warps runs one query at a time (work-stealing counter across
// blocks). The queue lives in the block's shared memory. A search step is:
//   1. every warp finds the M best unchecked candidates by itself (the queue
//      does not change meanwhile; they are marked after the next barrier);
//   2. in rounds, the warps expand candidates (at most G per warp and round, G *
//      degree <= buffer so a warp's fresh buffer cannot overflow; several warps
//      share a candidate's row when there are fewer candidates than warps): head
//      rows, visited test-and-set on the block's bitset, distances, the filter
//      against the queue's L-th distance at the start of the round; the
//      survivors of all warps are appended to one list;
//   3. that list is ranked by counting (a thread, or several, per element; a
//      bitonic network when it is long), each element's place in the queue is
//      found by binary search, and the queue's elements move up by the number
//      of list elements before them, read and written in chunks of registers.
// Each round's merge leaves the queue equal to the L best of (queue + round
// survivors), and the round's first insert position is the best survivor's,
// exactly as one flush of search_kernel (see the exactness note there), so
// ids and distance counts equal search_kernel's and the reference's.
//
// Bound by latency: a step is a chain of dependent loads (head row, visited
// word, rows) and of barriers. The form before sorted every warp's survivors,
// placed W lists into one by serial binary searches and moved the queue one
// element per thread and barrier pair, with the original ids loaded for every
// survivor (here only when two distances are equal): nine barriers a step, four
// now.
#pragma once

#include "search_kernel.cuh"

namespace panns {

constexpr int kBlockCtl = 16;  // control words in shared memory
// Longest list ranked by counting; above, the bitonic network (initial queues).
__host__ __device__ constexpr uint32_t block_rank_max(uint32_t W) { return 64u * W; }

// Shared memory of one block of W warps with a queue of queue_cap entries and
// warp buffers of buf.
__host__ __device__ inline uint32_t block_smem_bytes(uint32_t queue_cap, uint32_t W, uint32_t buf, uint32_t vis_smem) {
    return queue_cap * 8u                     // queue (dist, id)
           + W * buf * 8u                     // per-warp fresh ids and distances
           + W * buf * 12u                    // survivors of a round (dist, id, key)
           + block_rank_max(W) * 12u          // ranked survivors (dist, id, place)
           + W * kMaxM * 8u                   // per-warp picked candidates (id, place) / learned entries
           + W * 1024u                        // per-warp distance chains
           + kBlockCtl * 4u                   // control words
           + vis_smem * 4u;                   // visited bitset, where it fits
}

enum { BC_Q = 0, BC_CNT, BC_CNT2, BC_TIE, BC_DIST, BC_EDGES, BC_FULL };

// Total order of distances for ranking equal ones: floats as unsigned integers
// that compare the same way.
__device__ __forceinline__ uint32_t dist_key(float d) {
    const uint32_t b = __float_as_uint(d + 0.0f);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}

template <int W>
struct BlockMem {
    float *qd;
    uint32_t *qi;
    float *cD;       // survivors of the round
    uint32_t *cI, *cK;
    float *sD;       // ranked survivors
    uint32_t *sI, *sP;
    uint32_t *ctl;
};

// Ranks of the n <= block_rank_max(W) survivors by (distance, original id):
// writes (sD, sI) in that order and, with PLACE, sP = the number of queue
// elements (qd, qi)[0..sz) before each. Several adjacent threads count for one
// element when there are fewer elements than threads; the counts of smaller and
// of smaller or equal distances differ by more than the element itself only
// where distances are equal: then the block counts again by (distance,
// original id), a total order. Called by the whole block after a barrier; ends
// with one.
template <int W, bool PLACE>
__device__ __forceinline__ void block_rank(const BlockMem<W> &m, uint32_t n, uint32_t sz,
                                           const uint32_t *__restrict__ orig) {
    constexpr uint32_t T = W * 32;
    const uint32_t tid = threadIdx.x;
    const float4 *c4 = reinterpret_cast<const float4 *>(m.cD);
    const uint32_t quads = n / 4;
    if (n <= T / 4) {
        // Short lists (the usual case): eight lanes per element, which also
        // search the queue together, eight ways a step.
        const uint32_t part = tid & 7u, shift = tid & 24u;
        uint32_t width = 1;  // the search's first stride: sz <= 8 * width
        while (PLACE && width * 8 < sz) width *= 8;
        for (uint32_t e0 = 0; e0 < n; e0 += T / 8) {
            const uint32_t e = e0 + tid / 8;
            if (e0 + (tid & ~31u) / 8 >= n) break;  // warp-uniform
            const float d = e < n ? m.cD[e] : 0.f;
            const uint32_t id = e < n ? m.cI[e] : 0u;
            uint32_t less = 0, upto = 0;
            for (uint32_t q = part; q < quads; q += 8) {
                const float4 x = c4[q];
                less += (x.x < d ? 1u : 0u) + (x.y < d ? 1u : 0u) + (x.z < d ? 1u : 0u) + (x.w < d ? 1u : 0u);
                upto += (x.x <= d ? 1u : 0u) + (x.y <= d ? 1u : 0u) + (x.z <= d ? 1u : 0u) + (x.w <= d ? 1u : 0u);
            }
            if (4 * quads + part < n) {
                const float x = m.cD[4 * quads + part];
                less += x < d ? 1u : 0u;
                upto += x <= d ? 1u : 0u;
            }
            uint32_t both = less | upto << 16;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) both += __shfl_xor_sync(kFull, both, o);
            less = both & 0xffffu;
            upto = both >> 16;
            uint32_t place = 0;
            if (PLACE) {
                for (uint32_t wd = width; wd > 0; wd /= 8) {
                    const uint32_t p = place + (part + 1) * wd - 1;
                    bool before = false;
                    if (p < sz) {
                        const float md = m.qd[p];
                        before = md < d ||
                                 (md == d && __ldg(orig + (m.qi[p] & kIdMask)) < __ldg(orig + (id & kIdMask)));
                    }
                    place += wd * __popc((__ballot_sync(kFull, before) >> shift) & 0xffu);
                }
            }
            if (e < n && part == 0) {
                if (upto != less + 1) m.ctl[BC_TIE] = 1u;
                const uint32_t r = min(less, n - 1);
                m.sD[r] = d;
                m.sI[r] = id;
                if (PLACE) m.sP[r] = place;
            }
        }
    } else {
        uint32_t parts = 1;  // threads per element
        while (parts < 4 && n * parts * 2 <= T) parts *= 2;
        const uint32_t per = T / parts;  // elements per pass
        const uint32_t share = (quads + parts - 1) / parts;
        const uint32_t part = tid & (parts - 1);
        for (uint32_t e0 = 0; e0 < n; e0 += per) {  // block-uniform: the shuffles are too
            const uint32_t e = e0 + tid / parts;
            const float d = e < n ? m.cD[e] : 0.f;
            uint32_t less = 0, upto = 0;
            const uint32_t q1 = min(quads, (part + 1) * share);
#pragma unroll 2
            for (uint32_t q = part * share; q < q1; ++q) {
                const float4 x = c4[q];
                less += (x.x < d ? 1u : 0u) + (x.y < d ? 1u : 0u) + (x.z < d ? 1u : 0u) + (x.w < d ? 1u : 0u);
                upto += (x.x <= d ? 1u : 0u) + (x.y <= d ? 1u : 0u) + (x.z <= d ? 1u : 0u) + (x.w <= d ? 1u : 0u);
            }
            if (part == 0)
                for (uint32_t f = 4 * quads; f < n; ++f) {
                    less += m.cD[f] < d ? 1u : 0u;
                    upto += m.cD[f] <= d ? 1u : 0u;
                }
            for (uint32_t o = 1; o < parts; o <<= 1) {
                less += __shfl_xor_sync(kFull, less, o);
                upto += __shfl_xor_sync(kFull, upto, o);
            }
            if (e < n && part == 0) {
                if (upto != less + 1) m.ctl[BC_TIE] = 1u;
                const uint32_t r = min(less, n - 1), id = m.cI[e];
                m.sD[r] = d;
                m.sI[r] = id;
                if (PLACE) m.sP[r] = queue_rank<ORDER_PANNS>(m.qd, m.qi, sz, d, id & kIdMask, orig);
            }
        }
    }
    __syncthreads();
    if (m.ctl[BC_TIE]) {  // block-uniform
        for (uint32_t e = tid; e < n; e += T) m.cK[e] = __ldg(orig + (m.cI[e] & kIdMask));
        __syncthreads();
        if (tid == 0) m.ctl[BC_TIE] = 0u;
        for (uint32_t e = tid; e < n; e += T) {
            const float d = m.cD[e];
            const uint32_t kd = dist_key(d), ko = m.cK[e], id = m.cI[e];
            uint32_t r = 0;
            for (uint32_t f = 0; f < n; ++f) {
                const uint32_t fd = dist_key(m.cD[f]);
                r += fd < kd || (fd == kd && m.cK[f] < ko) ? 1u : 0u;
            }
            m.sD[r] = d;
            m.sI[r] = id;
            if (PLACE) m.sP[r] = queue_rank<ORDER_PANNS>(m.qd, m.qi, sz, d, id & kIdMask, orig);
        }
        __syncthreads();
    }
}

// Block-wide bitonic sort of the n survivors by (distance, original id), in
// place (the arrays hold a power of two >= n entries).
template <int W>
__device__ __forceinline__ void block_bitonic(const BlockMem<W> &m, uint32_t n, const uint32_t *__restrict__ orig) {
    constexpr uint32_t T = W * 32;
    const uint32_t tid = threadIdx.x;
    uint32_t p2 = 64;
    while (p2 < n) p2 <<= 1;
    for (uint32_t e = tid; e < p2; e += T) {
        if (e < n) {
            m.cK[e] = __ldg(orig + (m.cI[e] & kIdMask));
        } else {
            m.cD[e] = __int_as_float(0x7f800000);
            m.cI[e] = kFull;
            m.cK[e] = kFull;
        }
    }
    __syncthreads();
    for (uint32_t k = 2; k <= p2; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t p = tid; p < (p2 >> 1); p += T) {
                const uint32_t i = ((p & ~(j - 1)) << 1) | (p & (j - 1)), x = i | j;
                const float ad = m.cD[i], xd = m.cD[x];
                const uint32_t ak = m.cK[i], xk = m.cK[x];
                const bool up = (i & k) == 0;
                if (up ? plain_less(xd, xk, ad, ak) : plain_less(ad, ak, xd, xk)) {
                    m.cD[i] = xd;
                    m.cD[x] = ad;
                    m.cK[i] = xk;
                    m.cK[x] = ak;
                    const uint32_t t = m.cI[i];
                    m.cI[i] = m.cI[x];
                    m.cI[x] = t;
                }
            }
            __syncthreads();
        }
}

// Merge the n survivors (cD, cI) into the queue of size sz and capacity L.
// Returns the position of the best one (L when none is inserted); sz is
// updated. Called by the whole block with n and sz uniform, after a barrier;
// ends with one.
template <int W>
__device__ __forceinline__ uint32_t block_merge(const BlockMem<W> &m, uint32_t n, uint32_t &sz, uint32_t L,
                                                const uint32_t *__restrict__ orig) {
    constexpr uint32_t T = W * 32;
    constexpr int CH = 4;  // queue elements a thread moves between two barriers
    const uint32_t tid = threadIdx.x;
    if (n == 0) {
        __syncthreads();
        return L;
    }
    const float *sD = m.sD;
    const uint32_t *sI = m.sI;
    uint32_t *sP = m.sP;
    if (n <= block_rank_max(W)) {
        block_rank<W, true>(m, n, sz, orig);
    } else {
        block_bitonic<W>(m, n, orig);
        sD = m.cD;
        sI = m.cI;
        sP = m.cK;
        for (uint32_t i = tid; i < n; i += T)
            sP[i] = queue_rank<ORDER_PANNS>(m.qd, m.qi, sz, sD[i], sI[i] & kIdMask, orig);
        __syncthreads();
    }
    const uint32_t p0 = sP[0];
    const uint32_t end = min(L, sz + n);
    if (p0 >= L) {
        __syncthreads();  // sP is read before the next round writes it
        return L;
    }
    // A queue element moves up by the number of survivors before it: those
    // whose own count of queue elements before them is at most its index.
    const uint32_t steps = 32 - __clz(n);  // 2^steps > n
    uint32_t top = sz;
    while (true) {
        float d[CH];
        uint32_t id[CH], np[CH];
        if (top - p0 > T) {
            uint32_t j[CH], lo[CH];  // lo: survivors with sP <= j
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const uint32_t back = c * T + tid + 1;
                const bool have = back <= top - p0;
                j[c] = have ? top - back : 0u;
                d[c] = m.qd[j[c]];
                id[c] = m.qi[j[c]];
                lo[c] = 0;
                np[c] = have ? j[c] : L;
            }
            for (uint32_t b = 1u << (steps - 1); b > 0; b >>= 1) {
#pragma unroll
                for (int c = 0; c < CH; ++c)
                    if (lo[c] + b <= n && sP[lo[c] + b - 1] <= j[c]) lo[c] += b;
            }
#pragma unroll
            for (int c = 0; c < CH; ++c) np[c] += lo[c];
        } else {  // one element a thread
#pragma unroll
            for (int c = 1; c < CH; ++c) np[c] = L;
            const bool have = (uint32_t) tid < top - p0;
            const uint32_t j = have ? top - 1 - tid : 0u;
            d[0] = m.qd[j];
            id[0] = m.qi[j];
            uint32_t lo = 0;
            for (uint32_t b = 1u << (steps - 1); b > 0; b >>= 1)
                if (lo + b <= n && sP[lo + b - 1] <= j) lo += b;
            np[0] = have ? j + lo : L;
        }
        const bool last = top <= p0 + CH * T;
        __syncthreads();
#pragma unroll
        for (int c = 0; c < CH; ++c)
            if (np[c] < L) {
                m.qd[np[c]] = d[c];
                m.qi[np[c]] = id[c];
            }
        if (last) break;
        top -= CH * T;  // (the next chunk reads below what this one wrote)
    }
    for (uint32_t i = tid; i < n; i += T) {
        const uint32_t np = i + sP[i];
        if (np < L) {
            m.qd[np] = sD[i];
            m.qi[np] = sI[i];
        }
    }
    sz = end;
    __syncthreads();
    return p0;
}

template <int KIND, int CL, int W, int STORE>
__device__ void block_search_one(const SearchArgs &a, uint32_t q, uint8_t *smem, uint32_t *vis, uint32_t *dirty) {
    constexpr uint32_t T = W * 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    BlockMem<W> m;
    m.qd = reinterpret_cast<float *>(smem);
    m.qi = reinterpret_cast<uint32_t *>(m.qd + a.queue_cap);
    const uint32_t buf = a.block_buf;
    float *bd = reinterpret_cast<float *>(m.qi + a.queue_cap) + w * buf;
    uint32_t *bi = m.qi + a.queue_cap + W * buf + w * buf;
    m.cD = reinterpret_cast<float *>(m.qi + a.queue_cap + 2 * W * buf);
    m.cI = reinterpret_cast<uint32_t *>(m.cD + W * buf);
    m.cK = m.cI + W * buf;
    m.sD = reinterpret_cast<float *>(m.cK + W * buf);
    m.sI = reinterpret_cast<uint32_t *>(m.sD + block_rank_max(W));
    m.sP = m.sI + block_rank_max(W);
    uint32_t *cand = m.sP + block_rank_max(W) + w * 2 * kMaxM;
    uint32_t *cpos = cand + kMaxM;  // the candidates' places in the queue
    float *tmp = reinterpret_cast<float *>(m.sP + block_rank_max(W) + W * 2 * kMaxM) + w * 256;
    m.ctl = m.sP + block_rank_max(W) + W * 2 * kMaxM + W * 256;
    uint32_t *ctl = m.ctl;
    uint32_t *svis = ctl + kBlockCtl;
    const bool in_smem = a.vis_smem != 0;

    uint32_t L = a.Lq ? __ldg(a.Lq + q) : a.L;
    // Init ids: n_lrn learned entries (cand) then n_plain of the init list.
    uint32_t n_lrn = 0, n_plain = L;
    if (a.decisions) {
        const uint2 r = mlp_read_decision(a.decisions, a.dec_L_init, q, cand, lane);  // every warp its own copy
        n_lrn = r.x & 0xffu;
        n_plain = r.x >> 8;
        L = r.y;
    }
    const uint32_t n_init = n_lrn + n_plain;
    Dist<KIND, CL, STORE> D;
    D.load(a, q, lane);
    if (tid < kBlockCtl && tid != BC_Q) ctl[tid] = 0;
    for (uint32_t i = tid; i < a.vis_smem; i += T) svis[i] = 0;
    __syncthreads();

    uint32_t sz = 0, dcount = 0, n_dist = 0, n_edges = 0, n_expand = 0, n_iter = 0;
    // The warp's part of the list of visited words that went from zero to non-zero.
    const uint32_t dcap = a.dirty_cap / W;
    uint32_t *my_dirty = dirty + (size_t) w * dcap;
    uint32_t turn = 0;  // which of the two list counters the round uses

    // Test-and-set of a vertex's visited bit: was it clear? In shared memory
    // where the bitset fits beside the queue without costing resident blocks
    // (an atomic there takes a tenth of one in L2, and nothing is left to
    // clear), else in the block's slot of global memory.
    auto visit = [&](uint32_t id, bool valid) -> bool {
        const uint32_t bit = 1u << (id & 31);
        if (in_smem) return valid && !(atomicOr(svis + (id >> 5), bit) & bit);
        const uint32_t old = visit_issue(vis, id, valid);
        note_dirty(my_dirty, dcap, dcount, valid && old == 0, id >> 5);
        return valid && !(old & bit);
    };
    // Distances of the warp's fresh vertices, the filter against the queue's
    // L-th, the survivors appended to the round's list.
    auto finish_list = [&](uint32_t nb, bool filter) {
        if (nb) {
            if constexpr (STORE == STORE_FP32) {
                // 16 rows a pass; eight or fewer left over in a pass of eight
                const uint32_t wide = (nb & 15u) > 8u ? nb : nb & ~15u;
                if (wide) distances_wide<KIND, CL>(a, D.qv, bi, bd, wide, lane, tmp);
                if (wide < nb) D.distances(a, bi + wide, bd + wide, nb - wide, lane, tmp);
            } else {
                D.distances(a, bi, bd, nb, lane, tmp);
            }
        }
        n_dist += nb;
        const bool any_bound = filter && sz >= L;
        const float bound = any_bound ? m.qd[L - 1] : __int_as_float(0x7f800000);
        for (uint32_t b0 = 0; b0 < nb; b0 += 32) {
            const uint32_t b = b0 + lane;
            const float d = b < nb ? bd[b] : 0.f;
            const bool keep = b < nb && (!any_bound || !(d > bound));
            const uint32_t bm = __ballot_sync(kFull, keep);
            if (!bm) continue;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&ctl[BC_CNT + turn], (uint32_t) __popc(bm));
            base = __shfl_sync(kFull, base, 0);
            if (keep) {
                const uint32_t pos = base + __popc(bm & lanemask_lt());
                m.cD[pos] = d;
                m.cI[pos] = bi[b];
            }
        }
    };
    // The barrier after finish_list, and the list's length. The rounds count
    // alternately in two words: the other one is cleared here, which the
    // barriers of block_merge put before its next use.
    auto close_list = [&]() -> uint32_t {
        __syncthreads();
        const uint32_t n = ctl[BC_CNT + turn];
        turn ^= 1u;
        if (tid == 0) ctl[BC_CNT + turn] = 0;
        return n;
    };

    // Initial queue: the init ids (learned entries first, a repeated id
    // entering once), spread evenly over the warps.
    const uint32_t *init = a.init_ids + (size_t) q * a.init_stride;
    for (uint32_t r0 = 0; r0 < n_init; r0 += W * buf) {
        const uint32_t rest = min(n_init - r0, W * buf);
        const uint32_t per = ((rest + W - 1) / W + 15) & ~15u;  // <= buf, whole distance passes
        uint32_t nb = 0;
        const uint32_t lo = r0 + w * per, hi = min(r0 + rest, lo + per);
        for (uint32_t i0 = lo; i0 < hi; i0 += 32) {
            const uint32_t i = i0 + lane;
            const bool valid = i < hi;
            const uint32_t id = valid ? (i < n_lrn ? cand[i] : __ldg(init + (i - n_lrn))) : 0u;
            const bool ok = valid && id < a.n;
            if (valid && !ok) atomicOr(a.error, ERR_BAD_INIT);
            const bool fresh = visit(id, ok);
            const uint32_t bm = __ballot_sync(kFull, fresh);
            if (fresh) bi[nb + __popc(bm & lanemask_lt())] = id;
            nb += __popc(bm);
            __syncwarp();
        }
        finish_list(nb, false);
        const uint32_t n = close_list();
        block_merge<W>(m, n, sz, L, a.orig);
    }

    const uint32_t M = a.M, G = a.block_round;
    uint32_t k = 0;
    for (;;) {
        // 1. The step's candidates: every warp scans for itself, four entries
        // a lane (the queue's room is a multiple of 32).
        uint32_t cnt = 0, last_k = L;
        for (uint32_t p0 = k & ~3u; p0 < sz && cnt < M; p0 += 128) {
            const uint32_t p = p0 + 4 * lane;
            uint4 e = make_uint4(kChecked, kChecked, kChecked, kChecked);
            if (p < sz) e = *reinterpret_cast<const uint4 *>(m.qi + p);
            const uint32_t v[4] = {e.x, e.y, e.z, e.w};
            bool un[4];
            uint32_t before = 0, total = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                un[i] = !(v[i] & kChecked) && p + i >= k && p + i < sz;
                const uint32_t bm = __ballot_sync(kFull, un[i]);
                before += __popc(bm & lanemask_lt());
                total += __popc(bm);
            }
            uint32_t r = cnt + before, mine = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (un[i]) {
                    if (r < M) {
                        cand[r] = v[i];
                        cpos[r] = p + i;
                        mine = p + i + 1;
                    }
                    ++r;
                }
            mine = __reduce_max_sync(kFull, mine);
            if (mine) last_k = mine - 1;
            cnt = min(M, cnt + total);
        }
        __syncwarp();
        if (cnt == 0) break;  // block-uniform
        ++n_iter;
        n_expand += cnt;
        uint32_t nk = L;
        // Warps per candidate when there are fewer candidates than warps.
        uint32_t parts = 1;
        while (parts < W && cnt * parts * 2 <= W) parts *= 2;
        const uint32_t lead = W / parts;  // candidates expanded at once
        const uint32_t ci = w / parts, part = w & (parts - 1);
        // 2-3. Rounds of at most G candidates per warp.
        for (uint32_t r0 = 0; r0 < cnt; r0 += lead * G) {
            uint32_t gc = 0;
            while (gc < G && r0 + ci + lead * gc < cnt) ++gc;
            uint32_t nb = 0;
            if (gc) {
                uint32_t hv[kCandGroup], olds[kCandGroup];
#pragma unroll
                for (int j = 0; j < kCandGroup; ++j) {
                    if ((uint32_t) j >= gc) break;
                    hv[j] = __ldg(a.head + (size_t) cand[r0 + ci + lead * j] * kHeadWords + lane);
                }
                bool any_long = false;
#pragma unroll
                for (int j = 0; j < kCandGroup; ++j) {
                    if ((uint32_t) j >= gc) break;
                    const uint32_t dj = __shfl_sync(kFull, hv[j], 0);
                    if (part == 0) n_edges += 1 + dj;
                    any_long = any_long || dj > (uint32_t) kHeadNbrs;
                    bool valid = lane >= 1 && (uint32_t) lane <= min(dj, (uint32_t) kHeadNbrs) &&
                                 ((uint32_t) lane & (parts - 1)) == part;
                    if (valid && hv[j] >= a.n) {
                        atomicOr(a.error, ERR_BAD_ID);
                        valid = false;
                    }
                    if (!valid) hv[j] = kFull;
                    if (!in_smem) olds[j] = visit_issue(vis, hv[j], valid);
                }
#pragma unroll
                for (int j = 0; j < kCandGroup; ++j) {
                    if ((uint32_t) j >= gc) break;
                    const uint32_t id = hv[j];
                    const bool valid = id != kFull;
                    bool fresh;
                    if (in_smem) {
                        fresh = visit(id, valid);
                    } else {  // (all of them issued before any is used)
                        fresh = valid && !(olds[j] & (1u << (id & 31)));
                        note_dirty(my_dirty, dcap, dcount, valid && olds[j] == 0, id >> 5);
                    }
                    const uint32_t bm = __ballot_sync(kFull, fresh);
                    if (fresh) bi[nb + __popc(bm & lanemask_lt())] = id;
                    nb += __popc(bm);
                }
                if (any_long) {
                    for (uint32_t j = 0; j < gc; ++j) {
                        const uint32_t c = cand[r0 + ci + lead * j];
                        const uint32_t dj = __ldg(a.head + (size_t) c * kHeadWords);
                        if (dj <= (uint32_t) kHeadNbrs) continue;
                        const uint64_t off = __ldg(a.ovf_off + c);
                        for (uint32_t s0 = kHeadNbrs; s0 < dj; s0 += 32 * parts) {
                            const uint32_t s = s0 + part * 32 + lane;
                            bool valid = s < dj;
                            const uint32_t id = valid ? __ldg(a.ovf + off + (s - kHeadNbrs)) : 0u;
                            if (valid && id >= a.n) {
                                atomicOr(a.error, ERR_BAD_ID);
                                valid = false;
                            }
                            const bool fresh = visit(id, valid);
                            const uint32_t bm = __ballot_sync(kFull, fresh);
                            if (fresh) bi[nb + __popc(bm & lanemask_lt())] = id;
                            nb += __popc(bm);
                        }
                    }
                }
                __syncwarp();
            }
            finish_list(nb, true);
            const uint32_t n = close_list();
            // Every warp has its candidates: mark them (block_merge reads the
            // marks after its next barrier at the earliest).
            if (r0 == 0)
                for (uint32_t c = w + W * lane; c < cnt; c += W * 32) m.qi[cpos[c]] = cand[c] | kChecked;
            nk = min(nk, block_merge<W>(m, n, sz, L, a.orig));
        }
        k = nk <= last_k ? nk : last_k + 1;
    }

    if constexpr (STORE != STORE_FP32) {
        // Re-rank the final queue in exact float32 (reference lane order); the K
        // best by (distance, original id) go out.
        Dist<KIND, CL, STORE_FP32> E;
        E.load(a, q, lane);
        const uint32_t per = ((sz + W - 1) / W + 7) & ~7u;
        const uint32_t lo = min(sz, w * per), hi = min(sz, lo + per);
        E.distances(a, m.qi + lo, m.qd + lo, hi - lo, lane, tmp);
        __syncthreads();
        if (sz <= W * buf) {
            for (uint32_t i = tid; i < sz; i += T) {
                m.cD[i] = m.qd[i];
                m.cI[i] = m.qi[i] & kIdMask;
            }
            __syncthreads();
            const uint32_t *ids = m.sI;
            if (sz <= block_rank_max(W)) {
                block_rank<W, false>(m, sz, 0, a.orig);
            } else {
                block_bitonic<W>(m, sz, a.orig);
                ids = m.cI;
            }
            for (uint32_t i = tid; i < a.K; i += T)
                a.out_ids[(size_t) q * a.K + i] = i < sz ? __ldg(a.orig + ids[i]) : kFull;
        } else if (w == 0) {
            rerank_output(m.qd, m.qi, sz, a.K, a.orig, a.out_ids + (size_t) q * a.K, lane);
        }
    } else {
        for (uint32_t i = tid; i < a.K; i += T)
            a.out_ids[(size_t) q * a.K + i] = i < sz ? __ldg(a.orig + (m.qi[i] & kIdMask)) : kFull;
    }
    if (lane == 0) {
        atomicAdd(&ctl[BC_DIST], n_dist);
        atomicAdd(&ctl[BC_EDGES], n_edges);
        if (dcount > dcap) ctl[BC_FULL] = 1u;
    }
    __syncthreads();
    if (tid == 0 && a.out_stats) a.out_stats[q] = make_uint4(ctl[BC_DIST], n_expand, ctl[BC_EDGES], n_iter);
    // Clear the visited words this query set.
    if (in_smem) {
    } else if (!ctl[BC_FULL]) {
        for (uint32_t i = lane; i < dcount; i += 32) vis[my_dirty[i]] = 0u;
    } else {
        for (uint32_t i = tid; i < a.vis_words; i += T) vis[i] = 0u;
    }
    __syncthreads();
}

template <int KIND, int CL, int W, int STORE>
__global__ void __launch_bounds__(W * 32) search_block_kernel(SearchArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t slot = blockIdx.x;
    uint32_t *vis = a.visited + (size_t) slot * a.vis_words;
    uint32_t *dirty = a.dirty + (size_t) slot * a.dirty_cap;
    uint32_t *ctl = reinterpret_cast<uint32_t *>(smem + block_smem_bytes(a.queue_cap, W, a.block_buf, 0) - kBlockCtl * 4);
    for (;;) {
        if (threadIdx.x == 0) ctl[BC_Q] = atomicAdd(a.counter, 1u);
        __syncthreads();
        const uint32_t q = ctl[BC_Q];
        __syncthreads();
        if (q >= a.nq) break;
        block_search_one<KIND, CL, W, STORE>(a, q, smem, vis, dirty);
    }
}

}  // namespace panns
