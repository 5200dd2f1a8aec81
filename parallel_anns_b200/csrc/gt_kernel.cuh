// Float64 brute-force ground truth.
//
// The k results of any search are k distinct vertices, so the largest of their
// exact distances, tau, is an upper bound of the true k-th smallest distance.
// It is enough to collect the vertices whose float64 distance is <= tau (about
// k of them for a good search); an exact (distance, id) sort gives the top k.
// The collection is the tensor-core range screen (tc_screen.cu), whose lists
// gt_rank_kernel evaluates in float64 and ranks; one tiled float64 pass over the
// base collects instead (gt_collect_kernel) for a few queries, where the screen's
// fixed cost is more, and where its lists do not fit or do not hold (k > kGtMaxK, a
// bound so loose that refining it does not help, vectors past the screen's range).
// 10,000 queries x 1M x 96, k = 100: 174 ms in gt_collect_kernel, 3 ms in the
// screen, its operands and gt_rank_kernel.
// Distances are sum over dimensions, in order, of fma(t, t, acc) with
// t = (double) x - (double) q, in both kernels, so the search's own results
// meet their own bound bit for bit. Plays the role of
// tools/save_true_nearest_neighbors.cpp:16-35 (which scans in float32).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace panns {

constexpr int kGtQ = 64;    // queries per block tile
constexpr int kGtV = 128;   // vertices per block tile
constexpr int kGtK = 8;     // dimensions per shared-memory step

// tau[q] = max over the k ids of query q of its float64 distance, one chain over
// the dimensions a vertex. Bound by the gathers: rows in 16-byte loads (d is a
// multiple of 8), eight of a row's values in flight (10,000 x 100 rows of 96:
// 0.40 ms in 4-byte loads, 0.22 ms so).
__global__ void gt_tau_kernel(const float *__restrict__ base, int d, const float *__restrict__ queries,
                              uint32_t nq, const uint32_t *__restrict__ ids, uint32_t k,
                              double *__restrict__ tau) {
    const int lane = threadIdx.x & 31;
    const uint32_t q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= nq) return;
    const float *qr = queries + (size_t) q * d;
    double mx = 0.0;
    for (uint32_t i = lane; i < k; i += 32) {
        const float4 *x = reinterpret_cast<const float4 *>(base + (size_t) ids[(size_t) q * k + i] * d);
        const float4 *y = reinterpret_cast<const float4 *>(qr);
        double acc = 0.0;
        for (int j = 0; j < d / 4; j += 2) {
            const float4 a[2] = {__ldg(x + j), __ldg(x + j + 1)}, b[2] = {__ldg(y + j), __ldg(y + j + 1)};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float av[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, bv[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const double t = (double) av[e] - (double) bv[e];
                    acc = fma(t, t, acc);
                }
            }
        }
        mx = fmax(mx, acc);
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) tau[q] = mx;
}

// Grid: x = query tiles (fastest, so the tiles of one vertex range run
// together and share it through L2), y = vertex tiles v_tile0 + blockIdx.y
// (launched in slices of at most 65,535 tiles, the grid's y limit). 256 threads; thread
// (ty, tx) owns queries 4*ty..4*ty+3 and vertices tx + 16*j, j < 8.
__global__ void __launch_bounds__(256) gt_collect_kernel(const float *__restrict__ base, uint32_t n, int d,
                                                         const float *__restrict__ queries, uint32_t nq,
                                                         const double *__restrict__ tau, uint32_t cap,
                                                         uint32_t *__restrict__ cnt, double *__restrict__ cand_d,
                                                         uint32_t *__restrict__ cand_i, uint32_t v_tile0) {
    __shared__ double sq[kGtK][kGtQ];
    __shared__ double sv[kGtK][kGtV];
    const uint32_t q0 = blockIdx.x * kGtQ, v0 = (blockIdx.y + v_tile0) * kGtV;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    double acc[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0;
    for (int k0 = 0; k0 < d; k0 += kGtK) {
        for (int e = tid; e < kGtQ * kGtK; e += 256) {
            const int qq = e / kGtK, kk = e % kGtK;
            const uint32_t q = q0 + qq;
            sq[kk][qq] = (q < nq && k0 + kk < d) ? (double) queries[(size_t) q * d + k0 + kk] : 0.0;
        }
        for (int e = tid; e < kGtV * kGtK; e += 256) {
            const int vv = e / kGtK, kk = e % kGtK;
            const uint32_t v = v0 + vv;
            sv[kk][vv] = (v < n && k0 + kk < d) ? (double) base[(size_t) v * d + k0 + kk] : 0.0;
        }
        __syncthreads();
        const int kmax = min(kGtK, d - k0);
        for (int kk = 0; kk < kmax; ++kk) {
            double a[4], b[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = sq[kk][4 * ty + i];
#pragma unroll
            for (int j = 0; j < 8; ++j) b[j] = sv[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const double t = b[j] - a[i];
                    acc[i][j] = fma(t, t, acc[i][j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t q = q0 + 4 * ty + i;
        if (q >= nq) continue;
        const double tq = tau[q];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t v = v0 + tx + 16 * j;
            if (v < n && acc[i][j] <= tq) {
                const uint32_t pos = atomicAdd(cnt + q, 1u);
                if (pos < cap) {
                    cand_d[(size_t) q * cap + pos] = acc[i][j];
                    cand_i[(size_t) q * cap + pos] = v;
                }
            }
        }
    }
}

constexpr uint32_t kGtMaxK = 512;     // largest k of the screened path
constexpr uint32_t kGtList = 1024;    // vertices within the bound that gt_rank_kernel ranks

// out row i = row order[i] of `rows` (width d), and tau likewise.
__global__ void gt_gather_kernel(const float *__restrict__ rows, const double *__restrict__ tau,
                                 const uint32_t *__restrict__ order, uint32_t nq, uint32_t d, float *__restrict__ out,
                                 double *__restrict__ out_tau) {
    const uint32_t i = blockIdx.x;
    if (i >= nq) return;
    const size_t q = order[i];
    for (uint32_t j = threadIdx.x; j < d; j += blockDim.x) out[(size_t) i * d + j] = rows[q * d + j];
    if (threadIdx.x == 0) out_tau[i] = tau[q];
}

// tau[order[i]] = ts[i]: bounds back in query order.
__global__ void gt_scatter_tau_kernel(const double *__restrict__ ts, const uint32_t *__restrict__ order, uint32_t nq,
                                      double *__restrict__ tau) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nq) tau[order[i]] = ts[i];
}

// The vertices in layout order with every cell moved to a multiple of the
// screen's tile: perm[to[c] + i] = orig[from[c] + i]. One block per cell.
__global__ void gt_slots_kernel(const uint32_t *__restrict__ orig, const uint32_t *__restrict__ from,
                                const uint32_t *__restrict__ to, uint32_t *__restrict__ perm) {
    const uint32_t c = blockIdx.x, b = from[c], m = from[c + 1] - b;
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) perm[to[c] + i] = orig[b + i];
}

// One block of 128 threads per query i (row i of qs): the float64 distances of
// the screen's entries (splits lists of up to cap; entry y = position, vertex
// perm[position]), those within tau[i] ranked by (distance, vertex), the k best
// written to row order[i] of out_ids / out_dist. A query whose lists overflowed,
// or with more than kGtList vertices within tau, is not written: over[i] = 1,
// and tau[i] becomes the k-th smallest of the distances looked at, which is a
// bound of the answer too. d is a multiple of 4.
__global__ void __launch_bounds__(128) gt_rank_kernel(const float *__restrict__ base, int d,
                                                      const uint32_t *__restrict__ perm, const float *__restrict__ qs,
                                                      uint32_t nq, const uint32_t *__restrict__ order,
                                                      double *__restrict__ tau, uint32_t splits, uint32_t cap,
                                                      const uint2 *__restrict__ lists, const uint32_t *__restrict__ cnt,
                                                      uint32_t k, uint32_t *__restrict__ out_ids,
                                                      double *__restrict__ out_dist, uint32_t *__restrict__ over) {
    __shared__ double sd[kGtList];
    __shared__ uint32_t si[kGtList];
    __shared__ __align__(16) double sq[256];
    __shared__ uint32_t found;
    __shared__ double refined;
    const uint32_t i = blockIdx.x, tid = threadIdx.x;
    for (int e = tid; e < d; e += 128) sq[e] = (double) qs[(size_t) i * d + e];
    if (tid == 0) found = 0;
    __syncthreads();
    const double t0 = tau[i];
    bool full = false;
    for (uint32_t sp = 0; sp < splits; ++sp) {
        const uint32_t c = cnt[(size_t) sp * nq + i], m = min(c, cap);
        full = full || c > cap;
        const uint2 *list = lists + ((size_t) sp * nq + i) * cap;
        for (uint32_t e = tid; e < m; e += 128) {
            const uint32_t v = perm[list[e].y];
            const float4 *x = reinterpret_cast<const float4 *>(base + (size_t) v * d);
            double acc = 0.0;
#pragma unroll 4
            for (int j = 0; j < d / 4; ++j) {
                const float4 f = __ldg(x + j);
                double t = (double) f.x - sq[4 * j];
                acc = fma(t, t, acc);
                t = (double) f.y - sq[4 * j + 1];
                acc = fma(t, t, acc);
                t = (double) f.z - sq[4 * j + 2];
                acc = fma(t, t, acc);
                t = (double) f.w - sq[4 * j + 3];
                acc = fma(t, t, acc);
            }
            if (acc <= t0) {
                const uint32_t pos = atomicAdd(&found, 1u);
                if (pos < kGtList) {
                    sd[pos] = acc;
                    si[pos] = v;
                }
            }
        }
    }
    __syncthreads();
    const uint32_t n = min(found, kGtList);
    const bool bad = full || found > kGtList;
    if (tid == 0) {
        over[i] = bad ? 1u : n < k ? 2u : 0u;
        refined = t0;
    }
    __syncthreads();
    for (uint32_t e = tid; e < n; e += 128) {
        const double de = sd[e];
        const uint32_t ie = si[e];
        uint32_t rank = 0;
        for (uint32_t f = 0; f < n; ++f) rank += sd[f] < de || (sd[f] == de && si[f] < ie) ? 1u : 0u;
        if (bad) {
            if (rank + 1 == k) refined = de;
        } else if (rank < k) {
            out_ids[(size_t) order[i] * k + rank] = ie;
            if (out_dist) out_dist[(size_t) order[i] * k + rank] = de;
        }
    }
    __syncthreads();
    if (tid == 0 && bad) tau[i] = refined;
}

}  // namespace panns
