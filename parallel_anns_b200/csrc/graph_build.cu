// NSG-style graph construction on the GPU: exact k-NN lists, relative-
// neighbourhood (MRNG) pruning to R, medoid entry, reachability repair.
//
// Semantics (restated by po_build_nsg in oracle/panns_oracle.c):
//   * d64(x, y) = sum over j = 0..d-1, in order, of fma(t, t, acc) with
//     t = (double) x_j - (double) y_j (one float64 chain).
//   * knn(a) = the k vertices b != a with the smallest (d64(a, b), b).
//   * prune(a): walk knn(a) in order; b is kept unless some already kept c has
//     d64(c, b) < d64(a, b); at most R are kept (the NSG rule of
//     include/efanna2e/index_nsg.cpp:233-283 applied to exact k-NN lists).
//   * entry = the vertex with the smallest (d64(v, mean), v), mean = the float64
//     mean of the rows summed in id order.
//   * repair: from the entry, every vertex not reached (in id order) gets an
//     in-edge from the first reached vertex of its k-NN list (else the entry),
//     then everything it reaches is marked (index_nsg.cpp:638-718 plays this
//     part with a DFS tree).
// A screen finds each row's candidates, which are then ranked by d64. By default
// (n >= 1,024, d <= 256) it is the tcgen05 screen of tc_screen.cu, whose threshold
// provably holds all k nearest; the rows it reports (runs of equal distances longer
// than a list, clusters much smaller than the base, non-finite values) are screened
// here in float32 by squared differences. Else, or by name, all pairs are screened
// (||y||^2 - 2 x.y) in float32 on CUDA cores (tiled here, C = k + 8 candidates kept
// per row) or with TF32 tensor-core GEMMs (cuBLAS) folded tile by tile into the
// rows' lists (C = k + 32); these two equal the exact k-NN unless their rounding
// moves a true neighbour past 8 or 32 others.
#include <cublas_v2.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "../../include/panns_build.h"
#include "dev_scratch.h"
#include "graph_types.h"
#include "learned.h"
#include "tc_screen.h"

namespace panns {
namespace {

#define GCU(call)                                                                          \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess)                                                             \
            return set_error(PANNS_ECUDA, std::string(#call ": ") + cudaGetErrorString(e_)); \
    } while (0)

template <typename T>
using Buf = Scratch<T>;

constexpr int kBQ = 64;    // rows (queries) per block
constexpr int kBV = 128;   // candidate rows per tile
constexpr int kBK = 16;    // dimensions per shared-memory step
constexpr int kMaxC = 136; // screen list length (k + 8 <= 136)
constexpr uint32_t kTcMinRows = 1024;  // below, the float32 screen's single launch is as fast
constexpr uint32_t kMaxVecD = 256;  // rerank_kernel's shared-memory copy of a row

__global__ void sqnorm32_kernel(const float *__restrict__ x, uint32_t n, uint32_t d, float *__restrict__ out) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    float s = 0.f;
    for (uint32_t j = 0; j < d; ++j) s = fmaf(x[(size_t) r * d + j], x[(size_t) r * d + j], s);
    out[r] = s;
}

// Insert this warp's 32 candidates (dv, iv) (one per lane; +inf = none) into
// the sorted list (rd, ri)[0..c) of capacity C, by (distance, id): each one
// that beats the C-th in turn goes to its rank, the list shifting up by one.
__device__ __forceinline__ void list_insert(float *rd, uint32_t *ri, uint32_t &c, uint32_t C, float dv, uint32_t iv,
                                            int lane) {
    const float thr_d = c == C ? rd[C - 1] : __int_as_float(0x7f800000);
    const uint32_t thr_i = c == C ? ri[C - 1] : 0xffffffffu;
    bool want = dv < thr_d || (dv == thr_d && iv < thr_i);
    want = want && !(dv == __int_as_float(0x7f800000));
    uint32_t bm = __ballot_sync(0xffffffffu, want);
    while (bm) {
        const int src = __ffs(bm) - 1;
        bm &= bm - 1;
        const float sd = __shfl_sync(0xffffffffu, dv, src);
        const uint32_t si = __shfl_sync(0xffffffffu, iv, src);
        // still better than the C-th after earlier inserts?
        if (c == C && !(sd < rd[C - 1] || (sd == rd[C - 1] && si < ri[C - 1]))) continue;
        // position = number of entries smaller than (sd, si)
        uint32_t pos = 0;
        for (uint32_t e0 = 0; e0 < c; e0 += 32) {
            const uint32_t e = e0 + lane;
            const bool less = e < c && (rd[e] < sd || (rd[e] == sd && ri[e] < si));
            pos += __popc(__ballot_sync(0xffffffffu, less));
        }
        const uint32_t end = c < C ? c : C - 1;  // last index that moves
        // shift [pos, end) up by one, from the top down in chunks of 32
        for (int e0 = (int) end - 1; e0 >= (int) pos; e0 -= 32) {
            const int e = e0 - lane;
            float td = 0.f;
            uint32_t ti = 0;
            const bool mv = e >= (int) pos;
            if (mv) {
                td = rd[e];
                ti = ri[e];
            }
            __syncwarp();
            if (mv) {
                rd[e + 1] = td;
                ri[e + 1] = ti;
            }
            __syncwarp();
        }
        if (lane == 0) {
            rd[pos] = sd;
            ri[pos] = si;
        }
        __syncwarp();
        if (c < C) ++c;
    }
}

// Tensor-core screen, second half: G (nr x nc, row-major) holds -2 x_r . y_c
// for rows r0.. and candidates c0..; one warp per row merges ||y_c||^2 + G
// into the row's list (global ld / li / cnt, staged in shared memory).
__global__ void __launch_bounds__(256) topk_tile_kernel(const float *__restrict__ G, uint32_t nr, uint32_t nc,
                                                        uint32_t r0, uint32_t c0, const float *__restrict__ yn,
                                                        uint32_t n, uint32_t C, float *__restrict__ gld,
                                                        uint32_t *__restrict__ gli, uint32_t *__restrict__ gcnt) {
    __shared__ float sd[8][kMaxC];
    __shared__ uint32_t si[8][kMaxC];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t rr = blockIdx.x * 8 + w;
    if (rr >= nr) return;
    const uint32_t row = r0 + rr;
    uint32_t c = gcnt[row];
    for (uint32_t e = lane; e < c; e += 32) {
        sd[w][e] = gld[(size_t) row * C + e];
        si[w][e] = gli[(size_t) row * C + e];
    }
    __syncwarp();
    const float *g = G + (size_t) rr * nc;
    for (uint32_t j0 = 0; j0 < nc; j0 += 32) {
        const uint32_t j = j0 + lane, col = c0 + j;
        const bool ok = j < nc && col < n && col != row;
        const float dv = ok ? g[j] + yn[col] : __int_as_float(0x7f800000);
        list_insert(sd[w], si[w], c, C, dv, col, lane);
    }
    for (uint32_t e = lane; e < c; e += 32) {
        gld[(size_t) row * C + e] = sd[w][e];
        gli[(size_t) row * C + e] = si[w][e];
    }
    if (lane == 0) gcnt[row] = c;
}

// Float32 screen: for each of the kBQ rows of this block (rows q0.. of the
// base, or of the list `rows` of nr ids), the C candidates (all rows but
// itself) with the smallest (||y||^2 - 2 x.y, id), over tiles of kBV
// candidates. 256 threads: thread (ty, tx) computes a 4 x 8 block of the
// 64 x 128 tile; then warp w inserts the tile into the lists of rows 8w..8w+7.
//
// DIRECT: by the squared distance as a sum of squared differences, for the rows the
// tensor-core screen hands on. It takes two instructions a term instead of one, but
// its error follows the distance itself, wherever the origin and however far other
// rows are, which those rows (runs of equal distances, clusters much smaller than
// the base) depend on. Distances that overflow, or of a row with a NaN, count as
// equal, so that a list is filled (by id) all the same.
template <bool DIRECT>
__global__ void __launch_bounds__(256) screen_kernel(const float *__restrict__ x, uint32_t n, uint32_t d,
                                                     const float *__restrict__ xn, uint32_t C,
                                                     const uint32_t *__restrict__ rows, uint32_t nr,
                                                     uint32_t *__restrict__ out_ids) {
    extern __shared__ __align__(16) uint8_t sm[];
    float *Qs = reinterpret_cast<float *>(sm);                 // [kBK][kBQ]
    float *Vs = Qs + kBK * kBQ;                                // [kBK][kBV]
    float *D = Vs + kBK * kBV;                                 // [kBQ][kBV + 1]
    float *ld = D + kBQ * (kBV + 1);                           // [kBQ][C]
    uint32_t *li = reinterpret_cast<uint32_t *>(ld + kBQ * C); // [kBQ][C]
    uint32_t *cnt = li + kBQ * C;                              // [kBQ]
    uint32_t *qid = cnt + kBQ;                                 // [kBQ] row ids (~0: none)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t q0 = blockIdx.x * kBQ;
    for (int i = tid; i < kBQ; i += 256) {
        cnt[i] = 0;
        qid[i] = q0 + i < nr ? (rows ? rows[q0 + i] : q0 + i) : 0xffffffffu;
    }
    const int ty = tid / 16, tx = tid % 16;  // rows ty*4.., cols tx*8..
    __syncthreads();
    for (uint32_t v0 = 0; v0 < n; v0 += kBV) {
        float acc[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
        for (uint32_t k0 = 0; k0 < d; k0 += kBK) {
            for (int t = tid; t < kBK * kBQ; t += 256) {
                const int kk = t % kBK, qq = t / kBK;
                const uint32_t gq = qid[qq], gk = k0 + kk;
                Qs[kk * kBQ + qq] = (gq < n && gk < d) ? x[(size_t) gq * d + gk] : 0.f;
            }
            for (int t = tid; t < kBK * kBV; t += 256) {
                const int kk = t % kBK, vv = t / kBK;
                const uint32_t gv = v0 + vv, gk = k0 + kk;
                Vs[kk * kBV + vv] = (gv < n && gk < d) ? x[(size_t) gv * d + gk] : 0.f;
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < kBK; ++kk) {
                const float4 a4 = *reinterpret_cast<const float4 *>(Qs + kk * kBQ + ty * 4);
                const float4 b4 = *reinterpret_cast<const float4 *>(Vs + kk * kBV + tx * 8);
                const float4 b5 = *reinterpret_cast<const float4 *>(Vs + kk * kBV + tx * 8 + 4);
                const float a[4] = {a4.x, a4.y, a4.z, a4.w};
                const float b[8] = {b4.x, b4.y, b4.z, b4.w, b5.x, b5.y, b5.z, b5.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float t = DIRECT ? a[i] - b[j] : 0.f;
                        acc[i][j] = DIRECT ? fmaf(t, t, acc[i][j]) : fmaf(a[i], b[j], acc[i][j]);
                    }
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t gq = qid[ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t gv = v0 + tx * 8 + j;
                const bool ok = gv < n && gv != gq;
                const float v = DIRECT ? fminf(acc[i][j], 3.4e38f) : ok ? fmaf(-2.f, acc[i][j], xn[gv]) : 0.f;
                D[(ty * 4 + i) * (kBV + 1) + tx * 8 + j] = ok ? v : __int_as_float(0x7f800000);
            }
        }
        __syncthreads();
        // Insert: rows 8w..8w+7 of this warp, each candidate that beats the
        // row's current C-th (distance, id).
        for (int r = warp * 8; r < warp * 8 + 8; ++r) {
            uint32_t c = cnt[r];
            for (int j0 = 0; j0 < kBV; j0 += 32)
                list_insert(ld + r * C, li + r * C, c, C, D[r * (kBV + 1) + j0 + lane], v0 + j0 + lane, lane);
            if (lane == 0) cnt[r] = c;
            __syncwarp();
        }
        __syncthreads();
    }
    for (int r = warp; r < kBQ; r += 8) {
        const uint32_t gq = qid[r];
        if (gq >= n) continue;
        for (uint32_t e = lane; e < C; e += 32)
            out_ids[(size_t) gq * C + e] = e < cnt[r] ? li[r * C + e] : 0xffffffffu;
    }
}

// Float32 screen restricted to cells: block b screens up to kBQ rows of cell
// blk_cell[b], rows[blk_row0[b]] .. rows[blk_row0[b + 1]), against the members
// of the cell itself and of its P nearest cells (near[c * P ..]), keeping per
// row the C candidates with the smallest (||y||^2 - 2 x.y, id). The same
// tiling and list insertion as screen_kernel; candidates are read through the
// members list (cell by cell, ids ascending within a cell). DIRECT as there.
template <bool DIRECT>
__global__ void __launch_bounds__(256) screen_cells_kernel(
    const float *__restrict__ x, uint32_t n, uint32_t d, const float *__restrict__ xn, uint32_t C,
    const uint32_t *__restrict__ members, const uint32_t *__restrict__ cstart, const uint32_t *__restrict__ near,
    uint32_t P, const uint32_t *__restrict__ rows, const uint32_t *__restrict__ blk_cell,
    const uint32_t *__restrict__ blk_row0, uint32_t *__restrict__ out_ids) {
    extern __shared__ __align__(16) uint8_t sm[];
    float *Qs = reinterpret_cast<float *>(sm);                 // [kBK][kBQ]
    float *Vs = Qs + kBK * kBQ;                                // [kBK][kBV]
    float *D = Vs + kBK * kBV;                                 // [kBQ][kBV + 1]
    float *ld = D + kBQ * (kBV + 1);                           // [kBQ][C]
    uint32_t *li = reinterpret_cast<uint32_t *>(ld + kBQ * C); // [kBQ][C]
    uint32_t *cnt = li + kBQ * C;                              // [kBQ]
    uint32_t *qid = cnt + kBQ;                                 // [kBQ] row ids (~0: none)
    uint32_t *vid = qid + kBQ;                                 // [kBV] candidate ids of the tile (~0: none)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t cell = blk_cell[blockIdx.x];
    const uint32_t p0 = blk_row0[blockIdx.x], pend = blk_row0[blockIdx.x + 1];
    for (int i = tid; i < kBQ; i += 256) {
        cnt[i] = 0;
        qid[i] = p0 + i < pend ? rows[p0 + i] : 0xffffffffu;
    }
    const int ty = tid / 16, tx = tid % 16;  // rows ty*4.., cols tx*8..
    __syncthreads();
    for (uint32_t sgi = 0; sgi <= P; ++sgi) {
        const uint32_t sc = sgi == 0 ? cell : near[(size_t) cell * P + sgi - 1];
        if (sc == 0xffffffffu) continue;
        const uint32_t s0 = cstart[sc], s1 = cstart[sc + 1];
        for (uint32_t v0 = s0; v0 < s1; v0 += kBV) {
            for (int i = tid; i < kBV; i += 256) vid[i] = v0 + i < s1 ? members[v0 + i] : 0xffffffffu;
            __syncthreads();
            float acc[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
            for (uint32_t k0 = 0; k0 < d; k0 += kBK) {
                for (int t = tid; t < kBK * kBQ; t += 256) {
                    const int kk = t % kBK, qq = t / kBK;
                    const uint32_t gq = qid[qq], gk = k0 + kk;
                    Qs[kk * kBQ + qq] = (gq < n && gk < d) ? x[(size_t) gq * d + gk] : 0.f;
                }
                for (int t = tid; t < kBK * kBV; t += 256) {
                    const int kk = t % kBK, vv = t / kBK;
                    const uint32_t gv = vid[vv], gk = k0 + kk;
                    Vs[kk * kBV + vv] = (gv < n && gk < d) ? x[(size_t) gv * d + gk] : 0.f;
                }
                __syncthreads();
#pragma unroll
                for (int kk = 0; kk < kBK; ++kk) {
                    const float4 a4 = *reinterpret_cast<const float4 *>(Qs + kk * kBQ + ty * 4);
                    const float4 b4 = *reinterpret_cast<const float4 *>(Vs + kk * kBV + tx * 8);
                    const float4 b5 = *reinterpret_cast<const float4 *>(Vs + kk * kBV + tx * 8 + 4);
                    const float a[4] = {a4.x, a4.y, a4.z, a4.w};
                    const float b[8] = {b4.x, b4.y, b4.z, b4.w, b5.x, b5.y, b5.z, b5.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                        const float t = DIRECT ? a[i] - b[j] : 0.f;
                        acc[i][j] = DIRECT ? fmaf(t, t, acc[i][j]) : fmaf(a[i], b[j], acc[i][j]);
                    }
                }
                __syncthreads();
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t gq = qid[ty * 4 + i];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t gv = vid[tx * 8 + j];
                    const bool ok = gv < n && gv != gq;
                    const float v = DIRECT ? fminf(acc[i][j], 3.4e38f) : ok ? fmaf(-2.f, acc[i][j], xn[gv]) : 0.f;
                    D[(ty * 4 + i) * (kBV + 1) + tx * 8 + j] = ok ? v : __int_as_float(0x7f800000);
                }
            }
            __syncthreads();
            for (int r = warp * 8; r < warp * 8 + 8; ++r) {
                uint32_t c = cnt[r];
                for (int j0 = 0; j0 < kBV; j0 += 32)
                    list_insert(ld + r * C, li + r * C, c, C, D[r * (kBV + 1) + j0 + lane], vid[j0 + lane], lane);
                if (lane == 0) cnt[r] = c;
                __syncwarp();
            }
            __syncthreads();
        }
    }
    for (int r = warp; r < kBQ; r += 8) {
        const uint32_t gq = qid[r];
        if (gq >= n) continue;
        for (uint32_t e = lane; e < C; e += 32)
            out_ids[(size_t) gq * C + e] = e < cnt[r] ? li[r * C + e] : 0xffffffffu;
    }
}

// The cells' rows, each cell from the start of its first tile (the rest of the
// order is filled beforehand).
__global__ void __launch_bounds__(256) pad_cells_kernel(const uint32_t *__restrict__ members,
                                                        const uint32_t *__restrict__ start,
                                                        const uint32_t *__restrict__ tile0,
                                                        uint32_t *__restrict__ order) {
    const uint32_t c = blockIdx.x, b = start[c], m = start[c + 1] - b;
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) order[(size_t) tile0[c] * kTcM + i] = members[b + i];
}

// For every cell c (one block each), the P other cells whose centroids are
// nearest by (float64 squared distance, index); ~0 where there are fewer.
__global__ void __launch_bounds__(256) near_cells_kernel(const float *__restrict__ cent, uint32_t cells, uint32_t d,
                                                         uint32_t P, uint32_t *__restrict__ near) {
    constexpr int kMaxP = 8;
    __shared__ double bd[256 * kMaxP];
    __shared__ uint32_t bi[256 * kMaxP];
    const uint32_t c = blockIdx.x;
    double md[kMaxP];
    uint32_t mi[kMaxP];
    for (int t = 0; t < kMaxP; ++t) {
        md[t] = __longlong_as_double(0x7ff0000000000000ll);
        mi[t] = 0xffffffffu;
    }
    for (uint32_t j = threadIdx.x; j < cells; j += blockDim.x) {
        if (j == c) continue;
        double acc = 0.0;
        for (uint32_t e = 0; e < d; ++e) {
            const double t = (double) cent[(size_t) c * d + e] - (double) cent[(size_t) j * d + e];
            acc = fma(t, t, acc);
        }
        // insert (acc, j) into this thread's sorted best P
        if (acc < md[P - 1] || (acc == md[P - 1] && j < mi[P - 1])) {
            int pos = (int) P - 1;
            while (pos > 0 && (acc < md[pos - 1] || (acc == md[pos - 1] && j < mi[pos - 1]))) {
                md[pos] = md[pos - 1];
                mi[pos] = mi[pos - 1];
                --pos;
            }
            md[pos] = acc;
            mi[pos] = j;
        }
    }
    for (uint32_t t = 0; t < P; ++t) {
        bd[threadIdx.x * P + t] = md[t];
        bi[threadIdx.x * P + t] = mi[t];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t tot = blockDim.x * P;
        for (uint32_t t = 0; t < P; ++t) {  // P smallest of the block's lists
            uint32_t best = 0;
            for (uint32_t e = 1; e < tot; ++e)
                if (bd[e] < bd[best] || (bd[e] == bd[best] && bi[e] < bi[best])) best = e;
            near[(size_t) c * P + t] = bi[best];
            bd[best] = __longlong_as_double(0x7ff0000000000000ll);
            bi[best] = 0xffffffffu;
        }
    }
}

// Rows idx[0..m) of x gathered into out (m x d).
__global__ void gather_rows_f32_kernel(const float *__restrict__ x, uint32_t d, const uint32_t *__restrict__ idx,
                                       uint32_t m, float *__restrict__ out) {
    const size_t total = (size_t) m * d;
    for (size_t t = blockIdx.x * (size_t) blockDim.x + threadIdx.x; t < total; t += (size_t) gridDim.x * blockDim.x)
        out[t] = x[(size_t) idx[t / d] * d + t % d];
}

__device__ __forceinline__ double d64(const float *__restrict__ a, const float *__restrict__ b, uint32_t d) {
    double acc = 0.0;
    for (uint32_t j = 0; j < d; ++j) {
        const double t = (double) a[j] - (double) b[j];
        acc = fma(t, t, acc);
    }
    return acc;
}

// One warp per row a0 + r (r < na): float64 distances of its screened
// candidates (C slots, ~0 = none), ranked by (d64, id); the k best go out (ids
// and distances, row r of the chunk's knn / knn_d; a list short of k valid
// candidates ends in invalid ids, which the caller pre-sets). Bound by the
// float32 -> float64 conversions and the gathers of the candidates' rows: with
// d a multiple of 4 each lane streams its candidate's row in 16-byte loads
// against the row's float64 copy in shared memory (VEC), else by elements.
// 250,000 x 96: 8.8 ms with 4-byte loads over k + 32 slots, 3.0 ms so.
template <bool VEC>
__global__ void __launch_bounds__(256) rerank_kernel(const float *__restrict__ x, uint32_t n, uint32_t d,
                                                     const uint32_t *__restrict__ cand, uint32_t C, uint32_t k,
                                                     uint32_t a0, uint32_t na, uint32_t *__restrict__ knn,
                                                     double *__restrict__ knn_d) {
    __shared__ double sd[8][kMaxC];
    __shared__ uint32_t si[8][kMaxC];
    __shared__ __align__(16) double sx[VEC ? 8 : 1][VEC ? kMaxVecD : 2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t r = blockIdx.x * 8 + w;
    if (r >= na) return;
    const uint32_t a = a0 + r;
    const float *xa = x + (size_t) a * d;
    if (VEC)
        for (uint32_t e = lane; e < d; e += 32) sx[w][e] = (double) xa[e];
    uint32_t m = 0;  // valid candidates
    for (uint32_t e0 = 0; e0 < C; e0 += 32) {
        const uint32_t b = e0 + lane < C ? cand[(size_t) a * C + e0 + lane] : 0xffffffffu;
        const uint32_t bm = __ballot_sync(0xffffffffu, b < n);
        if (b < n) si[w][m + __popc(bm & ((1u << lane) - 1u))] = b;
        m += __popc(bm);
    }
    __syncwarp();
    for (uint32_t e = lane; e < m; e += 32) {
        const float *xb = x + (size_t) si[w][e] * d;
        double acc = 0.0;
        if (VEC) {
            const float4 *x4 = reinterpret_cast<const float4 *>(xb);
#pragma unroll 4
            for (uint32_t j = 0; j < d / 4; ++j) {
                const float4 v = __ldg(x4 + j);
                const double2 p = *reinterpret_cast<const double2 *>(&sx[w][4 * j]);
                const double2 q = *reinterpret_cast<const double2 *>(&sx[w][4 * j + 2]);
                double t = p.x - (double) v.x;
                acc = fma(t, t, acc);
                t = p.y - (double) v.y;
                acc = fma(t, t, acc);
                t = q.x - (double) v.z;
                acc = fma(t, t, acc);
                t = q.y - (double) v.w;
                acc = fma(t, t, acc);
            }
        } else {
            acc = d64(xa, xb, d);
        }
        sd[w][e] = acc;
    }
    __syncwarp();
    for (uint32_t e = lane; e < m; e += 32) {
        const double de = sd[w][e];
        const uint32_t ie = si[w][e];
        uint32_t rank = 0;
        for (uint32_t f = 0; f < m; ++f) {
            const double df = sd[w][f];
            const uint32_t jf = si[w][f];
            rank += (df < de || (df == de && jf < ie)) ? 1u : 0u;
        }
        if (rank < k) {
            knn[(size_t) r * k + rank] = ie;
            knn_d[(size_t) r * k + rank] = de;
        }
    }
}

// One warp per row a0 + r (r < na): MRNG pruning of its k-NN list (row r of
// the chunk's knn / knn_d) to at most R (row r of out, deg), reading the
// candidates' rows from global memory (any d; see prune_rows_kernel).
__global__ void prune_kernel(const float *__restrict__ x, uint32_t n, uint32_t d, const uint32_t *__restrict__ knn,
                             const double *__restrict__ knn_d, uint32_t k, uint32_t R, uint32_t na,
                             uint32_t *__restrict__ out, uint32_t *__restrict__ deg) {
    extern __shared__ uint32_t kept_all[];  // [8][R]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t r = blockIdx.x * 8 + w;
    if (r >= na) return;
    uint32_t *kept = kept_all + w * R;
    uint32_t nk = 0;
    for (uint32_t i = 0; i < k && nk < R; ++i) {
        const uint32_t b = knn[(size_t) r * k + i];
        if (b >= n) break;
        const double dab = knn_d[(size_t) r * k + i];
        const float *xb = x + (size_t) b * d;
        bool occl = false;
        for (uint32_t c0 = 0; c0 < nk && !occl; c0 += 32) {
            const uint32_t c = c0 + lane;
            const bool o = c < nk && d64(x + (size_t) kept[c] * d, xb, d) < dab;
            occl = __any_sync(0xffffffffu, o);
        }
        if (!occl) {
            if (lane == 0) kept[nk] = b;
            __syncwarp();
            ++nk;
        }
    }
    for (uint32_t e = lane; e < nk; e += 32) out[(size_t) r * R + e] = kept[e];
    if (lane == 0) deg[r] = nk;
}

// The same prune with the candidates' rows in shared memory (d a multiple of
// 4). The walk is turned round: when a candidate c is kept, the warp tests it
// against all later candidates that are not occluded yet (one per lane), so a
// row takes as many dependent steps as it keeps neighbours (about 18 of 64)
// and not one per candidate and 32 kept. d(c, b) < d(a, b) is decided in
// float32 where the two differ by more than float32 can be off (the squared
// differences are all positive, so the sum's relative error is at most
// (d + 3) 2^-24; kPruneSlack is over twice that), else by the float64 chain.
// Rows are (d / 4 rounded up to odd) 16-byte words apart, so that eight lanes
// reading eight rows hit distinct banks. Bound by the shared-memory reads.
// 250,000 x 96, k = 64: 61 ms with one candidate at a time in float64 from
// global memory, 6.4 ms so.
__host__ __device__ inline uint32_t prune_row_words(uint32_t d) { return (d / 4) | 1u; }
__host__ __device__ inline uint32_t prune_warp_bytes(uint32_t d, uint32_t k) {
    return k * prune_row_words(d) * 16 + ((k * 16 + 15) & ~15u);  // rows; distances, ids, list
}

__global__ void __launch_bounds__(128) prune_rows_kernel(const float *__restrict__ x, uint32_t n, uint32_t d,
                                                         const uint32_t *__restrict__ knn,
                                                         const double *__restrict__ knn_d, uint32_t k, uint32_t R,
                                                         uint32_t na, uint32_t *__restrict__ out,
                                                         uint32_t *__restrict__ deg) {
    extern __shared__ __align__(16) uint8_t prune_sm[];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t r = blockIdx.x * (blockDim.x >> 5) + w;
    if (r >= na) return;
    const uint32_t d4 = d / 4, words = prune_row_words(d);
    float4 *rows = reinterpret_cast<float4 *>(prune_sm + (size_t) w * prune_warp_bytes(d, k));
    double *dab = reinterpret_cast<double *>(rows + (size_t) k * words);
    uint32_t *ids = reinterpret_cast<uint32_t *>(dab + k);
    uint32_t *al = ids + k;
    // The list up to its first invalid id.
    uint32_t kv = k;
    for (uint32_t i0 = 0; i0 < k; i0 += 32) {
        const uint32_t i = i0 + lane;
        const uint32_t b = i < k ? knn[(size_t) r * k + i] : 0u;
        if (i < k) {
            ids[i] = b;
            dab[i] = knn_d[(size_t) r * k + i];
            al[i] = i;
        }
        const uint32_t bad = __ballot_sync(0xffffffffu, i < k && b >= n);
        if (bad) {
            kv = i0 + __ffs(bad) - 1;
            break;
        }
    }
    __syncwarp();
    for (uint32_t e = lane; e < kv * d4; e += 32) {
        const uint32_t i = e / d4, c = e - i * d4;
        const uint32_t dst = (uint32_t) __cvta_generic_to_shared(rows + (size_t) i * words + c);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                     "l"(reinterpret_cast<const float4 *>(x + (size_t) ids[i] * d) + c)
                     : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    const float slack = (float) (d + 8) * 1.2e-7f;
    uint32_t nk = 0, alive = kv;
    while (alive && nk < R) {
        const uint32_t ci = al[0];
        if (lane == 0) out[(size_t) r * R + nk] = ids[ci];
        ++nk;
        const float4 *rc = rows + (size_t) ci * words;
        uint32_t left = 0;
        for (uint32_t t0 = 1; t0 < alive; t0 += 32) {
            const uint32_t t = t0 + lane;
            const bool have = t < alive;
            const uint32_t j = have ? al[t] : ci;
            const float4 *rj = rows + (size_t) j * words;
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 4
            for (uint32_t q = 0; q < d4; ++q) {
                const float4 u = rc[q], v = rj[q];
                float y = u.x - v.x;
                s0 = fmaf(y, y, s0);
                y = u.y - v.y;
                s1 = fmaf(y, y, s1);
                y = u.z - v.z;
                s2 = fmaf(y, y, s2);
                y = u.w - v.w;
                s3 = fmaf(y, y, s3);
            }
            const float f = (s0 + s1) + (s2 + s3);
            bool keep = false;
            if (have) {
                const double dj = dab[j];
                if (f > 1e-30f && f < 1e37f && (double) f * (1.0 - (double) slack) > dj) {
                    keep = true;
                } else if (f > 1e-30f && f < 1e37f && (double) f * (1.0 + (double) slack) < dj) {
                    keep = false;
                } else {
                    keep = !(d64(reinterpret_cast<const float *>(rc), reinterpret_cast<const float *>(rj), d) < dj);
                }
            }
            const uint32_t bm = __ballot_sync(0xffffffffu, keep);
            if (keep) al[left + __popc(bm & ((1u << lane) - 1u))] = j;
            left += __popc(bm);
            __syncwarp();
        }
        alive = left;
    }
    if (lane == 0) deg[r] = nk;
}

// d64 of every row to one float64 point (the mean).
__global__ void dist_to_point_kernel(const float *__restrict__ x, uint32_t n, uint32_t d,
                                     const double *__restrict__ p, double *__restrict__ out) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    double acc = 0.0;
    for (uint32_t j = 0; j < d; ++j) {
        const double t = (double) x[(size_t) r * d + j] - p[j];
        acc = fma(t, t, acc);
    }
    out[r] = acc;
}

// The float64 mean of the rows, every dimension summed in row order (the order
// that fixes its last bits): one thread per dimension, a chain of n additions
// fed 64 rows ahead. The addition's latency bounds it (250,000 rows: 2 ms), so
// it runs beside the screen on a stream of its own; the same sum on the host
// took 10 ms.
__global__ void __launch_bounds__(32) mean_kernel(const float *__restrict__ x, uint32_t n, uint32_t d,
                                                  double *__restrict__ mean) {
    constexpr int U = 64;
    const uint32_t j = blockIdx.x * 32 + threadIdx.x;
    if (j >= d) return;
    const float *c = x + j;
    double s = 0.0;
    float cur[U];
    uint32_t r = 0;
    if (n >= U) {
#pragma unroll
        for (int u = 0; u < U; ++u) cur[u] = __ldg(c + (size_t) u * d);
        for (; r + 2 * U <= n; r += U) {
            float nxt[U];
#pragma unroll
            for (int u = 0; u < U; ++u) nxt[u] = __ldg(c + (size_t) (r + U + u) * d);
#pragma unroll
            for (int u = 0; u < U; ++u) s += (double) cur[u];
#pragma unroll
            for (int u = 0; u < U; ++u) cur[u] = nxt[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) s += (double) cur[u];
        r += U;
    }
    for (; r < n; ++r) s += (double) __ldg(c + (size_t) r * d);
    mean[j] = s / (double) n;
}

// The lowest index of the smallest value (one block); 0 if value 0 is a NaN.
__global__ void __launch_bounds__(1024) argmin64_kernel(const double *__restrict__ v, uint32_t n,
                                                        uint32_t *__restrict__ out) {
    __shared__ double bv[32];
    __shared__ uint32_t bi[32];
    double best = __longlong_as_double(0x7ff0000000000000ll);
    uint32_t at = 0xffffffffu;
    for (uint32_t i = threadIdx.x; i < n; i += 1024) {
        const double t = v[i];
        if (t < best || (t == best && i < at)) {
            best = t;
            at = i;
        }
    }
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int round = 0; round < 2; ++round) {
        for (int o = 16; o > 0; o >>= 1) {
            const double v2 = __shfl_xor_sync(0xffffffffu, best, o);
            const uint32_t i2 = __shfl_xor_sync(0xffffffffu, at, o);
            if (v2 < best || (v2 == best && i2 < at)) {
                best = v2;
                at = i2;
            }
        }
        if (round == 1) break;
        if (lane == 0) {
            bv[w] = best;
            bi[w] = at;
        }
        __syncthreads();
        if (w) return;
        best = bv[lane];
        at = bi[lane];
    }
    if (lane == 0) *out = v[0] != v[0] || at >= n ? 0u : at;
}

// Exclusive prefix sums of n words into out[0..n] (64 bits; out[n] = the
// total): sums of 4,096-word blocks, one block that scans those, the blocks again.
constexpr uint32_t kScanBlock = 4096;

__device__ __forceinline__ uint64_t block_scan_1024(uint64_t v, uint64_t *red, uint64_t &total) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int) lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) red[w] = incl;
    __syncthreads();
    uint64_t before = 0;
    total = 0;
    for (uint32_t i = 0; i < 32; ++i) {
        if (i < w) before += red[i];
        total += red[i];
    }
    return before + incl - v;
}

__global__ void __launch_bounds__(1024) scan_sums_kernel(const uint32_t *__restrict__ in, uint32_t n,
                                                         uint64_t *__restrict__ sums) {
    __shared__ uint64_t red[32];
    uint64_t v = 0;
    for (uint32_t e = 0; e < 4; ++e) {
        const uint64_t i = (uint64_t) blockIdx.x * kScanBlock + threadIdx.x * 4 + e;
        v += i < n ? in[i] : 0u;
    }
    uint64_t total;
    block_scan_1024(v, red, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) scan_blocks_kernel(uint64_t *__restrict__ sums, uint32_t m) {
    __shared__ uint64_t red[32];
    uint64_t base = 0;
    for (uint32_t b0 = 0; b0 < m; b0 += 1024) {
        const uint32_t b = b0 + threadIdx.x;
        const uint64_t v = b < m ? sums[b] : 0;
        uint64_t total;
        const uint64_t ex = block_scan_1024(v, red, total);
        if (b < m) sums[b] = base + ex;
        base += total;
    }
}

__global__ void __launch_bounds__(1024) scan_write_kernel(const uint32_t *__restrict__ in, uint32_t n,
                                                          const uint64_t *__restrict__ sums,
                                                          uint64_t *__restrict__ out) {
    __shared__ uint64_t red[32];
    const uint64_t i0 = (uint64_t) blockIdx.x * kScanBlock + threadIdx.x * 4;
    uint32_t x[4];
    uint64_t v = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        x[e] = i0 + e < n ? in[i0 + e] : 0u;
        v += x[e];
    }
    uint64_t total;
    uint64_t at = sums[blockIdx.x] + block_scan_1024(v, red, total);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (i0 + e <= n) out[i0 + e] = at;
        at += x[e];
    }
}

cudaError_t scan_words(const uint32_t *in, uint32_t n, uint64_t *out, cudaStream_t s) {
    // One block more than the words need, so that out[n] is always written.
    const uint32_t m = n / kScanBlock + 1;
    Scratch<uint64_t> sums;
    cudaError_t e = sums.alloc(m, s);
    if (e != cudaSuccess) return e;
    scan_sums_kernel<<<m, 1024, 0, s>>>(in, n, sums.p);
    scan_blocks_kernel<<<1, 1024, 0, s>>>(sums.p, m);
    scan_write_kernel<<<m, 1024, 0, s>>>(in, n, sums.p, out);
    return cudaGetLastError();
}

// Rows of up to R (deg[a] used) into CSR; one warp per row.
__global__ void __launch_bounds__(256) compact_kernel(const uint32_t *__restrict__ rows, uint32_t R,
                                                      const uint32_t *__restrict__ deg,
                                                      const uint64_t *__restrict__ off, uint32_t n,
                                                      uint32_t *__restrict__ out) {
    const uint32_t a = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (a >= n) return;
    const uint32_t m = deg[a];
    for (uint32_t e = lane; e < m; e += 32) out[off[a] + e] = rows[(size_t) a * R + e];
}

// Reverse edges. For every pruned edge a -> b (a ascending, then list order),
// b -> a is appended to b's list while it holds fewer than R and does not
// contain a already (efanna2e's InterInsert plays this part, with a re-prune on
// overflow instead of the cap). What b gets depends on b alone: the smallest
// ids among its in-neighbours that its pruned list lacks, ascending. So the
// pruned edges are transposed (counts, offsets, ids in any order), and one warp
// per vertex picks them. 200,000 vertices: 115 ms edge by edge on the host.
__global__ void __launch_bounds__(256) indegree_kernel(const uint32_t *__restrict__ rows, uint32_t R,
                                                       const uint32_t *__restrict__ deg, uint32_t n,
                                                       uint32_t *__restrict__ indeg) {
    const uint32_t a = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (a >= n) return;
    for (uint32_t e = lane; e < deg[a]; e += 32) atomicAdd(indeg + rows[(size_t) a * R + e], 1u);
}

__global__ void __launch_bounds__(256) transpose_kernel(const uint32_t *__restrict__ rows, uint32_t R,
                                                        const uint32_t *__restrict__ deg, uint32_t n,
                                                        const uint64_t *__restrict__ ioff,
                                                        uint32_t *__restrict__ fill, uint32_t *__restrict__ in) {
    const uint32_t a = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (a >= n) return;
    for (uint32_t e = lane; e < deg[a]; e += 32) {
        const uint32_t b = rows[(size_t) a * R + e];
        in[ioff[b] + atomicAdd(fill + b, 1u)] = a;
    }
}

constexpr uint32_t kRevList = 256;  // in-neighbours ranked in shared memory
__global__ void __launch_bounds__(256) reverse_kernel(uint32_t *__restrict__ rows, uint32_t R,
                                                      const uint32_t *__restrict__ deg, uint32_t n,
                                                      const uint64_t *__restrict__ ioff,
                                                      const uint32_t *__restrict__ in,
                                                      uint32_t *__restrict__ newdeg) {
    __shared__ uint32_t list[8][kRevList];
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.x * 8 + w;
    if (b >= n) return;
    const uint32_t d0 = deg[b];
    uint32_t *row = rows + (size_t) b * R;
    const uint32_t *src = in + ioff[b];
    const uint64_t m = ioff[b + 1] - ioff[b];
    const uint32_t want = R - d0;
    auto fresh = [&](uint32_t a) {  // not in b's pruned list
        bool has = false;
        for (uint32_t e = 0; e < d0; ++e) has = has || __ldg(row + e) == a;
        return !has;
    };
    uint32_t got = 0;
    if (m <= kRevList) {
        uint32_t c = 0;
        for (uint32_t i0 = 0; i0 < (uint32_t) m; i0 += 32) {
            const uint32_t i = i0 + lane;
            const uint32_t a = i < m ? src[i] : 0u;
            const bool keep = i < m && fresh(a);
            const uint32_t bm = __ballot_sync(0xffffffffu, keep);
            if (keep) list[w][c + __popc(bm & ((1u << lane) - 1u))] = a;
            c += __popc(bm);
        }
        __syncwarp();
        for (uint32_t i = lane; i < c; i += 32) {
            const uint32_t a = list[w][i];
            uint32_t rank = 0;
            for (uint32_t e = 0; e < c; ++e) rank += list[w][e] < a ? 1u : 0u;
            if (rank < want) row[d0 + rank] = a;
        }
        got = min(c, want);
    } else {
        // Many in-neighbours: the smallest one above the last, one at a time.
        uint32_t last = 0;
        while (got < want) {
            uint32_t best = 0xffffffffu;
            for (uint64_t i = lane; i < m; i += 32) {
                const uint32_t a = src[i];
                if (a < best && (got == 0 || a > last) && fresh(a)) best = a;
            }
            best = __reduce_min_sync(0xffffffffu, best);
            if (best == 0xffffffffu) break;
            if (lane == 0) row[d0 + got] = best;
            last = best;
            ++got;
        }
    }
    if (lane == 0) newdeg[b] = d0 + got;
}

// Parents of the repair's roots: the first vertex of root i's k-NN list that an
// earlier walk reached (walk[c] = 1 for the entry's, i + 2 for root i's), else
// the entry.
__global__ void __launch_bounds__(256) parent_kernel(const uint32_t *__restrict__ knn, uint32_t k, uint32_t n,
                                                     const uint32_t *__restrict__ roots, uint32_t m,
                                                     const uint32_t *__restrict__ walk, uint32_t entry,
                                                     uint32_t *__restrict__ parent) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    uint32_t p = entry;
    for (uint32_t e = 0; e < k; ++e) {
        const uint32_t c = knn[(size_t) roots[i] * k + e];
        if (c < n && walk[c] <= i + 1) {
            p = c;
            break;
        }
    }
    parent[i] = p;
}

}  // namespace

// The float32 screen of all rows, or (DIRECT) of the nr rows in the list `rows` (all
// without it).
template <bool DIRECT>
static int screen_fp32(const float *x, uint32_t n, uint32_t d, const float *xn, uint32_t C, const uint32_t *rows,
                       uint32_t nr, uint32_t *cand, cudaStream_t s) {
    const size_t smem = (size_t) (kBK * kBQ + kBK * kBV + kBQ * (kBV + 1)) * 4 + (size_t) kBQ * C * 8 + kBQ * 8;
    GCU(allow_shared((const void *) screen_kernel<DIRECT>));
    screen_kernel<DIRECT><<<(nr + kBQ - 1) / kBQ, 256, smem, s>>>(x, n, d, xn, C, rows, nr, cand);
    GCU(cudaGetLastError());
    return PANNS_OK;
}

// The float64 mean of the base, computed beside the screen.
struct MeanJob {
    cudaStream_t s = nullptr;
    cudaEvent_t ready = nullptr, done = nullptr;
    Scratch<double> mean;
    ~MeanJob() {
        if (s) cudaStreamSynchronize(s);
        mean.release();
        if (ready) cudaEventDestroy(ready);
        if (done) cudaEventDestroy(done);
        if (s) cudaStreamDestroy(s);
    }
    // x is complete on `from` at this point; `from` may use `mean` after wait().
    int start(const float *x, uint32_t n, uint32_t d, cudaStream_t from) {
        GCU(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        GCU(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
        GCU(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
        GCU(mean.alloc(d, s));
        GCU(cudaEventRecord(ready, from));
        GCU(cudaStreamWaitEvent(s, ready, 0));
        mean_kernel<<<(d + 31) / 32, 32, 0, s>>>(x, n, d, mean.p);
        GCU(cudaGetLastError());
        GCU(cudaEventRecord(done, s));
        return PANNS_OK;
    }
    int wait(cudaStream_t to) {
        GCU(cudaStreamWaitEvent(to, done, 0));
        return PANNS_OK;
    }
};

// The steps after the k-NN screen, shared by every construction: the C
// screened candidates of each row (cand, device, n x C; ~0 = none) ranked
// exactly by (d64, id) into k-NN lists, the MRNG prune to R, reverse edges, the
// entry (the row nearest the float64 mean) and the reachability repair. The
// lists stay on the device until they are a CSR graph; the walks of the repair
// follow it on the host, one after the other, and the lists of the vertices
// they start from are looked up on the device again. Rows go through the rank
// and the prune in chunks; k-NN lists above kKnnOnDevice bytes go to the host
// as they come.
constexpr size_t kKnnOnDevice = 4ull << 30;

static int finish_graph(int device, const float *x, uint32_t n, uint32_t d, uint32_t k, uint32_t R,
                        const uint32_t *cand, uint32_t C, MeanJob &mean, cudaStream_t s,
                        std::unique_ptr<panns_graph> &g, bool reverse = false) {
    const uint32_t chunk = std::min<uint32_t>(n, 1u << 23);
    const bool knn_host = (size_t) n * k * 4 > kKnnOnDevice;
    Buf<uint32_t> knn, pr, deg, entry;
    Buf<double> knn_d, dm;
    Buf<uint64_t> off;
    GCU(knn.alloc(knn_host ? (size_t) chunk * k : (size_t) n * k, s));
    GCU(knn_d.alloc((size_t) chunk * k, s));
    GCU(pr.alloc((size_t) n * R, s));
    GCU(deg.alloc(n, s));
    GCU(dm.alloc(n, s));
    GCU(entry.alloc(1, s));
    GCU(off.alloc((size_t) n + 1, s));
    g.reset(new panns_graph());
    g->n = n;
    g->k = k;
    g->device = device;
    if (knn_host) g->knn.resize((size_t) n * k);
    for (uint32_t a0 = 0; a0 < n; a0 += chunk) {
        const uint32_t na = std::min(chunk, n - a0);
        uint32_t *kn = knn_host ? knn.p : knn.p + (size_t) a0 * k;
        GCU(cudaMemsetAsync(kn, 0xff, (size_t) na * k * 4, s));
        if (d % 4 == 0 && d <= kMaxVecD)
            rerank_kernel<true><<<(na + 7) / 8, 256, 0, s>>>(x, n, d, cand, C, k, a0, na, kn, knn_d.p);
        else
            rerank_kernel<false><<<(na + 7) / 8, 256, 0, s>>>(x, n, d, cand, C, k, a0, na, kn, knn_d.p);
        GCU(cudaGetLastError());
        // Rows in shared memory while two blocks of at least one warp fit an SM.
        const uint32_t per_warp = prune_warp_bytes(d, k);
        uint32_t *prc = pr.p + (size_t) a0 * R;
        if (d % 4 == 0 && per_warp <= 112u * 1024u) {
            const uint32_t wpb = std::max(1u, std::min(4u, 112u * 1024u / per_warp));
            GCU(allow_shared((const void *) prune_rows_kernel));
            prune_rows_kernel<<<(na + wpb - 1) / wpb, wpb * 32, wpb * per_warp, s>>>(x, n, d, kn, knn_d.p, k, R, na, prc,
                                                                                    deg.p + a0);
        } else {
            prune_kernel<<<(na + 7) / 8, 256, 8 * R * 4, s>>>(x, n, d, kn, knn_d.p, k, R, na, prc, deg.p + a0);
        }
        GCU(cudaGetLastError());
        if (knn_host)
            GCU(cudaMemcpyAsync(g->knn.data() + (size_t) a0 * k, kn, (size_t) na * k * 4, cudaMemcpyDeviceToHost, s));
    }
    knn_d.release();
    // Entry: the row nearest the mean.
    int rc = mean.wait(s);
    if (rc) return rc;
    dist_to_point_kernel<<<(n + 255) / 256, 256, 0, s>>>(x, n, d, mean.mean.p, dm.p);
    argmin64_kernel<<<1, 1024, 0, s>>>(dm.p, n, entry.p);
    GCU(cudaGetLastError());
    GCU(cudaMemcpyAsync(&g->entry, entry.p, 4, cudaMemcpyDeviceToHost, s));
    if (reverse) {
        Buf<uint32_t> fill, in, deg2;
        Buf<uint64_t> ioff;
        GCU(fill.alloc(n, s));
        GCU(deg2.alloc(n, s));
        GCU(ioff.alloc((size_t) n + 1, s));
        GCU(cudaMemsetAsync(fill.p, 0, (size_t) n * 4, s));
        indegree_kernel<<<(n + 7) / 8, 256, 0, s>>>(pr.p, R, deg.p, n, fill.p);
        GCU(cudaGetLastError());
        GCU(scan_words(fill.p, n, ioff.p, s));
        uint64_t edges = 0;
        GCU(cudaMemcpyAsync(&edges, ioff.p + n, 8, cudaMemcpyDeviceToHost, s));
        GCU(cudaStreamSynchronize(s));
        GCU(in.alloc((size_t) edges, s));
        GCU(cudaMemsetAsync(fill.p, 0, (size_t) n * 4, s));
        transpose_kernel<<<(n + 7) / 8, 256, 0, s>>>(pr.p, R, deg.p, n, ioff.p, fill.p, in.p);
        reverse_kernel<<<(n + 7) / 8, 256, 0, s>>>(pr.p, R, deg.p, n, ioff.p, in.p, deg2.p);
        GCU(cudaGetLastError());
        GCU(cudaMemcpyAsync(deg.p, deg2.p, (size_t) n * 4, cudaMemcpyDeviceToDevice, s));
    }
    // The lists as a CSR graph, to the host (with room for one repair edge per vertex).
    GCU(scan_words(deg.p, n, off.p, s));
    std::vector<uint64_t> &go = g->off;
    go.resize((size_t) n + 1);
    GCU(cudaMemcpyAsync(go.data(), off.p, ((size_t) n + 1) * 8, cudaMemcpyDeviceToHost, s));
    GCU(cudaStreamSynchronize(s));
    const uint64_t edges = go[n];
    {
        Buf<uint32_t> csr;
        GCU(csr.alloc((size_t) edges, s));
        compact_kernel<<<(n + 7) / 8, 256, 0, s>>>(pr.p, R, deg.p, off.p, n, csr.p);
        GCU(cudaGetLastError());
        pr.release();
        g->nbrs.resize((size_t) edges, (size_t) edges + n);
        GCU(cudaMemcpyAsync(g->nbrs.data(), csr.p, (size_t) edges * 4, cudaMemcpyDeviceToHost, s));
        GCU(cudaStreamSynchronize(s));
    }
    // Reachability repair: walks over the lists, from the entry and then from
    // every vertex no walk has reached yet, in id order. walk[v] is the number of
    // the walk that reached v. A repair edge parent -> root is followed at once by
    // the walk from the root, so walks never need the repair edges themselves.
    std::vector<uint32_t> walk(n, 0), queue(n), roots;
    const uint32_t *nb = g->nbrs.data();
    auto follow = [&](uint32_t src, uint32_t number) {  // breadth-first
        size_t head = 0, tail = 0;
        walk[src] = number;
        queue[tail++] = src;
        while (head < tail) {
            if (head + 8 < tail) __builtin_prefetch(&go[queue[head + 8]]);
            if (head + 4 < tail) {
                const uint32_t *p = nb + go[queue[head + 4]];
                __builtin_prefetch(p);
                __builtin_prefetch(p + 16);
            }
            const uint32_t v = queue[head++];
            for (uint64_t e = go[v]; e < go[v + 1]; ++e) {
                const uint32_t u = nb[e];
                if (!walk[u]) {
                    walk[u] = number;
                    queue[tail++] = u;
                }
            }
        }
    };
    follow(g->entry, 1);
    for (uint32_t u = 0; u < n; ++u)
        if (!walk[u]) {
            roots.push_back(u);
            follow(u, (uint32_t) roots.size() + 1);
        }
    const uint32_t m = (uint32_t) roots.size();
    std::vector<uint32_t> parent(m);
    if (m && !knn_host) {
        Buf<uint32_t> droots, dwalk, dparent;
        GCU(droots.alloc(m, s));
        GCU(dwalk.alloc(n, s));
        GCU(dparent.alloc(m, s));
        GCU(cudaMemcpyAsync(droots.p, roots.data(), m * 4ull, cudaMemcpyHostToDevice, s));
        GCU(cudaMemcpyAsync(dwalk.p, walk.data(), (size_t) n * 4, cudaMemcpyHostToDevice, s));
        parent_kernel<<<(m + 255) / 256, 256, 0, s>>>(knn.p, k, n, droots.p, m, dwalk.p, g->entry, dparent.p);
        GCU(cudaGetLastError());
        GCU(cudaMemcpyAsync(parent.data(), dparent.p, m * 4ull, cudaMemcpyDeviceToHost, s));
        GCU(cudaStreamSynchronize(s));
    } else {
        for (uint32_t i = 0; i < m; ++i) {
            parent[i] = g->entry;
            for (uint32_t e = 0; e < k; ++e) {
                const uint32_t c = g->knn[(size_t) roots[i] * k + e];
                if (c < n && walk[c] <= i + 1) {
                    parent[i] = c;
                    break;
                }
            }
        }
    }
    g->repaired = m;
    // The repair edges at the ends of their parents' lists, in the order they
    // were made: rows move up, the last first.
    if (m) {
        std::vector<uint32_t> &more = queue;  // repair edges per vertex
        std::fill(more.begin(), more.end(), 0u);
        for (uint32_t i = 0; i < m; ++i) ++more[parent[i]];
        uint64_t shift = m;
        uint64_t end = go[n];
        go[n] += m;
        g->nbrs.n += m;
        for (uint32_t a = n; a-- > 0 && shift;) {
            const uint64_t b0 = go[a];
            shift -= more[a];
            memmove(g->nbrs.data() + b0 + shift, g->nbrs.data() + b0, (size_t) (end - b0) * 4);
            end = b0;
            go[a] = b0 + shift;
        }
        for (uint32_t i = 0; i < m; ++i) g->nbrs[(size_t) (go[parent[i] + 1] - more[parent[i]]--)] = roots[i];
    }
    for (uint32_t a = 0; a < n; ++a) g->width = std::max(g->width, (uint32_t) (go[a + 1] - go[a]));
    if (!knn_host) g->knn_dev = knn.take();
    return PANNS_OK;
}

}  // namespace panns

using namespace panns;

extern "C" {

int panns_build_nsg(int device, const float *base, uint32_t n, uint32_t d, uint32_t knn_k, uint32_t R,
                    panns_graph **out) {
    return panns_build_nsg_ex(device, base, n, d, knn_k, R, PANNS_SCREEN_AUTO, out);
}

int panns_build_nsg_ex(int device, const float *base, uint32_t n, uint32_t d, uint32_t knn_k, uint32_t R,
                       uint32_t screen, panns_graph **out) {
    if (!out || !base) return set_error(PANNS_EINVAL, "panns_build_nsg: NULL argument");
    *out = nullptr;
    if (n < 2 || d == 0) return set_error(PANNS_EINVAL, "panns_build_nsg: need n >= 2, d > 0");
    if (knn_k == 0 || knn_k >= n) return set_error(PANNS_EINVAL, "panns_build_nsg: need 0 < knn_k < n");
    if (knn_k + 8 > (uint32_t) kMaxC) return set_error(PANNS_EINVAL, "panns_build_nsg: knn_k > 128 is not supported");
    if (R == 0 || R > knn_k) return set_error(PANNS_EINVAL, "panns_build_nsg: need 0 < R <= knn_k");
    if (screen > PANNS_SCREEN_TC) return set_error(PANNS_EINVAL, "panns_build_nsg: unknown screen");
    const uint32_t k = knn_k;
    const uint32_t C_tc = std::min(std::min(knn_k + 32u, (uint32_t) kMaxC), n - 1);
    const bool automatic = screen == PANNS_SCREEN_AUTO;
    if (automatic)
        screen = n >= kTcMinRows && d <= 256 ? PANNS_SCREEN_TC : n < 100000 ? PANNS_SCREEN_FP32 : PANNS_SCREEN_TF32;
    if (!automatic && screen == PANNS_SCREEN_TC && !tc_screen_supported(n, d, C_tc))
        return set_error(PANNS_EINVAL, "panns_build_nsg: the tcgen05 screen needs d a multiple of 32 up to 128 "
                                       "and n >= 128");
    const bool tc = screen == PANNS_SCREEN_TF32;
    const bool tcg = screen == PANNS_SCREEN_TC;
    const uint32_t C = (tc || tcg) ? C_tc : std::min(std::min(knn_k + 8u, (uint32_t) kMaxC), n - 1);
    GCU(cudaSetDevice(device));
    cudaStream_t s = nullptr;
    GCU(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct SG {
        cudaStream_t s;
        ~SG() { cudaStreamDestroy(s); }
    } sg{s};
    Buf<float> x, xn;
    Buf<uint32_t> cand;
    GCU(x.alloc((size_t) n * d, s));
    GCU(xn.alloc(n, s));
    GCU(cand.alloc((size_t) n * C, s));
    GCU(cudaMemcpyAsync(x.p, base, (size_t) n * d * 4, cudaMemcpyHostToDevice, s));
    MeanJob mean;
    {
        const int rc = mean.start(x.p, n, d, s);
        if (rc) return rc;
    }
    sqnorm32_kernel<<<(n + 255) / 256, 256, 0, s>>>(x.p, n, d, xn.p);
    if (tcg) {
        int num_sms = 0;
        GCU(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, device));
        Buf<uint32_t> perm, fail, nfail;
        GCU(fail.alloc(n, s));
        GCU(nfail.alloc(1, s));
        int rc = PANNS_OK;
        uint32_t slots = n;
        if (n > 32 * kTcM) {  // below, every tile is near every other
            GCU(perm.alloc(tc_order_slots(n, true), s));
            rc = tc_locality_order(x.p, n, d, true, perm.p, &slots, s);
            if (rc) return rc;
        }
        bool safe = false;
        rc = tc_screen_knn(x.p, n, d, k, C, perm.p, slots, nullptr, cand.p, fail.p, nfail.p, &safe, num_sms, s);
        if (rc) return rc;
        // Rows that screen could not settle (long runs of equal distances,
        // non-finite values) go through the float32 one.
        uint32_t nf = n;
        if (safe) GCU(cudaMemcpyAsync(&nf, nfail.p, 4, cudaMemcpyDeviceToHost, s));
        GCU(cudaStreamSynchronize(s));
        if (nf) {
            rc = screen_fp32<true>(x.p, n, d, xn.p, C, safe ? fail.p : nullptr, nf, cand.p, s);
            if (rc) return rc;
            GCU(cudaStreamSynchronize(s));
        }
    } else if (!tc) {
        const int rc = screen_fp32<false>(x.p, n, d, xn.p, C, nullptr, n, cand.p, s);
        if (rc) return rc;
    } else {
        // -2 x.y for tiles of TR rows x TC candidates by TF32 tensor-core GEMMs
        // (cuBLAS, a plain library GEMM), each folded into the rows' lists.
        const uint32_t TR = std::min(n, 8192u), TC = std::min(n, 32768u);
        Buf<float> G, gld;
        Buf<uint32_t> gcnt;
        GCU(G.alloc((size_t) TR * TC, s));
        GCU(gld.alloc((size_t) n * C, s));
        GCU(gcnt.alloc(n, s));
        GCU(cudaMemsetAsync(gcnt.p, 0, n * 4ull, s));
        cublasHandle_t hb = nullptr;
        if (cublasCreate(&hb) != CUBLAS_STATUS_SUCCESS) return set_error(PANNS_ECUDA, "panns_build_nsg: cublasCreate failed");
        struct HB {
            cublasHandle_t h;
            ~HB() { cublasDestroy(h); }
        } hbg{hb};
        if (cublasSetStream(hb, s) != CUBLAS_STATUS_SUCCESS)
            return set_error(PANNS_ECUDA, "panns_build_nsg: cublasSetStream failed");
        const float alpha = -2.f, beta = 0.f;
        for (uint32_t r0 = 0; r0 < n; r0 += TR) {
            const uint32_t nr = std::min(TR, n - r0);
            for (uint32_t c0 = 0; c0 < n; c0 += TC) {
                const uint32_t nc = std::min(TC, n - c0);
                const cublasStatus_t st = cublasGemmEx(
                    hb, CUBLAS_OP_T, CUBLAS_OP_N, (int) nc, (int) nr, (int) d, &alpha, x.p + (size_t) c0 * d, CUDA_R_32F,
                    (int) d, x.p + (size_t) r0 * d, CUDA_R_32F, (int) d, &beta, G.p, CUDA_R_32F, (int) nc,
                    CUBLAS_COMPUTE_32F_FAST_TF32, CUBLAS_GEMM_DEFAULT);
                if (st != CUBLAS_STATUS_SUCCESS)
                    return set_error(PANNS_ECUDA, "panns_build_nsg: cublasGemmEx failed (" + std::to_string((int) st) + ")");
                topk_tile_kernel<<<(nr + 7) / 8, 256, 0, s>>>(G.p, nr, nc, r0, c0, xn.p, n, C, gld.p, cand.p, gcnt.p);
                GCU(cudaGetLastError());
            }
        }
        GCU(cudaStreamSynchronize(s));
    }
    std::unique_ptr<panns_graph> g;
    const int rc = finish_graph(device, x.p, n, d, k, R, cand.p, C, mean, s, g);
    if (rc) return rc;
    *out = g.release();
    return PANNS_OK;
}

int panns_build_nsg_cells(int device, const float *base, uint32_t n, uint32_t d, uint32_t knn_k, uint32_t R,
                          uint32_t cells, uint32_t probe, uint32_t sample, uint32_t iters, uint32_t seed,
                          uint32_t reverse, panns_graph **out) {
    if (!out || !base) return set_error(PANNS_EINVAL, "panns_build_nsg_cells: NULL argument");
    *out = nullptr;
    if (n < 2 || d == 0) return set_error(PANNS_EINVAL, "panns_build_nsg_cells: need n >= 2, d > 0");
    if (knn_k == 0 || knn_k >= n) return set_error(PANNS_EINVAL, "panns_build_nsg_cells: need 0 < knn_k < n");
    if (knn_k + 8 > (uint32_t) kMaxC) return set_error(PANNS_EINVAL, "panns_build_nsg_cells: knn_k > 128 is not supported");
    if (R == 0 || R > knn_k) return set_error(PANNS_EINVAL, "panns_build_nsg_cells: need 0 < R <= knn_k");
    const uint32_t S = std::min(n, std::max(sample, cells));
    if (cells < 1 || cells > S) return set_error(PANNS_EINVAL, "panns_build_nsg_cells: need 1 <= cells <= sample, n");
    if (probe > 8 || (probe >= cells && cells > 1)) return set_error(PANNS_EINVAL, "panns_build_nsg_cells: need probe <= 8 and probe < cells");
    const uint32_t k = knn_k, P = cells > 1 ? probe : 0u;
    const uint32_t C = std::min(knn_k + 16u, (uint32_t) kMaxC);
    GCU(cudaSetDevice(device));
    cudaStream_t s = nullptr;
    GCU(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct SG {
        cudaStream_t s;
        ~SG() { cudaStreamDestroy(s); }
    } sg{s};
    Buf<float> x, xn;
    GCU(x.alloc((size_t) n * d, s));
    GCU(xn.alloc(n, s));
    GCU(cudaMemcpyAsync(x.p, base, (size_t) n * d * 4, cudaMemcpyHostToDevice, s));
    MeanJob mean;
    {
        const int rc = mean.start(x.p, n, d, s);
        if (rc) return rc;
    }
    sqnorm32_kernel<<<(n + 255) / 256, 256, 0, s>>>(x.p, n, d, xn.p);
    GCU(cudaGetLastError());
    // Cells: Lloyd k-means on S rows at a fixed stride, then every row to its
    // nearest centroid; each cell's P nearest cells by centroid distance.
    std::vector<uint32_t> cellh(n), nearh((size_t) cells * std::max(P, 1u), 0xffffffffu), cstart(cells + 1);
    Buf<uint32_t> dmem, dstart;
    GCU(dmem.alloc(n, s));
    GCU(dstart.alloc(cells + 1, s));
    {
        Buf<uint32_t> sidx, sas, srep, dcell, dnear;
        Buf<float> xs, cent;
        std::vector<uint32_t> idx(S);
        for (uint32_t i = 0; i < S; ++i) idx[i] = (uint32_t) ((uint64_t) i * n / S);
        GCU(sidx.alloc(S, s));
        GCU(xs.alloc((size_t) S * d, s));
        GCU(sas.alloc(S, s));
        GCU(srep.alloc(cells, s));
        GCU(cent.alloc((size_t) cells * d, s));
        GCU(dcell.alloc(n, s));
        GCU(cudaMemcpyAsync(sidx.p, idx.data(), S * 4ull, cudaMemcpyHostToDevice, s));
        gather_rows_f32_kernel<<<1024, 256, 0, s>>>(x.p, d, sidx.p, S, xs.p);
        GCU(cudaGetLastError());
        int rc = kmeans_run(xs.p, S, d, cells, iters, seed, cent.p, sas.p, srep.p, s);
        if (rc) return rc;
        rc = nearest_centroid(x.p, n, d, cent.p, cells, dcell.p, s);
        if (rc) return rc;
        // Members of each cell in id order.
        GCU(cell_sort(dcell.p, n, cells, dstart.p, dmem.p, s));
        GCU(cudaMemcpyAsync(cellh.data(), dcell.p, n * 4ull, cudaMemcpyDeviceToHost, s));
        GCU(cudaMemcpyAsync(cstart.data(), dstart.p, (cells + 1) * 4ull, cudaMemcpyDeviceToHost, s));
        if (P) {
            GCU(dnear.alloc((size_t) cells * P, s));
            near_cells_kernel<<<cells, 256, 0, s>>>(cent.p, cells, d, P, dnear.p);
            GCU(cudaGetLastError());
            GCU(cudaMemcpyAsync(nearh.data(), dnear.p, (size_t) cells * P * 4, cudaMemcpyDeviceToHost, s));
        }
        GCU(cudaStreamSynchronize(s));
    }
    Buf<uint32_t> cand;
    GCU(cand.alloc((size_t) n * C, s));
    GCU(cudaMemsetAsync(cand.p, 0xff, (size_t) n * C * 4, s));
    // Tensor-core screen: every cell padded to whole tiles, a row block of one
    // cell against the tiles of the cell and of its near cells. Where padding
    // would more than double the rows (cells of a few dozen rows) the float32
    // screen runs, and it runs for the rows whose lists cannot be settled.
    uint64_t slots = 0;
    for (uint32_t c = 0; c < cells; ++c) slots += (cstart[c + 1] - cstart[c] + kTcM - 1) / kTcM * (uint64_t) kTcM;
    std::vector<uint32_t> left;  // rows for the float32 screen, cell by cell
    bool all_left = true;
    bool direct = false;  // the tensor-core screen ran
    size_t free_b = 0, total_b = 0;
    GCU(cudaMemGetInfo(&free_b, &total_b));
    if (d <= 256 && n >= kTcMinRows && slots <= 2ull * n && slots <= 0x7fffffffull &&
        tc_knn_bytes(slots, d) <= free_b / 5 * 3) {
        std::vector<uint32_t> tile0(cells + 1, 0), avail(cells, 0), blk;
        blk.reserve((size_t) (slots / kTcM));
        for (uint32_t c = 0; c < cells; ++c) {
            const uint32_t m = cstart[c + 1] - cstart[c], t = (m + kTcM - 1) / kTcM;
            blk.insert(blk.end(), t, c);
            tile0[c + 1] = tile0[c] + t;
            avail[c] = m;
            for (uint32_t i = 0; i < P; ++i) {
                const uint32_t o = nearh[(size_t) c * P + i];
                if (o != 0xffffffffu) avail[c] += cstart[o + 1] - cstart[o];
            }
        }
        int num_sms = 0;
        GCU(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, device));
        Buf<uint32_t> dorder, dblk, dt0, dnear, davail, fail, nfail;
        GCU(dorder.alloc((size_t) slots, s));
        GCU(dblk.alloc(blk.size(), s));
        GCU(dt0.alloc(cells + 1, s));
        GCU(dnear.alloc(nearh.size(), s));
        GCU(davail.alloc(cells, s));
        GCU(fail.alloc(n, s));
        GCU(nfail.alloc(1, s));
        GCU(cudaMemsetAsync(dorder.p, 0xff, (size_t) slots * 4, s));
        GCU(cudaMemcpyAsync(dblk.p, blk.data(), blk.size() * 4, cudaMemcpyHostToDevice, s));
        GCU(cudaMemcpyAsync(dt0.p, tile0.data(), (cells + 1) * 4ull, cudaMemcpyHostToDevice, s));
        pad_cells_kernel<<<cells, 256, 0, s>>>(dmem.p, dstart.p, dt0.p, dorder.p);
        GCU(cudaGetLastError());
        GCU(cudaMemcpyAsync(dnear.p, nearh.data(), nearh.size() * 4, cudaMemcpyHostToDevice, s));
        GCU(cudaMemcpyAsync(davail.p, avail.data(), cells * 4ull, cudaMemcpyHostToDevice, s));
        const TcCells tc{dblk.p, dt0.p, dnear.p, davail.p, P};
        bool safe = false;
        const int rc = tc_screen_knn(x.p, n, d, k, C, dorder.p, (uint32_t) slots, &tc, cand.p, fail.p, nfail.p, &safe,
                                     num_sms, s);
        if (rc) return rc;
        direct = true;
        all_left = !safe;
        if (safe) {
            uint32_t nf = 0;
            GCU(cudaMemcpyAsync(&nf, nfail.p, 4, cudaMemcpyDeviceToHost, s));
            GCU(cudaStreamSynchronize(s));
            left.resize(nf);
            if (nf) GCU(cudaMemcpyAsync(left.data(), fail.p, (size_t) nf * 4, cudaMemcpyDeviceToHost, s));
            GCU(cudaStreamSynchronize(s));
            std::sort(left.begin(), left.end(), [&cellh](uint32_t a, uint32_t b) {
                return cellh[a] != cellh[b] ? cellh[a] < cellh[b] : a < b;
            });
        }
    }
    if (all_left || !left.empty()) {
        // Blocks of up to kBQ rows of one cell.
        std::vector<uint32_t> blk_cell, blk_row0;
        const uint32_t rows = all_left ? n : (uint32_t) left.size();
        for (uint32_t r = 0, c = 0; r < rows;) {
            uint32_t end;
            if (all_left) {
                while (cstart[c + 1] <= r) ++c;
                end = std::min(cstart[c + 1], r + kBQ);
            } else {
                c = cellh[left[r]];
                for (end = r + 1; end < rows && end < r + kBQ && cellh[left[end]] == c;) ++end;
            }
            blk_cell.push_back(c);
            blk_row0.push_back(r);
            r = end;
        }
        blk_row0.push_back(rows);
        Buf<uint32_t> dnear, dbc, dbr, drows;
        GCU(dnear.alloc(nearh.size(), s));
        GCU(dbc.alloc(blk_cell.size(), s));
        GCU(dbr.alloc(blk_row0.size(), s));
        GCU(drows.alloc(left.size(), s));
        if (!left.empty())
            GCU(cudaMemcpyAsync(drows.p, left.data(), left.size() * 4, cudaMemcpyHostToDevice, s));
        GCU(cudaMemcpyAsync(dnear.p, nearh.data(), nearh.size() * 4, cudaMemcpyHostToDevice, s));
        GCU(cudaMemcpyAsync(dbc.p, blk_cell.data(), blk_cell.size() * 4, cudaMemcpyHostToDevice, s));
        GCU(cudaMemcpyAsync(dbr.p, blk_row0.data(), blk_row0.size() * 4, cudaMemcpyHostToDevice, s));
        const size_t smem = (size_t) (kBK * kBQ + kBK * kBV + kBQ * (kBV + 1)) * 4 + (size_t) kBQ * C * 8 +
                            (size_t) kBQ * 8 + (size_t) kBV * 4;
        const auto kern = direct ? screen_cells_kernel<true> : screen_cells_kernel<false>;
        GCU(allow_shared((const void *) kern));
        kern<<<(unsigned) blk_cell.size(), 256, smem, s>>>(x.p, n, d, xn.p, C, dmem.p, dstart.p, dnear.p, P,
                                                           all_left ? dmem.p : drows.p, dbc.p, dbr.p, cand.p);
        GCU(cudaGetLastError());
        GCU(cudaStreamSynchronize(s));
    }
    std::unique_ptr<panns_graph> g;
    const int rc = finish_graph(device, x.p, n, d, k, R, cand.p, C, mean, s, g, reverse != 0);
    if (rc) return rc;
    g->cells = cells;
    g->probe = P;
    g->cell.swap(cellh);
    g->near.swap(nearh);
    *out = g.release();
    return PANNS_OK;
}

int panns_graph_cells(const panns_graph *g, uint32_t *cells, uint32_t *probe, uint32_t *cell, uint32_t *near) {
    if (!g) return set_error(PANNS_EINVAL, "panns_graph_cells: NULL graph");
    if (cells) *cells = g->cells;
    if (probe) *probe = g->probe;
    if (cell && !g->cell.empty()) memcpy(cell, g->cell.data(), g->cell.size() * 4);
    if (near && g->probe) memcpy(near, g->near.data(), (size_t) g->cells * g->probe * 4);
    return PANNS_OK;
}

int panns_graph_info(const panns_graph *g, uint32_t *n, uint32_t *width, uint32_t *entry, uint64_t *n_edges,
                     uint32_t *repaired) {
    if (!g) return set_error(PANNS_EINVAL, "panns_graph_info: NULL graph");
    if (n) *n = g->n;
    if (width) *width = g->width;
    if (entry) *entry = g->entry;
    if (n_edges) *n_edges = g->off.empty() ? 0 : g->off.back();
    if (repaired) *repaired = g->repaired;
    return PANNS_OK;
}

int panns_graph_copy(const panns_graph *g, uint64_t *offsets, uint32_t *nbrs, uint32_t *knn) {
    if (!g) return set_error(PANNS_EINVAL, "panns_graph_copy: NULL graph");
    if (offsets) memcpy(offsets, g->off.data(), g->off.size() * 8);
    if (nbrs && !g->nbrs.empty()) memcpy(nbrs, g->nbrs.data(), g->nbrs.size() * 4);
    if (knn && g->knn_dev) {
        GCU(g->copy_knn(knn));
    } else if (knn) {
        memcpy(knn, g->knn.data(), g->knn.size() * 4);
    }
    return PANNS_OK;
}

int panns_graph_save_nsg(const panns_graph *g, const char *path) {
    if (!g || !path) return set_error(PANNS_EINVAL, "panns_graph_save_nsg: NULL argument");
    FILE *f = fopen(path, "wb");
    if (!f) return set_error(PANNS_EIO, std::string("panns_graph_save_nsg: cannot open ") + path);
    bool ok = fwrite(&g->width, 4, 1, f) == 1 && fwrite(&g->entry, 4, 1, f) == 1;
    for (uint32_t a = 0; ok && a < g->n; ++a) {
        const uint32_t k = (uint32_t) (g->off[a + 1] - g->off[a]);
        ok = fwrite(&k, 4, 1, f) == 1 && (k == 0 || fwrite(g->nbrs.data() + g->off[a], 4, k, f) == k);
    }
    ok = (fclose(f) == 0) && ok;
    return ok ? PANNS_OK : set_error(PANNS_EIO, std::string("panns_graph_save_nsg: write failed: ") + path);
}

int panns_graph_free(panns_graph *g) {
    delete g;
    return PANNS_OK;
}

}  // extern "C"
