// Distance screens on the 5th-generation tensor cores (tc_screen.cu): the
// k-NN screen of the graph construction (graph_build.cu) and the range screen
// of the ground truth (panns_abi.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace panns {

constexpr uint32_t kTcM = 128;  // rows per block, and columns per tile

// Shapes the k-NN screen is offered for by name (PANNS_SCREEN_TC): d a
// multiple of 32 up to 128, 0 < C <= 128, C < n, n >= 128.
bool tc_screen_supported(uint32_t n, uint32_t d, uint32_t C);

// Rows grouped by their nearest of a few pivot rows, so that a block of
// consecutive positions covers a small part of the space. Padded: every group
// starts at a multiple of kTcM positions, with ~0 (no row) in between, so no
// tile holds rows of two groups. tc_order_slots: positions at most; perm
// (device, that many entries): the row at each position; *slots: positions
// used. Without padding perm holds n entries and *slots = n. Enqueued on `s`
// and synchronised.
uint32_t tc_order_slots(uint32_t n, bool padded);
int tc_locality_order(const float *x, uint32_t n, uint32_t d, bool padded, uint32_t *perm, uint32_t *slots,
                      cudaStream_t s);

// The cells of a cell-restricted screen: `perm` lists the rows cell by cell,
// each cell padded with ~0 to a multiple of kTcM; the tiles of cell c are
// tile0[c] .. tile0[c + 1] (device, cells + 1 entries). A row is screened
// against its own cell and the P cells near[c * P ..] (~0: none).
struct TcCells {
    const uint32_t *blk_cell;  // cell of every row block (device)
    const uint32_t *tile0;
    const uint32_t *near;
    const uint32_t *avail;     // rows in a cell and its near cells together
    uint32_t P;
};

// k-NN candidates: cand[i * C + j], j < C, holds rows y != x_i of the base x
// (n x d float32, device), ~0 where there are fewer, in no particular order.
// They include the k nearest of the rows screened (all, or the cells' when
// `cells` is given) unless row i is listed in fail_rows[0 .. *fail_count)
// (device; for these rows cand is not written). *safe = false: a finite row is so
// far from the others that the error bound does not hold, cand is not to be used
// for any row. perm (device, `slots`
// entries, ~0 = no row; null = identity) is the order the rows are processed
// in. Enqueued on `s` and synchronised.
int tc_screen_knn(const float *x, uint32_t n, uint32_t d, uint32_t k, uint32_t C, const uint32_t *perm, uint32_t slots,
                  const TcCells *cells, uint32_t *cand, uint32_t *fail_rows, uint32_t *fail_count, bool *safe,
                  int num_sms, cudaStream_t s);

// Device memory tc_screen_knn takes for this many positions (besides the tile bounds).
size_t tc_knn_bytes(uint64_t slots, uint32_t d);

// Range lists: for query i (row qperm[i] of `queries`, nq rows of width d,
// device), every row y of x with ||y - q||^2 <= tau[i] (float64, by position i
// too), and few others: the entry e of split p is lists[(p * nq + i) * cap + e]
// = {screen distance bits, position in perm}, e < cnt[p * nq + i] (entries from
// cap on are counted, not stored). perm (`slots` positions, ~0 = no row): the
// order the rows of x are processed in. *safe = false: a vector is not finite, or so
// far from the others that the error bound does not hold; the lists are not to be
// used. splits: from
// tc_range_splits. Enqueued on `s` and synchronised.
constexpr uint32_t kTcMaxSplits = 8;
uint32_t tc_range_splits(uint32_t nq, int num_sms);
int tc_screen_range(const float *x, uint32_t n, uint32_t d, const uint32_t *perm, uint32_t slots,
                    const float *queries, const uint32_t *qperm, uint32_t nq, const double *tau, uint32_t splits,
                    uint2 *lists, uint32_t cap, uint32_t *cnt, bool *safe, int num_sms, cudaStream_t s);

}  // namespace panns
