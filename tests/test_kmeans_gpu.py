"""k-means seeding, the cell lists and the centroid means against numpy, at the
sizes where their kernels change: rows of one and several 128-wide passes, samples
that fill no block, one row per cell, more row chunks than one scan pass.

Coordinates are small integers, so every distance of the seeding and of the first
assignment is exact in float32 and the picks have one right answer; afterwards the
cells may differ only where two centroids are as close as the rounding of the
distances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [(300, 8, 1), (300, 40, 300), (4999, 96, 37), (5000, 136, 64), (2111, 256, 300),
                                   (140_001, 8, 3)])
def test_kmeans_against_numpy(n, d, k):
    from parallel_anns_b200 import learned as LE
    from parallel_anns_b200.searching import Index
    rng = np.random.default_rng(n + d)
    x = rng.integers(0, 64, size=(n, d)).astype(np.float32)
    x64 = x.astype(np.float64)
    with Index(0) as ix:
        ix.set_base(x)
        reps0, as0 = LE.kmeans(ix, k, 0, seed=7)
        reps1, as1 = LE.kmeans(ix, k, 1, seed=7)
    assert len(np.unique(x, axis=0)) == n  # distinct rows: a centre's nearest row is itself
    # Seeding: the farthest sample row each time, ties to the lower sample.
    S = min(n, 32 * k)
    idx = np.arange(S, dtype=np.int64) * n // S
    assert reps0[0] in idx
    mind = ((x64[idx] - x64[reps0[0]]) ** 2).sum(1)
    for c in range(1, k):
        assert reps0[c] == idx[mind.argmax()], c
        mind = np.minimum(mind, ((x64[idx] - x64[reps0[c]]) ** 2).sum(1))
    # First cells: the nearest centre, ties to the lower cell.
    best = np.full(n, np.inf)
    cell = np.zeros(n, np.uint32)
    for c in range(k):
        dist = ((x64 - x64[reps0[c]]) ** 2).sum(1)
        cell[dist < best] = c
        best = np.minimum(best, dist)
    assert np.array_equal(as0, cell)
    # One round: the means (exact sums), the cells by them, each cell's nearest row.
    cent = np.stack([(x64[cell == c].sum(0) / (cell == c).sum()).astype(np.float32) for c in range(k)]).astype(np.float64)
    dist = (x64 ** 2).sum(1)[:, None] - 2 * x64 @ cent.T + (cent ** 2).sum(1)
    # A split-TF32 product and its float32 sum: 2^-21 of each term and d roundings.
    tol = (d + 8) * 2.0 ** -22 * ((cent ** 2).sum(1).max() + 2 * np.sqrt((x64 ** 2).sum(1).max() * (cent ** 2).sum(1).max()))
    assert np.all(dist[np.arange(n), as1] <= dist.min(1) + 2 * tol)
    for c in range(k):
        rows = np.nonzero(as1 == c)[0]
        if rows.size == 0:
            continue
        own = ((x64[rows] - cent[c]) ** 2).sum(1)
        assert as1[reps1[c]] == c
        assert own[rows == reps1[c]][0] <= own.min() * (1 + (d + 8) * 2.0 ** -22) + 1e-9
    assert len(set(reps1.tolist())) == k  # empty cells got rows of their own
