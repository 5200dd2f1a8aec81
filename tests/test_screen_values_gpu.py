"""The tensor-core screens over the range of float32 values: bases scaled by powers
of two down to where squared norms leave float32, and up to where they overflow;
rows far from all others; rows with infinities and NaNs. A power of two changes no
float64 comparison, so the lists, graphs and ids equal those of the unscaled base,
and distances are its distances times the square."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SCALES = [-100, -70, -63, -55, 40, 62, 100]


def _mix(n, d, seed):
    from parallel_anns_b200 import datasets as ds
    return ds.gaussian_mixture(n, d, 64, 0.3, seed=seed, means_seed=seed)


@pytest.fixture(scope="module")
def small():
    x = _mix(4225, 96, 8)
    return x, O.build_nsg(x, 64, 40)


@pytest.mark.parametrize("e", SCALES)
def test_build_of_scaled_rows(small, e):
    from parallel_anns_b200.graph import build_nsg
    x, (og, oknn) = small
    g, knn = build_nsg(np.ldexp(x, e), R=40, knn_k=64, with_knn=True)
    assert np.array_equal(knn, oknn)
    assert g.entry == og.entry and np.array_equal(g.offsets, og.offsets) and np.array_equal(g.nbrs, og.nbrs)


@pytest.mark.parametrize("e", SCALES)
def test_ground_truth_of_scaled_rows(small, e):
    """As many queries as the screen takes, and few."""
    from parallel_anns_b200.searching import Index, ground_truth
    x, (og, _) = small
    from parallel_anns_b200.formats import NSGGraph
    q = _mix(4000, 96, 8)[::-1].copy()
    q[0] = 0.0  # far from the base's mean, in its units
    q[1] = x[17]
    oids, odist = O.ground_truth(x, q, 20)
    with Index(0) as ix:
        ix.set_base(np.ldexp(x, e))
        ix.set_graph(NSGGraph(og.width, og.entry, og.offsets, og.nbrs))
        for m in (4000, 3):
            ids, dist = ground_truth(ix, np.ldexp(q[:m], e), 20)
            assert np.array_equal(ids, oids[:m])
            np.testing.assert_allclose(np.ldexp(dist, -2 * e), odist[:m], rtol=98 * 2.0 ** -52, atol=0)


def _in_cells(x, knn, cell, near, k, rows):
    """Exact lists of `rows` over their cells and near cells (float64)."""
    x = x.astype(np.float64)
    for a in rows:
        cand = np.flatnonzero(np.isin(cell, [cell[a], *near[cell[a]]]))
        cand = cand[cand != a]
        dd = np.square(x[cand] - x[a]).sum(1)
        want = np.sort(dd)[:k]
        got = knn[a][knn[a] < x.shape[0]]
        assert got.size == want.size and np.unique(got).size == got.size and np.isin(got, cand).all(), a
        np.testing.assert_allclose(np.square(x[got] - x[a]).sum(1), want, rtol=1e-12, atol=0)


@pytest.mark.parametrize("e", [-70, -63, 62])
def test_cells_of_scaled_rows(e):
    from parallel_anns_b200.graph import build_nsg_cells
    n, k = 6000, 24
    x = np.ldexp(_mix(n, 32, 3), e)
    _, knn, (cell, near) = build_nsg_cells(x, R=16, knn_k=k, cells=12, probe=2, sample=n, iters=6, with_knn=True,
                                           with_cells=True)
    _in_cells(x, knn, cell, near, k, range(0, n, 11))


@pytest.mark.parametrize("n,far,kind", [(4096, 7, "outlier"), (9001, 4501, "outlier"), (9001, 4500, "nan"),
                                        (9001, 4501, "inf"), (5000, 3, "distant")])
def test_rows_unlike_the_others(n, far, kind):
    """One row past the error bound's range (9,001 rows: row 4,501 is not in the sample
    the scale comes from), with a NaN or an infinity, or merely distant: the others'
    lists and neighbours do not change."""
    from parallel_anns_b200.graph import build_nsg
    from parallel_anns_b200.searching import Index, ground_truth
    d, k = 40, 20
    x = _mix(n, d, 5)
    bad, ref = x.copy(), x.copy()
    value = {"outlier": 2.0 ** 62, "nan": np.nan, "inf": np.inf, "distant": 2.0 ** 13}[kind]
    bad[far], ref[far] = value, 2.0 ** 62
    rest = np.arange(n) != far
    oknn, _ = O.host_knn(ref, None, k)
    g, knn = build_nsg(bad, R=16, knn_k=k, with_knn=True)
    assert np.array_equal(knn[rest], oknn[rest])
    if kind in ("outlier", "inf"):  # all distances of the row itself are equal
        assert np.array_equal(knn[far], np.arange(k + 1)[np.arange(k + 1) != far][:k])
    q = _mix(2500, d, 5)[::-1].copy()
    oids, _ = O.ground_truth(ref, q, 10)
    with Index(0) as ix:
        ix.set_base(bad)
        ix.set_graph(g)
        for m in (2500, 5):
            assert np.array_equal(ground_truth(ix, q[:m], 10)[0], oids[:m])


@pytest.mark.parametrize("equal,offset", [(41, 0.0), (42, 0.0), (300, 0.0), (300, 100.0)])
def test_cells_with_long_runs_of_equal_rows(equal, offset):
    """Equal rows of one cell, as many as a row's list holds and more: the tensor-core
    screen cannot settle the rows near them, the others keep its lists. Every list is
    exact, ties by the lower id, wherever the origin is."""
    from parallel_anns_b200.graph import build_nsg_cells
    n, d, k = 6000, 32, 24
    x = _mix(n, d, 3)
    at = np.random.default_rng(equal).permutation(n)[:equal]
    x[at] = x[at[0]]
    x = (x + np.float32(offset)).astype(np.float32)
    _, knn, (cell, near) = build_nsg_cells(x, R=16, knn_k=k, cells=12, probe=2, sample=n, iters=6, with_knn=True,
                                           with_cells=True)
    assert np.unique(cell[at]).size == 1
    _in_cells(x, knn, cell, near, k, [*at[:60], *range(0, n, 11)])
    for a in at[:60]:
        if equal > k:
            assert np.array_equal(knn[a], np.sort(at[at != a])[:k])
