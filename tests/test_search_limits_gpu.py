"""Searches at the edge of what the kernels may assume: init lists with a repeated
vertex, searches that reach fewer than K vertices, distances that are not numbers."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _ring(n, deg):
    """Vertex v -> v + 1 .. v + deg (mod n)."""
    from parallel_anns_b200.formats import NSGGraph
    nb = (np.arange(n)[:, None] + 1 + np.arange(deg)) % n
    return NSGGraph(deg, 0, np.arange(n + 1, dtype=np.int64) * deg, nb.reshape(-1).astype(np.uint32))


@pytest.mark.parametrize("L", [5, 6, 40, 500])
def test_efanna_refuses_a_repeated_neighbour_of_the_entry(L):
    """The default efanna2e lists begin with the entry's neighbours; slot 5 repeats
    slot 2, so lists of more than five ids hold a vertex twice. The PANNS list takes
    every neighbour once."""
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.searching import Index
    rng = np.random.default_rng(L)
    n, K = 500, 5
    x, q = rng.random((n, 16), dtype=np.float32), rng.random((9, 16), dtype=np.float32)
    g = _ring(n, 8)
    g.nbrs[5] = g.nbrs[2]
    og = O.Graph.from_nsg(g)
    with Index(0) as ix:
        ix.set_base(x)
        ix.set_graph(g)
        if L <= 5:
            ids, _ = ix.search(q, K=K, L=L, mode=N.MODE_EFANNA, distance=N.DIST_L2)
            init = O.efanna_init_ids(og, L, q.shape[0])
            assert np.array_equal(ids, O.search_efanna(x, og, q, K, L, init_ids=init)[0])
        else:
            with pytest.raises(N.PannsError, match="duplicate init id"):
                ix.search(q, K=K, L=L, mode=N.MODE_EFANNA, distance=N.DIST_L2)
        ids, _ = ix.search(q, K=K, L=L, mode=N.MODE_TOP_M, M=4, distance=N.DIST_L2)
        assert np.array_equal(ids, O.search_top_m(x, og, q, K, L, 4, kind=O.DIST_L2)[0])
        g2 = _ring(n, 8)  # the next graph is judged by its own row
        ix.set_graph(g2)
        ids, _ = ix.search(q, K=K, L=L, mode=N.MODE_EFANNA, distance=N.DIST_L2)
        init = O.efanna_init_ids(O.Graph.from_nsg(g2), L, q.shape[0])
        assert np.array_equal(ids, O.search_efanna(x, O.Graph.from_nsg(g2), q, K, L, init_ids=init)[0])


@pytest.mark.parametrize("storage", [0, 1, 2])
def test_learned_search_that_reaches_fewer_than_k(storage):
    """Components of five vertices, two learned entries and one plain init id: at
    most fifteen vertices are reached, K is 40. The result slots left over hold ~0."""
    from parallel_anns_b200 import learned as LE
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.formats import NSGGraph
    from parallel_anns_b200.searching import Index
    rng = np.random.default_rng(storage)
    n, d, R, K, L = 1000, 24, 256, 40, 64
    x, q = rng.random((n, d), dtype=np.float32), rng.random((70, d), dtype=np.float32)
    v = np.arange(n)
    nb = (v // 5 * 5)[:, None] + (v[:, None] + 1 + np.arange(4)) % 5
    g = NSGGraph(4, 7, np.arange(n + 1, dtype=np.int64) * 4, nb.reshape(-1).astype(np.uint32))
    plain = O.prepare_init_ids(O.Graph.from_nsg(g), L)[0]
    model = LE.LearnedModel(d, R, LE.init_params(d, R, 3, 4.0), rng.permutation(n)[:R].astype(np.uint32))
    with Index(0) as ix:
        ix.set_base(x, storage=storage) if storage else ix.set_base(x)
        ix.set_graph(g)
        LE.attach(ix, model, E=2, L_init=1, use_L=False)
        for w in (0, 1, 2, 4, 8):
            ids, _ = ix.search(q, K=K, L=L, mode=N.MODE_TOP_M, M=4, flags=N.FLAG_LEARNED, storage=storage,
                               warps_per_query=w)
            _, fallback, entries = LE.record(ix, q.shape[0])
            assert not fallback.any()
            for i in range(q.shape[0]):
                reach = {int(u) // 5 * 5 + j for u in [plain, *entries[i]] for j in range(5)}
                assert {int(u) for u in ids[i, :len(reach)]} == reach, (w, i)
                assert (ids[i, len(reach):] == 0xFFFFFFFF).all(), (w, i)


def _graph(n, deg, seed):
    from parallel_anns_b200.formats import NSGGraph
    rng = np.random.default_rng(seed)
    nb = rng.integers(0, n, size=(n, deg), dtype=np.int64)
    nb[:, 0] = (np.arange(n) + 1) % n
    nb = (nb + (nb == np.arange(n)[:, None])) % n
    return NSGGraph(deg, 0, np.arange(n + 1, dtype=np.int64) * deg, nb.reshape(-1).astype(np.uint32))


@pytest.mark.parametrize("n,d,deg,L,M,K", [(5000, 24, 30, 64, 4, 50), (3000, 40, 60, 700, 8, 100),
                                           (9000, 16, 12, 300, 16, 300)])
def test_nan_counts_as_infinity(n, d, deg, L, M, K):
    """Rows and queries with a NaN: the same ids as with rows and queries whose
    squared distances overflow to infinity, in every kernel of the float32 search."""
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.searching import Index
    rng = np.random.default_rng(n)
    x, q = rng.random((n, d), dtype=np.float32), rng.random((40, d), dtype=np.float32)
    bad = rng.permutation(n)[:n // 3]
    xn, xi, qn, qi = x.copy(), x.copy(), q.copy(), q.copy()
    xn[bad, 3], xi[bad, 3] = np.nan, 1e30
    qn[::7, 1], qi[::7, 1] = np.nan, -1e30  # away from the rows': no difference is zero
    g = _graph(n, deg, L)
    og = O.Graph.from_nsg(g)
    with Index(0) as ix:
        ix.set_base(xn)
        ix.set_graph(g)
        ref, nd = O.search_top_m(xi, og, qi, K, L, M, kind=O.DIST_L2)
        for w in (0, 1, 2, 4, 8):
            ids, s = ix.search(qn, K=K, L=L, mode=N.MODE_TOP_M, M=M, distance=N.DIST_L2, warps_per_query=w)
            assert np.array_equal(ids, ref) and s["n_dist"] == nd, w
        ref, nd = O.search_pss(xi, og, qi, K, L, L, 2, 3, kind=O.DIST_L2)
        ids, s = ix.search(qn, K=K, L=L, mode=N.MODE_PSS_V5, distance=N.DIST_L2, T=3, X=2)
        assert np.array_equal(ids, ref) and s["n_dist"] == nd
        init = ix.efanna_init_ids(L, q.shape[0])
        ref, nd = O.search_efanna(xi, og, qi, K, L, init_ids=init)
        ids, s = ix.search(qn, K=K, L=L, mode=N.MODE_EFANNA, distance=N.DIST_L2, init_ids=init)
        assert np.array_equal(ids, ref) and s["n_dist"] == nd
        # the norm trick, where such rows have no counterpart: K different vertices
        for w in (1, 2, 8):
            ids, _ = ix.search(qn, K=K, L=L, mode=N.MODE_TOP_M, M=M, warps_per_query=w)
            assert ids.max() < n and all(np.unique(r).size == K for r in ids)


@pytest.mark.parametrize("storage", [1, 2])
def test_nan_in_reduced_copies(storage):
    """K different vertices, the same with any number of warps, where the reduced rows,
    their norms and the exact distances hold NaNs."""
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.searching import Index
    rng = np.random.default_rng(storage)
    n, d, K, L = 6000, 32, 60, 200
    x, q = rng.random((n, d), dtype=np.float32), rng.random((40, d), dtype=np.float32)
    x[rng.permutation(n)[:n // 3], 5] = np.nan
    q[::5, 2] = np.nan
    with Index(0) as ix:
        ix.set_base(x, storage=storage)
        ix.set_graph(_graph(n, 20, 1))
        one, _ = ix.search(q, K=K, L=L, mode=N.MODE_TOP_M, M=8, storage=storage, warps_per_query=1)
        assert one.max() < n and all(np.unique(r).size == K for r in one)
        for w in (0, 2, 4, 8):
            ids, _ = ix.search(q, K=K, L=L, mode=N.MODE_TOP_M, M=8, storage=storage, warps_per_query=w)
            assert np.array_equal(ids, one), w


def test_efanna_build_with_nan_rows():
    """IndexNSG::Build on rows with NaNs equals the build on rows with infinities in
    their place: every distance to such a row, its own included, is infinite."""
    from parallel_anns_b200.graph import efanna_build
    rng = np.random.default_rng(5)
    n, d = 600, 16
    x = rng.random((n, d), dtype=np.float32)
    knn = O.host_knn(x, None, 20)[0]
    xn, xi = x.copy(), x.copy()
    xn[::9, 2], xi[::9, 2] = np.nan, np.inf
    a, b = efanna_build(xn, knn, 60, 12, 80), efanna_build(xi, knn, 60, 12, 80)
    assert a.entry < n and a.nbrs.max() < n
    assert np.array_equal(a.offsets, b.offsets) and np.array_equal(a.nbrs, b.nbrs)


@pytest.mark.parametrize("warps", [1, 4])
def test_fp8_search_at_any_scale(warps):
    """Base and queries times a power of two: the FP8 rows are the same, their scales
    and the queries follow, so the ids do too. (No element is near zero, so none
    leaves half precision's range for another reason.)"""
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.searching import Index
    rng = np.random.default_rng(2)
    n, d, K, L = 5000, 64, 20, 60

    def rows(m):
        return ((0.5 + 0.5 * rng.random((m, d))) * rng.choice([-1, 1], (m, d))).astype(np.float32)

    x, q, g = rows(n), rows(50), _graph(n, 24, 4)
    want = None
    for e in (0, -30, -12, -6, -5, 5, 6, 7, 8, 20):
        with Index(0) as ix:
            ix.set_base(np.ldexp(x, e), storage=N.STORE_FP8)
            ix.set_graph(g)
            ids, _ = ix.search(np.ldexp(q, e), K=K, L=L, mode=N.MODE_TOP_M, M=4, storage=N.STORE_FP8,
                               warps_per_query=warps)
        want = ids if want is None else want
        assert np.array_equal(ids, want), e


def test_fp8_search_of_integers():
    """Integers up to 255: queries times their scales and 2^12 are past half precision.
    The FP8 search finds what the float32 search finds, but for a few."""
    from parallel_anns_b200 import datasets as ds
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.graph import build_nsg
    from parallel_anns_b200.searching import Index
    x, q = ds.uint8_cube(12_000, 128, seed=3), ds.uint8_cube(200, 128, seed=4)
    with Index(0) as ix:
        ix.set_base(x, storage=N.STORE_FP8)
        ix.set_graph(build_nsg(x, R=64, knn_k=64))
        a, _ = ix.search(q, K=50, L=400, mode=N.MODE_TOP_M, M=4)
        b, _ = ix.search(q, K=50, L=400, mode=N.MODE_TOP_M, M=4, storage=N.STORE_FP8)
        far, _ = ix.search(q * np.float32(1000), K=50, L=400, mode=N.MODE_TOP_M, M=4, storage=N.STORE_FP8)
    assert np.mean([np.intersect1d(u, v).size / 50 for u, v in zip(a, b)]) > 0.95
    assert far.max() < 12_000 and all(np.unique(r).size == 50 for r in far)
