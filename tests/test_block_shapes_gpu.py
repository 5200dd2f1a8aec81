"""The several-warps search kernel in the forms its launch rule picks: 2 to 16
warps per query, the visited bitset in shared and in global memory, survivor lists
on both sides of the counting limit, rows longer than a head row, equal distances.
Ids and distance counts equal the one-warp kernel's and the oracle's."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _random_graph(n, deg, seed):
    from parallel_anns_b200.formats import NSGGraph
    rng = np.random.default_rng(seed)
    nb = rng.integers(0, n, size=(n, deg), dtype=np.int64)
    nb[:, 0] = (np.arange(n) + 1) % n  # a ring keeps every vertex reachable
    nb = (nb + (nb == np.arange(n)[:, None])) % n
    return NSGGraph(deg, 0, np.arange(n + 1, dtype=np.int64) * deg, nb.reshape(-1).astype(np.uint32))


@pytest.mark.parametrize("n,d,deg,L,M,integer", [
    (2_000_003, 8, 8, 100, 8, False),   # the bitset does not fit shared memory
    (30_000, 24, 50, 64, 4, False),     # overflow lists, fewer candidates than warps
    (20_000, 40, 100, 700, 64, False),  # many candidates a step, long survivor lists
    (5_000, 16, 40, 300, 16, True),     # equal distances
    (3_000, 128, 200, 1, 1, False), (9_000, 256, 33, 1100, 5, False)])
def test_block_shapes_equal_one_warp_and_oracle(n, d, deg, L, M, integer):
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.searching import Index
    rng = np.random.default_rng(n + L)
    x = rng.integers(0, 4, size=(n, d)).astype(np.float32) if integer else rng.random((n, d), dtype=np.float32)
    q = rng.integers(0, 4, size=(5, d)).astype(np.float32) if integer else rng.random((5, d), dtype=np.float32)
    g = _random_graph(n, deg, L)
    K = min(L, 50)
    with Index(0) as ix:
        ix.set_base(x)
        ix.set_graph(g)
        one, s1 = ix.search(q, K=K, L=L, mode=N.MODE_TOP_M, M=M, warps_per_query=1)
        for w in (0, 2, 4, 8):
            ids, s = ix.search(q, K=K, L=L, mode=N.MODE_TOP_M, M=M, warps_per_query=w)
            assert np.array_equal(ids, one), w
            assert all(s[f] == s1[f] for f in ("n_dist", "n_expand", "n_edges", "n_iter")), w
        # a batch the rule gives fewer warps
        many, sm = ix.search(np.repeat(q, 80, axis=0), K=K, L=L, mode=N.MODE_TOP_M, M=M)
        assert np.array_equal(many, np.repeat(one, 80, axis=0)) and sm["n_dist"] == 80 * s1["n_dist"]
    ref, nd = O.search_top_m(x, O.Graph.from_nsg(g), q, K, L, M)
    assert np.array_equal(one, ref) and s1["n_dist"] == nd


@pytest.mark.parametrize("n,shared", [(2_000_003, False), (40_000, True)])
def test_one_warp_and_pss_with_either_bitset(n, shared):
    """PSS_v5, efanna2e and the one-warp kernel on a base whose visited bits fit
    shared memory and on one where they do not."""
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.searching import Index
    rng = np.random.default_rng(n)
    d, L, K = 16, 60, 20
    x, q = rng.random((n, d), dtype=np.float32), rng.random((70, d), dtype=np.float32)
    g = _random_graph(n, 12, 3)
    og = O.Graph.from_nsg(g)
    assert shared == (n // 8 < 200_000)
    with Index(0) as ix:
        ix.set_base(x)
        ix.set_graph(g)
        for T, X in ((1, 1), (4, 2), (7, 1)):
            ids, s = ix.search(q, K=K, L=L, mode=N.MODE_PSS_V5, distance=N.DIST_L2, T=T, X=X)
            ref, nd = O.search_pss(x, og, q, K, L, L, X, T, kind=O.DIST_L2)
            assert np.array_equal(ids, ref) and s["n_dist"] == nd, (T, X)
        init = ix.efanna_init_ids(L, q.shape[0])
        ids, s = ix.search(q, K=K, L=L, mode=N.MODE_EFANNA, distance=N.DIST_L2, init_ids=init)
        ref, nd = O.search_efanna(x, og, q, K, L, init_ids=init)
        assert np.array_equal(ids, ref) and s["n_dist"] == nd
        ids, s = ix.search(q, K=K, L=L, mode=N.MODE_TOP_M, M=3, distance=N.DIST_L2, warps_per_query=1)
        ref, nd = O.search_top_m(x, og, q, K, L, 3, kind=O.DIST_L2)
        assert np.array_equal(ids, ref) and s["n_dist"] == nd
