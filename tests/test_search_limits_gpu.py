"""Searches at the edge of what the kernels may assume: init lists with a repeated
vertex, searches that reach fewer than K vertices."""
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
