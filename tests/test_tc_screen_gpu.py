"""The tensor-core screens of graph construction and ground truth where they
can go wrong: first and last sizes of each path, operand widths on both sides of
a 64-wide slice, ties longer than a list, data far from the origin, bounds that
overflow the range lists. Graphs and ids are compared for equality with the
oracle's; distances are sums of d positive float64 terms, each side within
(d + 2) 2^-53 of the exact value."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _data(kind, n, d, seed):
    from parallel_anns_b200 import datasets as ds
    if kind == "u8":
        return ds.uint8_cube(n, d, seed=seed)
    x = ds.gaussian_mixture(n, d, 64, 0.3, seed=seed, means_seed=seed) if d >= 8 else \
        np.random.default_rng(seed).random((n, d), dtype=np.float32)
    if kind == "far":
        return (x + np.float32(100.0)).astype(np.float32)
    if kind == "ties":  # more equal rows than a list holds
        x[::7] = x[0]
    return x


@pytest.mark.parametrize("n,d,k,R,kind", [
    (1023, 96, 64, 50, "mix"), (1024, 96, 64, 50, "mix"), (4096, 24, 32, 20, "mix"), (4097, 24, 32, 20, "mix"),
    (4225, 61, 20, 12, "mix"), (4224, 62, 1, 1, "mix"), (2500, 3, 16, 8, "mix"), (5000, 256, 128, 70, "mix"),
    (2000, 253, 100, 40, "mix"), (6000, 128, 64, 64, "u8"), (5000, 96, 64, 50, "far"), (4500, 32, 16, 8, "ties")])
def test_automatic_build_equals_oracle(n, d, k, R, kind):
    from parallel_anns_b200.graph import build_nsg
    x = _data(kind, n, d, n + d)
    g, knn = build_nsg(x, R=R, knn_k=k, with_knn=True)
    og, oknn = O.build_nsg(x, k, R)
    assert np.array_equal(knn, oknn)
    assert g.entry == og.entry and np.array_equal(g.offsets, og.offsets) and np.array_equal(g.nbrs, og.nbrs)


@pytest.mark.parametrize("n,d,nq,k,kind", [
    (300, 24, 1, 10, "mix"), (4095, 96, 129, 100, "mix"), (9000, 200, 300, 50, "mix"), (6000, 96, 40, 512, "mix"),
    (6000, 96, 40, 513, "mix"), (7000, 128, 200, 100, "u8"), (6000, 32, 100, 10, "ties")])
def test_ground_truth_equals_oracle(n, d, nq, k, kind):
    from parallel_anns_b200.graph import build_nsg
    from parallel_anns_b200.searching import Index, ground_truth
    x = _data(kind, n, d, n)
    q = np.concatenate([_data(kind if kind != "ties" else "mix", nq, d, n), x[:1]])  # and a vertex itself
    with Index(0) as ix:
        ix.set_base(x)
        ix.set_graph(build_nsg(x, R=16, knn_k=24))
        ids, dist = ground_truth(ix, q, k)
    oids, odist = O.ground_truth(x, q, k)
    assert np.array_equal(ids, oids)
    np.testing.assert_allclose(dist, odist, rtol=(d + 2) * 2.0 ** -52, atol=0)


@pytest.mark.parametrize("n,d,k,kind", [(6000, 32, 10, "ties"), (3001, 96, 1, "far"), (6000, 24, 100, "mix")])
def test_ground_truth_of_few_and_of_many_queries(n, d, k, kind):
    """Few queries take the tiled pass, many the screen: the same answers."""
    from parallel_anns_b200.graph import build_nsg
    from parallel_anns_b200.searching import Index, ground_truth
    x = _data(kind, n, d, n)
    q = _data("far" if kind == "far" else "mix", 5000, d, n)
    q[-1] = x[0]
    oids, odist = O.ground_truth(x, q, k)
    with Index(0) as ix:
        ix.set_base(x)
        ix.set_graph(build_nsg(x, R=16, knn_k=24))
        for nq in (1, 31, 33, 5000):
            ids, dist = ground_truth(ix, q[-nq:], k)
            assert np.array_equal(ids, oids[-nq:]), nq
            np.testing.assert_allclose(dist, odist[-nq:], rtol=(d + 2) * 2.0 ** -52, atol=0)


def test_ground_truth_with_loose_bounds():
    """Two groups no edge joins: searches for the second see only the first, so
    their bounds hold more vertices than a list does and are refined."""
    from parallel_anns_b200.formats import NSGGraph
    from parallel_anns_b200.graph import build_nsg
    from parallel_anns_b200.searching import Index, ground_truth
    rng = np.random.default_rng(3)
    a = rng.random((5000, 32), dtype=np.float32)
    x = np.concatenate([a, a + np.float32(0.5)])
    half = build_nsg(a, R=16, knn_k=24)
    off = np.concatenate([half.offsets, half.offsets[1:] + half.offsets[-1]])
    nbrs = np.concatenate([half.nbrs, half.nbrs + 5000]).astype(np.uint32)
    q = (rng.random((150, 32), dtype=np.float32) + np.float32(0.5)).astype(np.float32)
    with Index(0) as ix:
        ix.set_base(x)
        ix.set_graph(NSGGraph(half.width, half.entry, off, nbrs))
        ids, dist = ground_truth(ix, q, 20)
    oids, odist = O.ground_truth(x, q, 20)
    assert np.array_equal(ids, oids)
    np.testing.assert_allclose(dist, odist, rtol=34 * 2.0 ** -52, atol=0)


def test_ground_truth_with_loose_bounds_of_many_queries():
    """The same with as many queries as the screen takes, so that its lists
    overflow and are refined."""
    from parallel_anns_b200.formats import NSGGraph
    from parallel_anns_b200.graph import build_nsg
    from parallel_anns_b200.searching import Index, ground_truth
    rng = np.random.default_rng(4)
    a = rng.random((5000, 32), dtype=np.float32)
    x = np.concatenate([a, a + np.float32(0.5)])
    half = build_nsg(a, R=16, knn_k=24)
    off = np.concatenate([half.offsets, half.offsets[1:] + half.offsets[-1]])
    nbrs = np.concatenate([half.nbrs, half.nbrs + 5000]).astype(np.uint32)
    q = (rng.random((3000, 32), dtype=np.float32) + np.float32(0.5)).astype(np.float32)
    with Index(0) as ix:
        ix.set_base(x)
        ix.set_graph(NSGGraph(half.width, half.entry, off, nbrs))
        ids, dist = ground_truth(ix, q, 20)
    oids, odist = O.ground_truth(x, q, 20)
    assert np.array_equal(ids, oids)
    np.testing.assert_allclose(dist, odist, rtol=34 * 2.0 ** -52, atol=0)


def test_threads_with_different_widths():
    """Constructions and ground truths of different widths at the same time."""
    from concurrent.futures import ThreadPoolExecutor

    from parallel_anns_b200.graph import build_nsg
    from parallel_anns_b200.searching import Index, ground_truth

    def work(d):
        x, q = _data("mix", 3000, d, d), _data("mix", 70, d, d)
        got = []
        for _ in range(6):
            g = build_nsg(x, R=16, knn_k=24)
            with Index(0) as ix:
                ix.set_base(x)
                ix.set_graph(g)
                got.append((g.entry, g.nbrs, *ground_truth(ix, q, 10)))
        return got

    widths = [8, 64, 136, 256]
    with ThreadPoolExecutor(len(widths)) as pool:
        for d, got in zip(widths, pool.map(work, widths)):
            x, q = _data("mix", 3000, d, d), _data("mix", 70, d, d)
            og, _ = O.build_nsg(x, 24, 16)
            oids, _ = O.ground_truth(x, q, 10)
            for entry, nbrs, ids, _ in got:
                assert entry == og.entry and np.array_equal(nbrs, og.nbrs) and np.array_equal(ids, oids), d
